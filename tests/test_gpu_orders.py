"""The one-point-per-block FP64 kernels at the edges of their tile splits.

Orders just below, at and above each padded order (8, 16, 24, 32, 48, then
every multiple of 8 up to 104, above it of 16), leads
of another order than the device, layers with their own blocks, and both tile
splits of order 9..16 (chosen by the number of points).  Random systems at an
eta that keeps the decimation well conditioned, against the CPU oracle to the
parity bound of the FP64 path, 1e-10 of the largest entry.
"""

import numpy as np
import pytest
import torch

from negfpy_b200 import _lib, engine
from oracle import negf_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-10
ETA = 0.05


def _herm(rng, n):
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (a + a.conj().T) / (2 * np.sqrt(n)) + 2.0 * np.eye(n)


def _any(rng, n, m):
    return 0.6 * (rng.standard_normal((n, m)) + 1j * rng.standard_normal((n, m))) / np.sqrt(n + m)


def _system(n, nl, nr, layers, seed):
    rng = np.random.default_rng(seed)
    lead = lambda m: (_herm(rng, m), _any(rng, m, m))  # noqa: E731
    return {"l": lead(nl), "r": lead(nr), "on": [_herm(rng, n) for _ in range(layers)],
            "cp": [_any(rng, n, n) for _ in range(layers - 1)], "vl": _any(rng, n, nl), "vr": _any(rng, n, nr)}


def _solve(s, omegas):
    c = lambda x: x[None]  # noqa: E731
    lead = lambda b: {"d00": c(b[0]), "d01": c(b[1]), "d10": None}  # noqa: E731
    cp = np.stack(s["cp"]) if s["cp"] else np.zeros((1,) + s["on"][0].shape, dtype=complex)
    sysobj = engine.StackedSystem.from_arrays(lead(s["l"]), lead(s["r"]), np.stack(s["on"])[None], cp[None],
                                              len(s["on"]), s["vl"][None], s["vr"][None], same_leads=False)
    om = torch.as_tensor(omegas, device="cuda")
    ki = torch.zeros(om.numel(), dtype=torch.int32, device="cuda")
    eta = torch.full_like(om, ETA)
    g = engine.sgf_sr(*sysobj.lead_l, om, eta, ki, want_dos=True)
    r = sysobj.transmission(om, ki, eta)
    assert int(r["status"].abs().sum()) == 0 and int(g["status"].abs().sum()) == 0
    return g["g"].cpu().numpy(), g["dos"].cpu().numpy(), r["T"].cpu().numpy(), g["iters"].cpu().numpy()


@pytest.mark.parametrize("n,nl,nr,layers", [
    (2, 2, 2, 3), (7, 8, 7, 1), (8, 8, 3, 4), (9, 9, 9, 2), (15, 16, 2, 3), (16, 16, 16, 3), (17, 17, 9, 2),
    (23, 24, 23, 3), (24, 24, 24, 1), (25, 25, 8, 2), (31, 32, 31, 2), (32, 32, 32, 3), (33, 33, 25, 2),
    (40, 40, 41, 2), (47, 48, 47, 3), (48, 48, 48, 2), (5, 48, 20, 2), (49, 49, 48, 2), (56, 57, 56, 1),
    (64, 64, 10, 3), (65, 65, 64, 2), (72, 72, 72, 2), (73, 80, 73, 2), (81, 88, 50, 1), (89, 96, 89, 2),
    (96, 96, 96, 3), (97, 104, 97, 2), (104, 104, 104, 2), (105, 105, 104, 2), (20, 104, 60, 3)])
def test_orders_match_oracle(n, nl, nr, layers):
    s = _system(n, nl, nr, layers, seed=100 * n + nl)
    omegas = np.array([0.3, 1.1, 1.9])
    g, dos, t, it = _solve(s, omegas)
    for i, w in enumerate(omegas):
        ref, nit = O.sancho_rubio(w, *s["l"], None, ETA)
        assert it[i] == nit
        assert np.max(np.abs(g[i] - ref)) <= TOL * np.max(np.abs(ref))
        d = O.lead_surface_dos(w, *s["l"], None, ETA)
        assert abs(dos[i] - d) <= 10 * TOL * max(abs(d), 1.0)
        tr = O.transmission_point(w, s["on"], s["cp"], (*s["l"], None), (*s["r"], None), ETA, vl=s["vl"], vr=s["vr"],
                                  idx_l=np.arange(n), idx_r=np.arange(n * (layers - 1), n * layers))
        assert abs(t[i] - tr) <= TOL * max(abs(tr), 1.0)


@pytest.mark.parametrize("n,nl,nr,layers,points", [
    (106, 112, 60, 2, 3), (112, 112, 112, 1, 150), (113, 113, 113, 2, 150), (121, 128, 121, 3, 3), (128, 128, 128, 2, 150),
    (129, 129, 129, 2, 3), (8, 150, 8, 2, 3), (161, 161, 100, 2, 3), (192, 192, 192, 2, 3), (193, 193, 193, 1, 3),
    (225, 225, 225, 2, 3), (249, 256, 249, 2, 3), (256, 256, 256, 2, 3)])
def test_large_orders_match_oracle(n, nl, nr, layers, points):
    """Strips of 32 columns at their remainders, block sizes at the edges of their
    classes, and up to order 128 both forms (chosen by the number of points)."""
    s = _system(n, nl, nr, layers, seed=100 * n + nl)
    omegas = np.resize([0.3, 1.1, 1.9], points)
    g, dos, t, it = _solve(s, omegas)
    for i, w in enumerate(omegas[:3]):
        ref, nit = O.sancho_rubio(w, *s["l"], None, ETA)
        assert it[i] == nit
        assert np.max(np.abs(g[i] - ref)) <= TOL * np.max(np.abs(ref))
        d = O.lead_surface_dos(w, *s["l"], None, ETA)
        assert abs(dos[i] - d) <= 10 * TOL * max(abs(d), 1.0)
        tr = O.transmission_point(w, s["on"], s["cp"], (*s["l"], None), (*s["r"], None), ETA, vl=s["vl"], vr=s["vr"],
                                  idx_l=np.arange(n), idx_r=np.arange(n * (layers - 1), n * layers))
        assert abs(t[i] - tr) <= TOL * max(abs(tr), 1.0)
        for x in (g, dos, t, it):
            assert all(np.array_equal(x[i], x[k]) for k in range(i, points, 3))


@pytest.mark.parametrize("n", [96, 120, 150])
@pytest.mark.parametrize("shift", [16, 240])
def test_workspace_at_any_16_byte_boundary(n, shift):
    """A workspace that starts 16 bytes off a 32-byte boundary gives the same
    surface GF and T as an aligned one."""
    s = _system(n, n, n, 2, seed=n)
    c = lambda x: torch.as_tensor(x[None], device="cuda").contiguous()  # noqa: E731
    om = torch.tensor([0.3, 1.1, 1.9], dtype=torch.float64, device="cuda")
    eta = torch.full_like(om, ETA)
    ki = torch.zeros(3, dtype=torch.int32, device="cuda")
    h00, h01, on, cp = c(s["l"][0]), c(s["l"][1]), c(np.stack(s["on"])), c(np.stack(s["cp"]))
    vl, vr = c(s["vl"]), c(s["vr"])
    ref = engine.sgf_sr(h00, h01, None, om, eta, ki)
    tref, _ = engine.rgf_transmission(on, cp, 2, vl, vr, ref["g"], ref["g"], om, eta, ki, None)
    lib, ptr = _lib.load(), _lib.ptr
    need = [int(lib.negf_sgf_workspace_bytes(n)), int(lib.negf_rgf_workspace_bytes(n, n, n))]
    ws = torch.empty(max(need) + 512, dtype=torch.uint8, device="cuda")
    off = -ws.data_ptr() % 256 + shift
    g, t = torch.empty_like(ref["g"]), torch.empty_like(tref)
    st, it = torch.empty_like(ki), torch.empty_like(ki)
    _lib.check(lib.negf_sgf_sr_f64(n, 3, ptr(h00), ptr(h01), None, 0, ptr(ki), ptr(om), ptr(eta), 1e-12, 200, ptr(g), None,
                                   ptr(it), ptr(st), ptr(ws[off:]), need[0], _lib.stream_handle(None)), "negf_sgf_sr_f64")
    _lib.check(lib.negf_rgf_transmission_f64(
        n, n, n, 2, 3, ptr(on), 0, n * n, ptr(cp), 0, n * n, ptr(vl), 0, ptr(vr), 0, ptr(g), n * n, ptr(g), n * n, ptr(ki),
        ptr(om), ptr(eta), None, ptr(t), ptr(st), ptr(ws[off:]), need[1], _lib.stream_handle(None)),
        "negf_rgf_transmission_f64")
    assert torch.equal(g, ref["g"]) and torch.equal(t, tref)


@pytest.mark.parametrize("n,nl,nr,layers,points", [
    (1, 2, 1, 2, 700), (15, 16, 9, 1, 700), (16, 16, 16, 3, 1300), (17, 20, 17, 2, 700), (32, 32, 32, 2, 800),
    (33, 33, 30, 3, 500), (48, 48, 48, 2, 500), (49, 64, 49, 1, 40), (64, 64, 64, 3, 310), (65, 80, 65, 2, 40),
    (80, 80, 80, 2, 40), (81, 96, 81, 3, 40), (96, 96, 96, 2, 160), (97, 97, 97, 2, 40)])
def test_reduced_precision_orders(n, nl, nr, layers, points):
    """The refined solve to the FP64 bound and the mixed one to its FP32-level
    bound (1e-4) against the FP64 kernels, at the edges of the padded orders and
    with more points than the launch holds blocks."""
    s = _system(n, nl, nr, layers, seed=11 * n + nl)
    c = lambda x: torch.as_tensor(x[None], device="cuda").contiguous()  # noqa: E731
    om = torch.linspace(0.2, 2.2, points, dtype=torch.float64, device="cuda")
    eta = torch.full_like(om, ETA)
    ki = torch.zeros(points, dtype=torch.int32, device="cuda")
    rl = engine.sgf_sr(c(s["l"][0]), c(s["l"][1]), None, om, eta, ki)
    rr = engine.sgf_sr(c(s["r"][0]), c(s["r"][1]), None, om, eta, ki)
    args = (c(np.stack(s["on"])), c(np.stack(s["cp"])) if layers > 1 else None, layers, c(s["vl"]), c(s["vr"]), rl["g"],
            rr["g"], om, eta, ki, None)
    t, st = engine.rgf_transmission(*args)
    tm, sm = engine.rgf_transmission(*args, precision="mixed")
    tr, sr, steps = engine.rgf_transmission_refine64(*args)
    assert int(st.abs().sum()) == 0 and int(sm.abs().sum()) == 0 and int(sr.abs().sum()) == 0
    scale = t.abs().clamp(min=1.0)
    assert float(((tr - t).abs() / scale).max()) <= TOL
    assert float(((tm - t).abs() / scale).max()) <= 1e-4
    assert int(steps.min()) >= 1 and int(steps.max()) <= engine.REFINE_MAX_STEPS


@pytest.mark.parametrize("n", [9, 12, 16])
def test_both_splits_of_order_16_agree_bitwise(n):
    s = _system(n, n, n, 4, seed=n)
    omegas = np.linspace(0.1, 2.5, 1200)  # above the few-points split, whose largest call is 592
    g, dos, t, it = _solve(s, omegas)
    for a, b in ((0, 592), (592, 593), (600, 1193)):
        gp, dp, tp, ip = _solve(s, omegas[a:b])
        for x, y in ((g, gp), (dos, dp), (t, tp), (it, ip)):
            assert np.array_equal(x[a:b], y)


def _dense(s, z, sl, sr):
    """A of the device as a torch complex128 matrix (differentiable in the blocks)."""
    n, layers = s["on"][0].shape[0], len(s["on"])
    rows = []
    for i in range(layers):
        row = [torch.zeros((n, n), dtype=torch.complex128) for _ in range(layers)]
        row[i] = z * torch.eye(n, dtype=torch.complex128) - s["on"][i]
        if i == 0:
            row[i] = row[i] - sl
        if i == layers - 1:
            row[i] = row[i] - sr
        if i + 1 < layers:
            row[i + 1] = -s["cp"][i]
        if i > 0:
            row[i - 1] = -s["cp"][i - 1].mH
        rows.append(torch.cat(row, 1))
    return torch.cat(rows, 0)


@pytest.mark.parametrize("n,nl,nr,layers", [
    (3, 3, 3, 2), (16, 16, 9, 1), (17, 24, 17, 3), (25, 25, 25, 2), (33, 48, 33, 2), (49, 49, 64, 2), (65, 65, 72, 3),
    (73, 73, 80, 2), (81, 96, 81, 2), (97, 97, 104, 2), (105, 105, 105, 2)])
def test_adjoint_and_full_green_orders(n, nl, nr, layers):
    """The adjoint blocks, self-energy adjoints, surface-GF adjoint and full G at
    the edges of their padded orders, against torch autograd through the dense
    device matrix (1e-10 of the largest entry: the solves are well conditioned
    at this eta)."""
    s = _system(n, nl, nr, layers, seed=7 * n + layers)
    w, z = 1.1, (1.1 + 1j * ETA) ** 2
    c = lambda x: torch.as_tensor(x[None], device="cuda").contiguous()  # noqa: E731
    om = torch.tensor([w], dtype=torch.float64, device="cuda")
    eta = torch.full_like(om, ETA)
    ki = torch.zeros(1, dtype=torch.int32, device="cuda")
    rl = engine.sgf_sr(c(s["l"][0]), c(s["l"][1]), None, om, eta, ki)
    rr = engine.sgf_sr(c(s["r"][0]), c(s["r"][1]), None, om, eta, ki)
    on = c(np.stack(s["on"]))
    cp = c(np.stack(s["cp"])) if layers > 1 else None
    vl, vr = c(s["vl"]), c(s["vr"])
    wt = torch.ones(1, dtype=torch.float64, device="cuda")
    t, st, x_on, x_cp, xs_l, xs_r = engine.rgf_adjoint(on, cp, layers, vl, vr, rl["g"], rr["g"], om, eta, ki, None, wt,
                                                       want_sigma=True, deterministic=True)
    gg, gsl, gsr, gst = engine.device_green(on, cp, layers, vl, vr, rl["g"], rr["g"], om, eta, ki, None)
    ad = engine.sgf_adjoint(c(s["l"][1]), None, vl, rl["g"], xs_l, ki, deterministic=True)
    assert int(st[0]) == 0 and int(gst[0]) == 0 and int(ad["status"][0]) == 0
    # reference: leaves are the blocks, V_L, V_R and both surface GFs
    lf = lambda x: torch.as_tensor(x).clone().requires_grad_(True)  # noqa: E731
    ref = {"on": [lf(b) for b in s["on"]], "cp": [lf(b) for b in s["cp"]]}
    tvl, tvr = lf(s["vl"]), lf(s["vr"])
    tg = [lf(r["g"][0].cpu().numpy()) for r in (rl, rr)]
    sl, sr = tvl @ tg[0] @ tvl.mH, tvr @ tg[1] @ tvr.mH
    sl.retain_grad(), sr.retain_grad()
    g = torch.linalg.inv(_dense(ref, z, sl, sr))
    g0 = g[:n, (layers - 1) * n:]
    tt = torch.trace(1j * (sl - sl.mH) @ g0 @ (1j * (sr - sr.mH)) @ g0.mH).real
    tt.backward()
    near = lambda a, b: float((a - b).abs().max()) <= TOL * float(b.abs().max())  # noqa: E731
    adj = lambda x: 2.0 * x.cpu().conj().transpose(-1, -2)  # noqa: E731  (torch's gradient from X)
    assert abs(t[0].item() - tt.item()) <= TOL * max(1.0, abs(tt.item()))
    assert near(gg[0].cpu(), g.detach()) and near(gsl[0].cpu(), sl.detach()) and near(gsr[0].cpu(), sr.detach())
    assert near(adj(x_on[0]), torch.stack([b.grad for b in ref["on"]]))
    if layers > 1:
        assert near(adj(x_cp[0]), torch.stack([b.grad for b in ref["cp"]]))
    assert near(adj(xs_l[0]), sl.grad) and near(adj(xs_r[0]), sr.grad)
    assert near(adj(ad["v"][0]), tvl.grad)
    # H00bar = g Lam g with Lam - Q Lam P = gbar, P = g H01, Q = H01^H g, gbar = V^H X V
    gl, h01 = rl["g"][0].cpu(), torch.as_tensor(s["l"][1])
    v, x = tvl.detach(), xs_l[0].cpu()
    lam, a, b = v.mH @ x @ v, h01.mH @ gl, gl @ h01
    for _ in range(60):
        lam, a, b = lam + a @ lam @ b, a @ a, b @ b
    h00 = gl @ lam @ gl
    assert near(ad["h00"][0].cpu(), h00)
    assert near(ad["h01"][0].cpu(), gl @ h01.mH @ h00 + (h00 @ h01 @ gl).mH)


@pytest.mark.parametrize("n", [3, 16, 23, 32, 48, 64, 72, 80, 96, 104])
@pytest.mark.parametrize("layers", [1, 2])
def test_last_diagonal_block_of_full_green(n, layers):
    """G_{L-1,L-1} is read back by other lanes than wrote it: many points, every
    padded order, equal points bitwise equal and the block the oracle's to 1e-10."""
    s = _system(n, n, n, layers, seed=31 * n + layers)
    distinct, points = 3, 600
    c = lambda x: torch.as_tensor(x[None], device="cuda").contiguous()  # noqa: E731
    om = torch.tensor(np.resize([0.3, 1.1, 1.9], points), device="cuda")
    eta = torch.full_like(om, ETA)
    ki = torch.zeros(points, dtype=torch.int32, device="cuda")
    rl = engine.sgf_sr(c(s["l"][0]), c(s["l"][1]), None, om, eta, ki)
    rr = engine.sgf_sr(c(s["r"][0]), c(s["r"][1]), None, om, eta, ki)
    g, sl, sr, st = engine.device_green(c(np.stack(s["on"])), c(np.stack(s["cp"])) if layers > 1 else None, layers,
                                        c(s["vl"]), c(s["vr"]), rl["g"], rr["g"], om, eta, ki, None)
    assert int(st.abs().sum()) == 0
    sl, sr = sl.cpu(), sr.cpu()
    on = {"on": [torch.as_tensor(b) for b in s["on"]], "cp": [torch.as_tensor(b) for b in s["cp"]]}
    for i in range(distinct):
        same = g[i::distinct]
        assert torch.equal(same, same[:1].expand_as(same))
        ref = torch.linalg.inv(_dense(on, (float(om[i]) + 1j * ETA) ** 2, sl[i], sr[i]))[-n:, -n:]
        assert float((g[i, -n:, -n:].cpu() - ref).abs().max()) <= TOL * float(ref.abs().max())
