"""Failing points among good ones, more points than the launch holds blocks.

Every block takes failing and good points in turn, so whatever a failure leaves
behind (panels, status words, Tensor Memory, workspace) meets a good point.  A
failing point reports its status and NaN; the good ones are bitwise those of a
call without failing points.

The failures: a matrix with an exactly zero row and column in the middle (z - D
at omega = 1, eta = 0), NaN in a block, couplings whose products overflow, a
sweep limit that is too small.
"""

import numpy as np
import pytest
import torch

from negfpy_b200 import _lib, engine, workloads as W
from negfpy_b200.batch import UnevenBatch

pytestmark = pytest.mark.gpu
ETA = 0.05
GOOD, SINGULAR, NAN, HUGE = range(4)  # the k sets


def _herm(rng, n):
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (a + a.conj().T) / (2 * np.sqrt(n)) + 2.0 * np.eye(n)


def _any(rng, n):
    return 0.6 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2 * n)


def _singular(d):
    """d with z - d singular at z = 1: row and column n // 2 of z - d are zero."""
    j = d.shape[-1] // 2
    d = d.copy()
    d[j, :] = d[:, j] = 0.0
    d[j, j] = 1.0
    return d


def _with_nan(d):
    d = d.copy()
    d[d.shape[-1] - 1, 0] = np.nan
    return d


def _up(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda")


def _near(a, b):
    """Sums over points of which one has zeros among its terms: their order differs,
    by less than 1000 roundings."""
    return float((a - b).abs().max()) <= 1000 * 2.3e-16 * max(float(b.abs().max()), 1.0)


def _kinds(points, kinds):
    """k set of every point: each third point fails, the kinds in turn."""
    k = np.zeros(points, dtype=np.int32)
    bad = np.arange(1, points, 3)
    k[bad] = np.resize(kinds, bad.size)
    return k


def _omegas(k):
    om = np.linspace(0.3, 2.1, k.size)
    om[k == SINGULAR] = 1.0
    eta = np.where(k == SINGULAR, 0.0, ETA)
    return _up(om), _up(eta), torch.as_tensor(k, device="cuda")


def _points(n):
    """More than the kernels of the order hold at once."""
    return 900 if n <= 16 else 700 if n <= 48 else 330


EXPECTED = {GOOD: _lib.OK, SINGULAR: _lib.SINGULAR, NAN: _lib.NONFINITE, HUGE: _lib.UNSTABLE}
ORDERS = [2, 8, 16, 24, 32, 33, 48, 56, 72, 96, 104]


@pytest.mark.parametrize("n,points", [(n, _points(n)) for n in ORDERS] + [(16, 500), (105, 140), (120, 330), (150, 200),
                                                                        (192, 200), (250, 160)])
def test_decimation(n, points):
    rng = np.random.default_rng(n)
    d00, d01 = _herm(rng, n), _any(rng, n)
    h00 = _up(np.stack([d00, _singular(d00), _with_nan(d00), d00]))
    h01 = _up(np.stack([d01, 0 * d01, d01, 1e200 * d01]))
    k = _kinds(points, [SINGULAR, NAN, HUGE])
    om, eta, ki = _omegas(k)
    r = engine.sgf_sr(h00, h01, None, om, eta, ki, want_dos=True)
    assert r["status"].tolist() == [EXPECTED[int(x)] for x in k]
    good = torch.as_tensor(np.nonzero(k == GOOD)[0], device="cuda")
    ref = engine.sgf_sr(h00, h01, None, om[good], eta[good], ki[good], want_dos=True)
    for key in ("g", "dos", "iters"):
        assert torch.equal(r[key][good], ref[key])
    failed = torch.as_tensor(k != GOOD, device="cuda")
    assert bool(torch.isnan(r["dos"][failed]).all())
    # the sweep limit: d01 = 0 is done after one sweep, the others are not
    kz = torch.as_tensor(np.arange(points) % 2, device="cuda", dtype=torch.int32)
    eta = torch.full_like(om, ETA)
    pair = (_up(np.stack([d00, d00])), _up(np.stack([d01, 0 * d01])), None)
    r = engine.sgf_sr(*pair, om, eta, kz, maxiter=2)
    assert r["status"].tolist() == [_lib.OK if x else _lib.MAXITER for x in kz.tolist()]
    ref = engine.sgf_sr(*pair, om[1::2].contiguous(), eta[1::2].contiguous(), kz[1::2].contiguous())
    assert torch.equal(r["g"][1::2], ref["g"]) and torch.equal(r["iters"][1::2], ref["iters"])


def _device(n, layers, rng):
    """Blocks of the k sets GOOD, SINGULAR, NAN: the middle layer fails, uncoupled where
    it is singular, so that its pivots are exact zeros."""
    on = np.stack([_herm(rng, n) for _ in range(layers)])
    cp = np.stack([_any(rng, n) for _ in range(max(layers - 1, 1))])
    m = layers // 2
    ons, onn, cps = on.copy(), on.copy(), cp.copy()
    ons[m] = _singular(on[m])
    onn[m] = _with_nan(on[m])
    cps[max(m - 1, 0)] = 0.0
    return _up(np.stack([on, ons, onn])), _up(np.stack([cp, cps, cp])), _up(np.stack([_any(rng, n)] * 3))


def _solve_args(n, layers, points):
    """Arguments of the device solves, and the statuses they should report.  One point in
    seven has a failed lead; a one-layer singular device has its contacts off."""
    rng = np.random.default_rng(3 * n + layers)
    on, cp, v = _device(n, layers, rng)
    if layers == 1:
        v = v.clone()
        v[SINGULAR] = 0.0
    k = _kinds(points, [SINGULAR, NAN])
    om, eta, ki = _omegas(k)
    lead = (_up(_herm(rng, n)), _up(_any(rng, n)))
    g = engine.sgf_sr(*lead, None, om, torch.full_like(om, ETA))["g"]
    lst = torch.zeros(points, dtype=torch.int32, device="cuda")
    lst[5::7] = _lib.MAXITER
    want = [int(b) or EXPECTED[int(a)] for a, b in zip(k, lst.tolist())]
    return (on, cp if layers > 1 else None, layers, v, v, g, g, om, eta, ki, lst), want


def _good(args, want):
    """The arguments at the good points only, and their indices."""
    i = torch.as_tensor(np.nonzero(np.array(want) == 0)[0], device="cuda")
    on, cp, layers, vl, vr, gl, gr, om, eta, ki, lst = args
    return (on, cp, layers, vl, vr, gl[i], gr[i], om[i], eta[i], ki[i], lst[i]), i


@pytest.mark.parametrize("solve", ["f64", "mixed", "refined"])
@pytest.mark.parametrize("layers", [1, 3])
@pytest.mark.parametrize("n,points", [(n, _points(n)) for n in ORDERS] + [(16, 500), (105, 140), (120, 330), (192, 160)])
def test_device_solve(solve, layers, n, points):
    args, want = _solve_args(n, layers, points)
    run = {"f64": engine.rgf_transmission, "mixed": lambda *a: engine.rgf_transmission(*a, precision="mixed"),
           "refined": engine.rgf_transmission_refine64}[solve]
    out = run(*args)
    assert out[1].tolist() == want
    assert bool(torch.isnan(out[0][torch.as_tensor(np.array(want) != 0, device="cuda")]).all())
    only, i = _good(args, want)
    ref = run(*only)
    assert int(ref[1].abs().sum()) == 0
    for x, y in zip(out, ref):
        assert torch.equal(x[i], y)


@pytest.mark.parametrize("layers", [1, 3])
@pytest.mark.parametrize("n", [3, 16, 24, 32, 48, 64, 72, 80, 96, 104, 112])
def test_adjoints_and_full_green(n, layers):
    points = 620 if n <= 32 else 330
    args, want = _solve_args(n, layers, points)
    only, i = _good(args, want)
    w = torch.linspace(0.2, 1.0, points, dtype=torch.float64, device="cuda")
    cp = args[1] if layers > 1 else torch.zeros((3, 0, n, n), dtype=torch.complex128, device="cuda")
    full = lambda a, wt: engine.rgf_adjoint(a[0], cp, *a[2:], wt, want_sigma=True, deterministic=True)  # noqa: E731
    t, st, gon, gcp, xl, xr = full(args, w)
    tr, sr, ron, rcp, rl, rr = full(only, w[i])
    assert st.tolist() == want and int(sr.abs().sum()) == 0
    assert torch.equal(t[i], tr) and torch.equal(xl[i], rl) and torch.equal(xr[i], rr)
    assert _near(gon[GOOD], ron[GOOD]) and _near(gcp[GOOD], rcp[GOOD])
    G, _, _, st = engine.device_green(*args)
    R, _, _, sr = engine.device_green(*only)
    assert st.tolist() == want and int(sr.abs().sum()) == 0 and torch.equal(G[i], R)


@pytest.mark.parametrize("n", [3, 16, 24, 32, 48, 72, 96, 104, 112])
def test_surface_gf_adjoint(n):
    points = 620 if n <= 32 else 330
    rng = np.random.default_rng(n)
    h01, v = _up(np.stack([_any(rng, n), np.zeros((n, n))])), _up(np.stack([_any(rng, n)] * 2))
    g = engine.sgf_sr(_up(_herm(rng, n)), h01[0], None, torch.linspace(0.3, 2.1, points, dtype=torch.float64, device="cuda"),
                      torch.full((points,), ETA, dtype=torch.float64, device="cuda"))["g"]
    xs = _up(np.stack([_any(rng, n)] * points))
    ki = torch.zeros(points, dtype=torch.int32, device="cuda")
    lst = torch.zeros_like(ki)
    lst[5::7] = _lib.SINGULAR
    bad = torch.zeros(points, dtype=torch.bool, device="cuda")
    bad[1::3] = True
    xs[bad, n - 1, 0] = float("nan")
    ki[bad] = 1  # the failing points add to another k set
    run = lambda i, **kw: engine.sgf_adjoint(h01, None, v, g[i], xs[i], ki[i], lst[i], deterministic=True, **kw)  # noqa: E731
    r = run(slice(None))
    want = [s or (_lib.NONFINITE if b else 0) for s, b in zip(lst.tolist(), bad.tolist())]
    assert r["status"].tolist() == want
    good = torch.as_tensor(np.nonzero(np.array(want) == 0)[0], device="cuda")
    ref = run(good)
    assert int(ref["status"].abs().sum()) == 0
    for key in ("h00", "h01", "v"):
        assert _near(r[key][0], ref[key][0])
    # the sweep limit: h01 = 0 is done after one doubling
    ki[:] = 0
    ki[::2] = 1
    xs[bad, n - 1, 0] = 0.0
    lst[:] = 0
    st = run(slice(None), maxiter=1)["status"]
    assert st.tolist() == [0 if x else _lib.MAXITER for x in ki.tolist()]


def _batch_system(shape, seed, kind, rng):
    ny, nz = shape
    p, kps = W.spring_network(seed, ny, nz), W.kgrid(3)
    st = W.material_kspace_stack(p, kps, n_layers=1)
    lead = {x: np.array(st[x]) for x in ("d00", "d01", "d10")}
    on, cp = np.repeat(st["onsite"], 3, 1), np.repeat(st["d01"][:, None], 2, 1)
    wmax = W.estimate_omega_max(p, nk=2)
    om, eta = np.array([0.31, 0.57]) * wmax, 1e-6 * wmax * wmax
    if kind == "nan lead":
        lead["d00"][:, -1, 0] = np.nan
    if kind == "huge lead":
        lead["d01"], lead["d10"] = 1e200 * lead["d01"], 1e200 * lead["d10"]
    if kind == "nan device":
        on[:, 1, -1, 0] = np.nan
    if kind == "singular device":
        om, eta = np.array([1.0, 1.0]), 0.05
        for k in range(3):
            on[k, 1] = _singular(on[k, 1])
        cp[:, 0] = 0.0
    return W.Workload(kind, om, kps, lead, lead, on, cp, 3, eta=eta, eta_device=0.0 if kind == "singular device" else None)


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("blocks_per_sm", [1, 2])
def test_batch(precision, blocks_per_sm):
    rng = np.random.default_rng(0)
    kinds = {"good": _lib.OK, "nan lead": _lib.NONFINITE, "huge lead": _lib.UNSTABLE, "nan device": _lib.NONFINITE,
             "singular device": _lib.SINGULAR}
    shapes = [(2, 4), (4, 8), (5, 9), (8, 8)]  # 24, 96, 135, 192
    ws = [_batch_system(s, 50 + i, kind, rng) for i, s in enumerate(shapes) for kind in kinds]
    b = UnevenBatch(ws)
    it = b.items([w.omegas for w in ws], "interleave")
    r = b.solve(it, precision, blocks_per_sm=blocks_per_sm)
    st = r["status"].reshape(len(ws), -1)
    for i, w in enumerate(ws):
        assert st[i].tolist() == [kinds[w.name]] * st.shape[1], (i, w.name)
    t = r["T"].reshape(len(ws), -1)
    only = [w for w in ws if w.name == "good"]
    bg = UnevenBatch(only)
    ref = bg.solve(bg.items([w.omegas for w in only]), precision, blocks_per_sm=blocks_per_sm)["T"].reshape(len(only), -1)
    at = [i for i, w in enumerate(ws) if w.name == "good"]
    assert torch.equal(t[at], ref)
    rest = [i for i in range(len(ws)) if i not in at]
    assert bool(torch.isnan(t[rest]).all())
