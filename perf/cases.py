"""Measured cases of the per-(omega, k) phonon NEGF path.

Every case goes through a public entry point of ``negfpy_b200`` on a seeded
spring network (3 degrees of freedom per atom, ``ny * nz`` atoms in a
principal layer), with eta = 1e-6 omega_max^2, and returns what the call
returns.  ``exact`` restates the same quantities in plain torch, complex128.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from negfpy_b200 import adjoint, batch, dos, models, negf, spectrum, workloads

SWEEPS = 17  # doubling sweeps of a decimation at eta = 1e-6 omega_max^2 (mean of the benchmark grid)


def listed():
    return [
        # One (omega, k) point through negfpy's scalar call (its unit of work): graphene's size in the
        # studies, n = 24, 40 layers.  Latency and launches.
        dict(name="point_n24", kind="point", ny=2, nz=4, ky=1, kz=0, omegas=1, layers=40, disorder=False,
             contacts="matched", precision="f64"),
        # The monatomic chain of the first benchmark configuration: 1000 omega, 8 layers.
        dict(name="chain_1000", kind="chain", omegas=1000, layers=8),
        # One omega of an adaptive k average at silicon's size: n = 12, 30 layers, 18 x 18 k.
        dict(name="kavg_n12", kind="kavg", ny=2, nz=2, ky=18, kz=18, omegas=1, layers=30, disorder=False,
             contacts="matched", precision="f64"),
        # A transmission spectrum at TaN's size, n = 24, 30 layers with mass disorder (every layer its own blocks).
        dict(name="grid_n24", kind="grid", ny=2, nz=4, ky=12, kz=12, omegas=64, layers=30, disorder=True,
             contacts="matched", precision="f64"),
        # A thin sheet between interface contacts (two different leads), n = 45: an odd order of the studies' kind.
        dict(name="sheet_n45", kind="grid", ny=3, nz=5, ky=20, kz=0, omegas=120, layers=2, disorder=False,
             contacts="interface", precision="f64"),
        # The benchmark's slab, n = 48, 20 layers, 64 k, on a part of its omega grid.
        dict(name="slab_n48", kind="grid", ny=2, nz=8, ky=64, kz=0, omegas=256, layers=20, disorder=False,
             contacts="matched", precision="f64"),
        # The bulk configuration, n = 96, 40 layers, 2D k grid.
        dict(name="bulk_n96", kind="grid", ny=4, nz=8, ky=8, kz=8, omegas=32, layers=40, disorder=False,
             contacts="matched", precision="f64"),
        # Reduced precision with refinement, n = 48.
        dict(name="refined_n48", kind="grid", ny=2, nz=8, ky=16, kz=0, omegas=128, layers=20, disorder=False,
             contacts="matched", precision="refined"),
        # Surface DOS spectrum of one lead over a k line, n = 48.
        dict(name="dos_n48", kind="dos", ny=2, nz=8, ky=16, kz=0, omegas=64, layers=1, disorder=False,
             contacts="matched", precision="f64"),
        # The whole device Green's function of one point, n = 36, 20 layers.
        dict(name="green_n36", kind="green", ny=2, nz=6, ky=1, kz=0, omegas=1, layers=20, disorder=True,
             contacts="matched", precision="f64"),
        # T and its gradient in all eight block tensors, n = 72, 30 disordered layers (a differentiation step).
        dict(name="grad_n72", kind="grad", ny=4, nz=6, ky=8, kz=0, omegas=96, layers=30, disorder=True,
             contacts="matched", precision="f64"),
        # Many systems of different orders (24 .. 192), lengths and k lines in one launch.
        dict(name="batch_uneven", kind="batch", systems=12, omegas=4, kmax=32, lmin=10, lmax=40, precision="f64"),
    ]


_SHAPES = [(1, 1), (1, 2), (2, 2), (1, 5), (1, 7), (2, 4), (3, 3), (2, 5), (3, 4), (2, 7), (3, 5), (2, 8), (4, 4),
           (3, 6), (4, 5), (3, 7), (4, 6), (5, 5), (4, 7), (5, 6), (4, 8), (5, 7), (5, 8)]


def draw(rng):
    """One more case: kinds by use, orders 3 .. 120 (odd ones among them), sizes spread over their logarithm."""
    def loguni(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    top = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["point", "chain", "kavg", "grid", "grid", "grid", "dos", "green", "grad", "batch"])
        if kind == "chain":
            return dict(kind="chain", omegas=loguni(16, 20000), layers=loguni(1, 64))
        if kind == "batch":
            c = dict(kind="batch", systems=rng.randint(2, 24), omegas=loguni(1, 8), kmax=loguni(1, 48),
                     lmin=loguni(1, 10), lmax=loguni(11, 60), precision=rng.choice(["f64", "f64", "mixed"]))
        else:
            ny, nz = rng.choice(_SHAPES)
            kz = rng.choice([0, 0, loguni(1, 16)])
            c = dict(kind=kind, ny=ny, nz=nz, ky=loguni(1, 64 if kz == 0 else 16), kz=kz, omegas=loguni(1, 512),
                     layers=loguni(1, 60), disorder=rng.random() < 0.4, contacts="matched", precision="f64")
            if kind in ("point", "kavg", "green"):
                c["omegas"] = 1
            if kind in ("point", "green"):
                c["ky"], c["kz"] = 1, 0
            if kind == "green":
                c["layers"] = min(c["layers"], 24)
            if kind == "dos":
                c["layers"], c["disorder"] = 1, False
                c["omegas"] = min(c["omegas"], max(1, 2048 // (c["ky"] * max(c["kz"], 1))))
            if kind == "grad":
                c["kz"], c["layers"], c["ky"] = 0, max(2, min(c["layers"], 30)), min(c["ky"], 16)
            if kind == "grid":
                c["contacts"] = rng.choice(["matched", "matched", "interface"])
                c["precision"] = rng.choice(["f64", "f64", "f64", "mixed", "refined"])
        if work(c)["flops"] <= top:
            return c


# ------------------------------------------------------------------ inputs --
def _n(c):
    return 1 if c["kind"] == "chain" else 3 * c["ny"] * c["nz"]


def _nk(c):
    return c["ky"] * max(c["kz"], 1)


def _systems(c):
    """Order (ny, nz), layers and k points of each system of a batch."""
    shapes = list(workloads.UNEVEN_SHAPES.values())
    m = c["systems"]
    for i in range(m):
        layers = c["lmin"] + (7 * i) % (c["lmax"] - c["lmin"] + 1)
        yield shapes[i % len(shapes)], layers, 1 + (11 * i + 5) % c["kmax"]


def _network(c, seed):
    """Springs, masses, k points, omegas and eta of a case."""
    two_d = c["kz"] > 0
    params = workloads.spring_network(seed, c["ny"], c["nz"], periodic_y=True, periodic_z=two_d)
    kps = workloads.kgrid(c["ky"], c["kz"])
    wmax = workloads.estimate_omega_max(params, nk=2, two_d=two_d)
    rng = np.random.default_rng(seed + 77)
    w = c["omegas"]
    om = (np.arange(w) + rng.uniform(0.3, 0.9)) * (1.05 * wmax / w) if w > 1 else np.array([rng.uniform(0.2, 0.6) * wmax])
    lm = None
    if c["disorder"]:
        lm = np.asarray(params.masses)[None, :] * rng.uniform(0.85, 1.15, size=(c["layers"], params.n_atoms))
    return SimpleNamespace(params=params, kps=kps, om=om, eta=1e-6 * wmax * wmax, lm=lm)


def prepare(case, seed):
    c, s = case, SimpleNamespace(case=case)
    if c["kind"] == "chain":
        rng = np.random.default_rng(seed)
        p = models.ChainParams(float(rng.uniform(0.8, 1.2)), float(rng.uniform(0.8, 1.2)))
        s.p, s.eta = p, 1e-8
        s.om = (np.arange(c["omegas"]) + 0.5) * (models.analytic_band_max(p) / c["omegas"])
        s.device, s.lead = models.device_perfect_chain(c["layers"], p), models.lead_blocks(p)
        return s
    if c["kind"] == "batch":
        wls = []
        for i, ((ny, nz), layers, nk) in enumerate(_systems(c)):
            x = _network(dict(ny=ny, nz=nz, ky=nk, kz=0, omegas=c["omegas"], layers=layers, disorder=False),
                         1000 * seed + i)
            st = models.material_kspace_stack(x.params, x.kps, n_layers=1)
            lead = {k: st[k] for k in ("d00", "d01", "d10")}
            wls.append(workloads.Workload("s%d" % i, x.om, x.kps, lead, lead, st["onsite"], st["d01"][:, None], layers,
                                          eta=x.eta, uniform_layers=True))
        s.wls, s.batch = wls, batch.UnevenBatch(wls)
        s.items = s.batch.items([w.omegas for w in wls])
        return s
    x = _network(c, seed)
    s.x, s.om, s.kps, s.eta = x, x.om, x.kps, x.eta
    if c["kind"] == "grad":
        st = models.material_kspace_stack(x.params, x.kps, layer_masses=x.lm, n_layers=c["layers"])
        up = lambda a: torch.as_tensor(a, device="cuda").contiguous().requires_grad_(True)  # noqa: E731
        s.blocks = [up(a) for a in (st["onsite"], st["coupling"], st["d10"], st["d01"], st["d00"], st["d01"], st["d00"],
                                    st["d01"])]
        w, k = len(x.om), len(x.kps)
        omega = torch.as_tensor(np.repeat(x.om, k), device="cuda")
        ki = torch.arange(k, device="cuda", dtype=torch.int32).repeat(w)
        s.points = adjoint.PointGrid(omega, torch.full_like(omega, x.eta), ki, w, k, c["layers"])
        s.weight = torch.as_tensor(np.random.default_rng(seed + 5).uniform(0.1, 1.0, size=(w, k)), device="cuda")
        return s
    if c["contacts"] == "interface":
        s.lead_l, s.lead_r, s.vl, s.vr = models.interface_contacts(x.params)
    else:
        s.lead_l = s.lead_r = models.material_kspace_lead(x.params)
        s.vl = s.vr = None
    s.device = models.material_kspace_device(c["layers"], x.params, x.lm)
    return s


def run(state):
    s, c = state, state.case
    kind = c["kind"]
    if kind == "chain":
        return spectrum.transmission_grid(s.om, None, s.device, s.lead, s.lead, eta=s.eta)
    if kind == "grid":
        r = spectrum.transmission_grid(s.om, s.kps, s.device, s.lead_l, s.lead_r, eta=s.eta, device_to_lead_left=s.vl,
                                       device_to_lead_right=s.vr, precision=c["precision"])
        return {k: r[k] for k in ("T", "status", "iters_left", "iters_right")}
    if kind == "point":
        return negf.transmission(float(s.om[0]), s.device, s.lead_l, s.lead_r, eta=s.eta, kpar=s.kps[0])
    if kind == "kavg":
        t, info = negf.transmission_kavg_adaptive(float(s.om[0]), s.device, s.lead_l, s.lead_r, s.kps,
                                                  eta_values=(s.eta, 10 * s.eta))
        return {"T": t, "n_success": info["n_success"]}
    if kind == "dos":
        return dos.lead_surface_dos_spectrum(s.om, s.lead_l, kpoints=s.kps, eta=s.eta)
    if kind == "green":
        return negf.device_green_function(float(s.om[0]), s.device, s.lead_l, s.lead_r, eta=s.eta, kpar=s.kps[0])
    if kind == "grad":
        t = adjoint.TransportFunction.apply(*s.blocks, s.points)
        return [t.detach(), *torch.autograd.grad(t, s.blocks, grad_outputs=s.weight)]
    r = s.batch.solve(s.items, c["precision"], blocks_per_sm=2)
    return {k: r[k] for k in ("T", "status", "iters")}


# -------------------------------------------------------------------- work --
def _point_flops(n, layers, leads, solve=True):
    sgf = (SWEEPS * 7 + 1) * 8.0 * n ** 3
    return leads * sgf + ((5 * (layers - 1) + 7) * 8.0 * n ** 3 if solve else 0.0)


def work(case):
    """Operations (8 real per complex multiply-add, an inverse as one product): SWEEPS sweeps of six products and an
    inverse per distinct lead, four products and an inverse per layer; bytes: blocks in, results out."""
    c = case
    if c["kind"] == "batch":
        fl = by = 0.0
        for (ny, nz), layers, nk in _systems(c):
            n = 3 * ny * nz
            fl += c["omegas"] * nk * _point_flops(n, layers, 1)
            by += nk * 5 * n * n * 16 + c["omegas"] * nk * 16
        return {"bytes": by, "flops": fl}
    n = _n(c)
    if c["kind"] == "chain":
        return {"bytes": c["omegas"] * 24.0, "flops": c["omegas"] * _point_flops(1, c["layers"], 1)}
    pts, layers = _nk(c) * c["omegas"], c["layers"]
    m = n * n * 16.0
    blocks = _nk(c) * m * (3 + (2 * layers - 1 if c["disorder"] else 2))
    if c["kind"] == "dos":
        return {"bytes": _nk(c) * 3 * m + pts * 8, "flops": pts * _point_flops(n, 1, 1, solve=False)}
    if c["kind"] == "green":
        return {"bytes": blocks + layers * layers * m, "flops": _point_flops(n, layers, 1) + layers * layers * 8.0 * n ** 3}
    if c["kind"] == "grad":
        # two decimations and the solve; backward: two sweeps, column, row and adjoint blocks, two Stein sums
        back = 14.0 * layers + 2 * (SWEEPS * 4 + 12)
        return {"bytes": 2 * blocks + pts * 8, "flops": pts * (_point_flops(n, layers, 2) + back * 8.0 * n ** 3)}
    leads = 2 if c["contacts"] == "interface" else 1
    return {"bytes": blocks + pts * 16.0, "flops": pts * _point_flops(n, layers, leads)}


# ------------------------------------------------------------------- exact --
def _phase(terms, kps):
    ks = np.array([(tuple(k) + (0.0, 0.0))[:2] for k in kps])
    sh = np.array(list(terms.keys()), dtype=float)
    ph = np.exp(1j * (ks[:, :1] * sh[:, 0] + ks[:, 1:] * sh[:, 1]))
    return np.einsum("kt,tij->kij", ph, np.stack([np.asarray(v, dtype=complex) for v in terms.values()]))


def _blocks(c, x):
    """Lead (d00, d01) pairs, couplings and layer blocks of every k, as CUDA tensors."""
    p = x.params
    m = 1.0 / np.sqrt(np.repeat(np.asarray(p.masses), p.dof_per_atom))
    phi00, phi01 = _phase(p.fc00_terms, x.kps), _phase(p.fc01_terms, x.kps)
    weigh = lambda a, f, b: f[:, None] * a * b[None, :]  # noqa: E731
    d00, d01 = weigh(phi00, m, m), weigh(phi01, m, m)
    lm = np.repeat(np.asarray(p.masses)[None], c["layers"], 0) if x.lm is None else x.lm
    ms = 1.0 / np.sqrt(np.repeat(lm, p.dof_per_atom, axis=1))
    on = np.stack([weigh(phi00, f, f) for f in ms], 1)
    cp = np.stack([weigh(phi01, f, g) for f, g in zip(ms[:-1], ms[1:])], 1) if c["layers"] > 1 else on[:, :0]
    herm = lambda a: np.conj(np.swapaxes(a, -1, -2))  # noqa: E731
    if c["contacts"] == "interface":
        fc10 = {(-a, -b): np.asarray(v, dtype=complex).conj().T for (a, b), v in p.fc01_terms.items()}
        left = weigh(_phase(fc10, x.kps), m, m)
        right = weigh(_phase({(-a, -b): v.T for (a, b), v in fc10.items()}, x.kps), m, m)
        vl, vr = herm(right), right
    else:
        left = right = d01
        vl, vr = herm(d01), d01
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    return [up(a) for a in (on, cp, vl, vr, d00, left, d00, right)]


def _surface(z, d00, d01):
    """(z - eps_s)^-1 by decimation, batched; d10 = d01^H."""
    eye = torch.eye(d00.shape[-1], dtype=d00.dtype, device=d00.device)
    e = es = d00
    al, be = d01, d01.mH
    for _ in range(200):
        g = torch.linalg.inv(z * eye - e)
        ag, bg = al @ g, be @ g
        agb = ag @ be
        es, e = es + agb, e + agb + bg @ al
        al, be = ag @ al, bg @ be
        with torch.no_grad():
            if max(float(al.abs().max()), float(be.abs().max())) < 1e-12:
                break
    return torch.linalg.inv(z * eye - es)


def _solve(z, on, cp, vl, vr, gl, gr, full=False):
    """T of points whose blocks are already per point (on [P, L, n, n]); full: G and both self-energies instead."""
    eye = torch.eye(on.shape[-1], dtype=on.dtype, device=on.device)
    layers = on.shape[1]
    sl, sr = vl @ gl @ vl.mH, vr @ gr @ vr.mH
    if full:
        n, dim = on.shape[-1], layers * on.shape[-1]
        a = z[0, 0, 0] * torch.eye(dim, dtype=on.dtype, device=on.device)
        for i in range(layers):
            a[i * n:(i + 1) * n, i * n:(i + 1) * n] -= on[0, i]
            if i + 1 < layers:
                a[i * n:(i + 1) * n, (i + 1) * n:(i + 2) * n] -= cp[0, i]
                a[(i + 1) * n:(i + 2) * n, i * n:(i + 1) * n] -= cp[0, i].mH
        a[:n, :n] -= sl[0]
        a[-n:, -n:] -= sr[0]
        s1, s2 = torch.zeros_like(a), torch.zeros_like(a)
        s1[:n, :n], s2[-n:, -n:] = sl[0], sr[0]
        return [torch.linalg.inv(a).cpu().numpy(), s1.cpu().numpy(), s2.cpu().numpy()]
    m = z * eye - on[:, 0] - sl
    g = torch.linalg.inv(m - sr if layers == 1 else m)
    g0 = g
    for i in range(1, layers):
        ci = cp[:, i - 1]
        m = z * eye - on[:, i] - ci.mH @ g @ ci
        g = torch.linalg.inv(m - sr if i == layers - 1 else m)
        g0 = g0 @ ci @ g
    gam_l, gam_r = 1j * (sl - sl.mH), 1j * (sr - sr.mH)
    return ((gam_l @ g0 @ gam_r) * g0.conj()).sum((-1, -2)).real


def _zs(om, eta):
    return ((om + 1j * eta) ** 2).to(torch.complex128)[:, None, None]


def _exact_points(om, ki, eta, b, surface_only=False):
    """T (or the DOS) of points in groups that fit the card."""
    on, cp, vl, vr, l0, l1, r0, r1 = b
    n, layers = on.shape[-1], on.shape[1]
    same = torch.equal(l1, r1)
    step = max(1, int((4 << 30) // (16 * n * n * (2 * layers + 12))))
    out = []
    for a in range(0, om.numel(), step):
        w, k = om[a:a + step], ki[a:a + step]
        z = _zs(w, eta)
        gl = _surface(z, l0[k], l1[k])
        if surface_only:
            out.append(w / math.pi * -2.0 * gl.diagonal(dim1=-2, dim2=-1).imag.sum(-1))
            continue
        gr = gl if same else _surface(z, r0[k], r1[k])
        out.append(_solve(z, on[k], cp[k], vl[k], vr[k], gl, gr))
    return torch.cat(out)


def exact(case, seed):
    c = case
    if c["kind"] == "chain":
        s = prepare(case, seed)
        on, cp = 2.0 * s.p.spring / s.p.mass, -s.p.spring / s.p.mass
        full = lambda v, *shape: torch.full(shape, v, dtype=torch.complex128, device="cuda")  # noqa: E731
        layers = c["layers"]
        b = [full(on, 1, layers, 1, 1), full(cp, 1, layers - 1, 1, 1)] + [full(v, 1, 1, 1) for v in (cp, cp, on, cp, on, cp)]
        om = torch.as_tensor(s.om, device="cuda")
        t = _exact_points(om, torch.zeros(om.numel(), dtype=torch.int64, device="cuda"), s.eta, b)
        return {"T": t.cpu().numpy()[:, None], "status": None, "iters_left": None, "iters_right": None}
    if c["kind"] == "batch":
        out = []
        for i, ((ny, nz), layers, nk) in enumerate(_systems(c)):
            d = dict(ny=ny, nz=nz, ky=nk, kz=0, omegas=c["omegas"], layers=layers, disorder=False, contacts="matched")
            x = _network(d, 1000 * seed + i)
            om = torch.as_tensor(np.repeat(x.om, nk), device="cuda")
            out.append(_exact_points(om, torch.arange(nk, device="cuda").repeat(len(x.om)), x.eta, _blocks(d, x)))
        return {"T": torch.cat(out), "status": None, "iters": None}
    x = _network(c, seed)
    b = _blocks(c, x)
    nk, nw = len(x.kps), len(x.om)
    om = torch.as_tensor(np.repeat(x.om, nk), device="cuda")
    ki = torch.arange(nk, device="cuda").repeat(nw)
    if c["kind"] == "green":
        z = _zs(om, x.eta)
        gl = _surface(z, b[4], b[5])
        gr = _surface(z, b[6], b[7])
        return _solve(z, b[0], b[1], b[2], b[3], gl, gr, full=True)
    if c["kind"] == "grad":
        weight = torch.as_tensor(np.random.default_rng(seed + 5).uniform(0.1, 1.0, size=(nw, nk)), device="cuda").reshape(-1)
        n, layers = b[0].shape[-1], c["layers"]
        step = max(1, int((20 << 30) // (16 * n * n * (12 * layers + 450))))
        leaves = [t.clone().requires_grad_(True) for t in b]
        ts, grads = [], [torch.zeros_like(t) for t in b]
        for a in range(0, om.numel(), step):
            on, cp, vl, vr, l0, l1, r0, r1 = leaves
            k, z = ki[a:a + step], _zs(om[a:a + step], x.eta)
            t = _solve(z, on[k], cp[k], vl[k], vr[k], _surface(z, l0[k], l1[k]), _surface(z, r0[k], r1[k]))
            for acc, g in zip(grads, torch.autograd.grad(t, leaves, grad_outputs=weight[a:a + step])):
                acc += g
            ts.append(t.detach())
        return [torch.cat(ts).reshape(nw, nk), *grads]
    t = _exact_points(om, ki, x.eta, b, surface_only=c["kind"] == "dos")
    if c["kind"] == "dos":
        return t.reshape(nw, nk).mean(1).cpu().numpy()
    if c["kind"] == "point":
        return float(t[0])
    if c["kind"] == "kavg":
        return {"T": float(t.mean()), "n_success": None}
    return {"T": t.reshape(nw, nk).cpu().numpy(), "status": None, "iters_left": None, "iters_right": None}
