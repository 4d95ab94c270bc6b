"""Workspace of the kernels that keep matrices of every layer (adjoint, full G)
at orders up to 32: four blocks an SM while that fits 512 MiB, else two; results
on both sides of the line."""

import numpy as np
import pytest
import torch

from negfpy_b200 import _lib, engine

pytestmark = pytest.mark.gpu
LINE = 512 << 20


def _needs(n, layers):
    """(query, bytes of two blocks an SM) of the adjoint and of the full G."""
    lib = _lib.load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    np_ = next(p for p in (16, 24, 32) if n <= p)
    sigma = 2 * n * n
    for query, mats in ((lib.negf_adjoint_workspace_bytes, 11 + 2 * layers),
                        (lib.negf_device_green_workspace_bytes, 1 + 3 * layers)):
        yield int(query(n, n, n, layers)), 256 + 2 * sms * (mats * np_ * np_ + sigma) * 16


@pytest.mark.parametrize("n", [3, 16, 20, 24, 30, 32])
@pytest.mark.parametrize("layers", [1, 18, 30, 60, 100, 300])
def test_workspace_is_bounded(n, layers):
    for need, two in _needs(n, layers):
        assert need == 2 * (two - 256) + 256 if 2 * (two - 256) <= LINE else need == two


@pytest.mark.parametrize("n,layers", [(32, 17), (32, 24), (20, 48)])
def test_results_on_both_sides(n, layers):
    """More points than two blocks an SM hold: equal points are bitwise equal, and
    T and G_{0,L-1} those of the device solve to 1e-10."""
    rng = np.random.default_rng(n + layers)
    a = rng.standard_normal((2, layers, n, n)) + 1j * rng.standard_normal((2, layers, n, n))
    on = (a[0] + a[0].conj().swapaxes(-1, -2)) / (2 * np.sqrt(n)) + 2 * np.eye(n)
    up = lambda x: torch.as_tensor(np.ascontiguousarray(x[None]), device="cuda")  # noqa: E731
    on, cp, v = up(on), up(0.4 * a[1, 1:] / np.sqrt(n)), up(0.4 * a[1, 0] / np.sqrt(n))
    points, distinct = 320, 4
    om = torch.tensor(np.resize([0.8, 1.1, 1.4, 1.7], points), device="cuda")
    eta = torch.full_like(om, 0.05)
    ki = torch.zeros(points, dtype=torch.int32, device="cuda")
    g = engine.sgf_sr(on[:, 0].contiguous(), v, None, om, eta, ki)["g"]
    args = (on, cp, layers, v[0][None], v[0][None], g, g, om, eta, ki, None)
    t, st = engine.rgf_transmission(*args)
    ta, sa, _, _, xl, xr = engine.rgf_adjoint(*args, torch.ones_like(om), want_sigma=True, deterministic=True)
    gg, _, _, sg = engine.device_green(*args)
    assert int(st.abs().sum()) == 0 and int(sa.abs().sum()) == 0 and int(sg.abs().sum()) == 0
    assert float(((ta - t).abs() / t.abs().clamp(min=1.0)).max()) <= 1e-10
    for x in (ta, xl, xr, gg):
        for i in range(distinct):
            same = x[i::distinct]
            assert torch.equal(same, same[:1].expand_as(same))
    s = v[0] @ g[0] @ v[0].mH
    gam = 1j * (s - s.mH)
    g0 = gg[0, :n, -n:]
    tr = torch.trace(gam @ g0 @ gam @ g0.mH).real
    assert float((tr - t[0]).abs()) <= 1e-10 * max(1.0, abs(float(t[0])))
