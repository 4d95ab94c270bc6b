"""Host-side shortcuts of the calls: one upload of several blocks, vectorised
acceptance of the eta ladder, one resolution of a lead shared by both sides."""

import numpy as np
import pytest
import torch

from negfpy_b200 import engine, negf
from negfpy_b200.types import Device1D, LeadBlocks


@pytest.mark.parametrize("big", [3, 200])
def test_upload_equals_separate_conversions(big):
    rng = np.random.default_rng(0)
    arrays = [rng.standard_normal((2, 3, 3)), None, rng.standard_normal((1, big, big)) * 1j,
              np.arange(8, dtype=np.int32).reshape(2, 4)[:, ::2], torch.ones((2, 2), dtype=torch.float64),
              [[1.0, 2.0], [3.0, 4.0]], rng.standard_normal((4, 4)).astype(np.complex64).T]
    for a, t in zip(arrays, engine._upload(arrays, torch.device("cpu"))):
        if a is None:
            assert t is None
            continue
        ref = engine._c(a, torch.device("cpu"))
        assert t.dtype == torch.complex128 and t.is_contiguous() and t.shape == ref.shape and torch.equal(t, ref)


@pytest.mark.parametrize("limit", [None, 2.0])
def test_accepted_is_classify(limit):
    t = np.array([0.5, -0.5, -1e-12, np.nan, np.inf, 3.0, 1.0, -0.0, np.nan])
    st = np.array([0, 0, 0, 0, 0, 0, 3, 0, -1], dtype=np.int32)
    ref = [negf._classify(a, b, limit, 1e-10) is None for a, b in zip(t, st)]
    assert negf._accepted(t, st, limit, 1e-10).tolist() == ref


def test_a_shared_lead_gives_the_same_system():
    rng = np.random.default_rng(1)
    d = rng.standard_normal((3, 3))
    blocks = lambda: LeadBlocks(d00=d + d.T, d01=0.3 * d, d10=0.3 * d.T)  # noqa: E731
    dev = Device1D([d + d.T] * 2, [0.3 * d])
    one = blocks()
    a = negf.point_system(0.7, dev, one, one, 1e-3, omega_scale=2.0)
    b = negf.point_system(0.7, dev, one, blocks(), 1e-3, omega_scale=2.0)
    assert negf._same_lead(a["lead_l"], a["lead_r"]) and negf._same_lead(b["lead_l"], b["lead_r"])
    for key in ("vl", "vr", "onsite", "coupling"):
        assert np.array_equal(a[key], b[key])


@pytest.mark.parametrize("bad", ["object", ">f8", "longdouble", "clongdouble", "datetime64[s]", "U8", "reversed"])
@pytest.mark.parametrize("size", [3, 200])
def test_upload_refuses_what_a_conversion_refuses(bad, size):
    a = np.arange(float(size * size)).reshape(size, size)
    a = a[::-1] if bad == "reversed" else a.astype(bad)
    with pytest.raises((TypeError, ValueError)) as ref:
        engine._c(a, torch.device("cpu"))
    with pytest.raises(ref.type):
        engine._upload([np.ones((2, 2)), a], torch.device("cpu"))
