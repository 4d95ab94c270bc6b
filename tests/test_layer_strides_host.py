"""Blocks of fewer layers than the call solves are refused before a kernel
could read past them; one block for all layers, and more than needed, are not."""

import numpy as np
import pytest
import torch

from negfpy_b200 import engine
from negfpy_b200.batch import UnevenBatch

K, N = 2, 3


def _blocks(onsite, coupling):
    z = lambda m: torch.zeros((K, m, N, N), dtype=torch.complex128)  # noqa: E731
    return z(onsite), None if coupling is None else z(coupling)


ACCEPTED = [(1, 1, 4), (4, 3, 4), (5, 6, 4), (1, None, 1), (3, 0, 1), (1, 1, 2), (4, 1, 4), (1, 3, 4)]
REFUSED = [(3, 3, 4), (4, 2, 4), (2, 1, 3), (4, 0, 2), (1, 2, 4), (0, 1, 3)]


@pytest.mark.parametrize("onsite,coupling,layers", ACCEPTED)
def test_strides(onsite, coupling, layers):
    on, cp = _blocks(onsite, coupling)
    (on_ks, on_ls), c, (cp_ks, cp_ls) = engine.layer_strides(on, cp, layers)
    assert (on_ks, on_ls) == (onsite * N * N, 0 if onsite == 1 else N * N)
    if layers == 1:
        assert c is None and (cp_ks, cp_ls) == (0, 0)
    else:
        assert c is cp and (cp_ks, cp_ls) == (coupling * N * N, 0 if coupling == 1 else N * N)
    assert engine.layer_strides(on[:1], cp, layers)[0][0] == 0  # one k set serves every k


@pytest.mark.parametrize("onsite,coupling,layers", REFUSED)
def test_too_few_layers_are_refused(onsite, coupling, layers, monkeypatch):
    on, cp = _blocks(onsite, coupling)
    lead = torch.zeros((K, N, N), dtype=torch.complex128)
    with pytest.raises(ValueError, match="n_layers"):
        engine.layer_strides(on, cp, layers)
    with pytest.raises(ValueError, match="n_layers"):
        UnevenBatch._record(engine.StackedSystem((lead,) * 3, (lead,) * 3, on, cp, layers, lead, lead, True), 1e-6, 1e-6)
    monkeypatch.setattr(engine, "_dev", lambda: torch.device("cpu"))
    d = {k: np.zeros((K, N, N)) for k in ("d00", "d01", "d10")}
    with pytest.raises(ValueError, match="n_layers"):
        engine.StackedSystem.from_arrays(d, d, on, cp, layers)
