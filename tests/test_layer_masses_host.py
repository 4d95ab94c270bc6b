"""Per-layer masses of ``models.material_kspace_stack``: the first ``n_layers``
rows count, missing rows are an error."""

import numpy as np
import pytest

from negfpy_b200 import workloads as W
from negfpy_b200.models import MaterialKspaceParams, material_kspace_device, material_kspace_stack

KPTS = [(0.3,), (-1.1,)]


def _one_atom():
    fc00 = {(0, 0): np.array([[3.0]]), (1, 0): np.array([[-0.5]]), (-1, 0): np.array([[-0.5]])}
    return MaterialKspaceParams(masses=np.array([1.0]), fc00_terms=fc00, fc01_terms={(0, 0): np.array([[-1.0]])},
                                dof_per_atom=1)


def _blocks_by_layer(params, masses):
    """onsite and coupling from one mass row at a time."""
    st = material_kspace_stack(params, KPTS)
    rep = lambda m: 1.0 / np.sqrt(np.repeat(m, params.dof_per_atom))  # noqa: E731
    m0 = rep(params.masses)
    phi00, phi01 = (st[x] / m0[:, None] / m0[None, :] for x in ("d00", "d01"))
    ms = [rep(m) for m in masses]
    on = np.stack([a[:, None] * phi00 * a[None, :] for a in ms], 1)
    cp = np.stack([a[:, None] * phi01 * b[None, :] for a, b in zip(ms, ms[1:])], 1)
    return on, cp


@pytest.mark.parametrize("rows", [3, 5])
def test_the_first_n_layers_rows_count(rows):
    params = W.spring_network(4, 1, 2)
    masses = np.random.default_rng(0).uniform(0.8, 1.2, size=(rows, params.n_atoms))
    st = material_kspace_stack(params, KPTS, layer_masses=masses, n_layers=3)
    on, cp = _blocks_by_layer(params, masses[:3])
    n = params.ndof
    assert st["onsite"].shape == (2, 3, n, n) and st["coupling"].shape == (2, 2, n, n)
    assert np.allclose(st["onsite"], on, rtol=1e-13, atol=1e-13)
    assert np.allclose(st["coupling"], cp, rtol=1e-13, atol=1e-13)


def test_missing_rows_are_an_error():
    params = W.spring_network(4, 1, 2)
    with pytest.raises(IndexError):
        material_kspace_stack(params, KPTS, layer_masses=np.ones((2, params.n_atoms)), n_layers=3)


@pytest.mark.parametrize("masses", [None, np.ones((2, 2))])
def test_no_layers_are_an_error(masses):
    with pytest.raises(ValueError):
        material_kspace_stack(W.spring_network(4, 1, 2), KPTS, layer_masses=masses, n_layers=0)


def test_one_mass_per_layer_of_a_one_atom_model():
    masses = np.array([1.0, 2.0, 3.0])
    st = material_kspace_stack(_one_atom(), KPTS, layer_masses=masses, n_layers=3)
    ref = material_kspace_stack(_one_atom(), KPTS, layer_masses=masses[:, None], n_layers=3)
    for key in ("onsite", "coupling"):
        assert np.array_equal(st[key], ref[key])
    dev = material_kspace_device(3, _one_atom(), masses[:, None]).device_builder(KPTS[0])
    assert np.array_equal(np.stack(dev.onsite_blocks), st["onsite"][0])
