"""The tuning keys that are accepted without effect (4, 8 and 9) change no bit."""
import importlib

import pytest
import torch

from problems import engine_atoms, engine_geometry, make_atoms, make_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["2d", "2p5d"])
@pytest.mark.parametrize("key,values", [(4, (0, 1 << 30)), (8, (0, 1)), (9, (1, 4))])
def test_keys_without_effect(eng, cuda_ready, kind, key, values):
    lib = importlib.import_module("2018_dictionary_tomography_gb300._lib")
    g = make_geometry(kind, 70, 50)
    geom = engine_geometry(g)
    atoms = engine_atoms(*make_atoms(2 if kind == "2d" else 3, 200, 5, rdiag=(2, 15)))
    out = []
    for v in values:
        pp = eng.Plan(lib.GR_OP_PROJECT, atoms, geom).set(key, v)
        pd = eng.Plan(lib.GR_OP_DERIVS_2, atoms, geom).set(key, v)
        R = eng.radproj(atoms, geom, plan=pp)
        out.append((R,) + eng.atom_derivs(atoms, geom, "field", R, None, 1.0, order=2, plan=pd))
    assert all(torch.equal(a, b) for a, b in zip(*out))
