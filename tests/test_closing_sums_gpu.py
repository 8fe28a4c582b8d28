"""The closing sums over angle chunks: no, one and several threads per value, every
remainder of a batch of partials, blocks of both sizes, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import atom_normwise_relerr, engine_atoms, engine_geometry, entry_relerr, f32, make_atoms, make_geometry

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("kind,order", [("2d", 1), ("2d", 2), ("2p5d", 1), ("2p5d", 2)])
@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 131])
def test_every_number_of_chunks(eng, cuda_ready, kind, order, chunks):
    N = 5
    g = make_geometry(kind, 4 * chunks, 21)
    geom, lib = engine_geometry(g), __import__("importlib").import_module("2018_dictionary_tomography_gb300._lib")
    I, x, r = make_atoms(2 if kind == "2d" else 3, N, chunks)
    atoms = engine_atoms(I, x, r)
    # eight atoms' places and four angles a warp: a chunk every four angles
    plan = eng.Plan(lib.GR_OP_DERIVS_1 if order == 1 else lib.GR_OP_DERIVS_2, atoms, geom)
    plan.set(7, 0).set(6, 0).set(0, 1 << 20).set(1, 1).set(2, 32)
    C = f32(np.random.default_rng(chunks).uniform(0.5, 1.5, g.shape))
    _f, G, H = eng.atom_derivs(atoms, geom, "field", torch.from_numpy(C).float().cuda(), None, 1.0,
                               order=order, plan=plan)
    out = [go.atom_derivs("field", I[j], x[j], r[j], g, C, 2, beta=np.ones(g.shape)) for j in range(N)]
    assert entry_relerr(G.cpu().numpy(), np.array([o[1] for o in out])) < TOL
    if order == 2:
        assert atom_normwise_relerr(H.cpu().numpy(), np.array([o[2] for o in out])) < TOL
