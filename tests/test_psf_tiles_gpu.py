"""The pixel-integrated kernels where they can go wrong: detectors around a tile's
edges, supports wider than a tile or inside one cell, atom counts around one and
several staging passes, queues of cells from one to many pairs, every number of
pairs per block.  Tolerance: the repository's FP32 bar, 1e-5 of the oracle
(gradients per parameter entry, Hessians per atom normwise)."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import (atom_normwise_relerr, engine_atoms, engine_geometry, entry_relerr,
                      make_atoms, make_geometry, relerr)

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("kind,A,D,N,rdiag", [
    ("2d", 3, 31, 1, (0.6, 1.0)), ("2d", 5, 33, 300, (3, 6)), ("2d", 4, 64, 1100, (3, 8)),
    ("2p5d", 3, 15, 1, (0.6, 1.0)), ("2p5d", 2, 17, 257, (4, 8)), ("3d", 4, 33, 70, (3, 8)),
    ("3d", 4, 48, 129, (5, 9)), ("3d", 4, 16, 40, (40, 60)),
])
def test_pixel_integrated_forward(eng, cuda_ready, kind, A, D, N, rdiag):
    g = make_geometry(kind, A, D)
    I, x, r = make_atoms(2 if kind == "2d" else 3, N, N + D, rdiag=rdiag, roff=0.5)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    ref = go.psf_radproj(I, x, r, g)
    R = eng.radproj(atoms, geom, psf=True)
    assert relerr(R.cpu().numpy(), ref) < TOL
    # the fused loss: positive terms of two roundings each, summed with carries
    data = torch.from_numpy(1.1 * ref + 0.01 * ref.max()).float().cuda()
    fw = eng.fit_forward(atoms, geom, data, "l2", psf=True)
    assert torch.equal(fw["alpha"], R - data)
    want = 0.5 * (fw["alpha"].double() ** 2).sum().item()
    assert abs(float(fw["loss"]) - want) < 1e-6 * want


@pytest.mark.parametrize("kind,A,D,N", [("2d", 3, 31, 1), ("2d", 40, 33, 7), ("2d", 9, 48, 70),
                                        ("2p5d", 3, 15, 1), ("2p5d", 33, 17, 3), ("3d", 9, 20, 40)])
@pytest.mark.parametrize("order", [1, 2])
def test_pixel_integrated_derivatives(eng, cuda_ready, kind, A, D, N, order):
    g = make_geometry(kind, A, D)
    I, x, r = make_atoms(2 if kind == "2d" else 3, N, N + D, rdiag=(3, 6), roff=0.8)
    C = (go.psf_radproj(I[:1] * 1.1, x[:1], r[:1], g) + 0.001).astype(np.float32).astype(np.float64)
    f, G, H = eng.atom_derivs(engine_atoms(I, x, r), engine_geometry(g), "l2_atom",
                              torch.from_numpy(C).float(), order=order, psf=True)
    pick = np.linspace(0, N - 1, min(N, 8)).astype(int)
    out = [go.psf_atom_derivs("l2", I[j], x[j], r[j], g, C, 2) for j in pick]
    assert relerr(f.cpu().numpy()[pick], np.array([o[0] for o in out])) < TOL
    assert entry_relerr(G.cpu().numpy()[pick], np.array([o[1] for o in out])) < TOL
    if order == 2:
        assert atom_normwise_relerr(H.cpu().numpy()[pick], np.array([o[2] for o in out])) < TOL
