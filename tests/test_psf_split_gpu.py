"""The pixel-integrated derivatives in each form of their dispatch: 4, 2 and 1 lanes a
pair in 2D, 8, 16 and 32 pairs a warp in 3D, at the largest number of one form and one
more, with supports of one cell and of many.  Tolerance: the repository's FP32 bar,
1e-5 of the oracle (gradients per parameter entry, Hessians over all atoms)."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import (engine_atoms, engine_geometry, entry_relerr, make_atoms, make_geometry,
                      relerr)

pytestmark = pytest.mark.gpu
TOL = 1e-5
SMS = 152
# the most pairs of one form (2D), the most blocks of 4 atoms (gradients) or of one
# (Hessians) in 3D: (blocks, angles)
LINES = {("2d", 1): ((SMS * 8, 32), (SMS * 16, 32), (1000, 2), (3000, 4)),
         ("2d", 2): ((SMS * 4, 32), (SMS * 8, 32), (1500, 8), (1500, 9), (1500, 16), (1500, 17)),
         ("2p5d", 1): ((SMS * 20 - 1, 3), (SMS * 60 - 1, 3)),
         ("2p5d", 2): ((SMS * 20 - 1, 3), (SMS * 40 - 1, 3))}


@pytest.mark.parametrize("kind,order,blocks,A", [(k, o, b + more, A) for (k, o), bs in LINES.items()
                                                 for b, A in bs for more in (0, 1)])
@pytest.mark.parametrize("D,rdiag", [(24, (3, 6)), (9, (0.6, 1.0)), (33, (20, 40))])
def test_forms(eng, cuda_ready, kind, order, blocks, A, D, rdiag):
    # (2D gradients of 32 angles: four chunks of 8, a quarter of the atoms)
    N = blocks * (4 if order == 1 and A < 8 else 1)
    g = make_geometry(kind, A, D)
    I, x, r = make_atoms(2 if kind == "2d" else 3, N, N + D, rdiag=rdiag, roff=0.2 * rdiag[0])
    C = (go.psf_radproj(I[:1] * 1.1, x[:1], r[:1], g) + 0.001).astype(np.float32).astype(np.float64)
    f, G, H = eng.atom_derivs(engine_atoms(I, x, r), engine_geometry(g), "l2_atom",
                              torch.from_numpy(C).float(), order=order, psf=True)
    pick = np.unique(np.concatenate([np.linspace(0, N - 1, 24).astype(int), [1, 2, 3, N - 2]]))
    out = [go.psf_atom_derivs("l2", I[j], x[j], r[j], g, C, 2) for j in pick]
    assert relerr(f.cpu().numpy()[pick], np.array([o[0] for o in out])) < TOL
    assert entry_relerr(G.cpu().numpy()[pick], np.array([o[1] for o in out])) < TOL
    if order == 2:
        # (the same atoms alone, in the form for few blocks)
        few = eng.atom_derivs(engine_atoms(I[pick], x[pick], r[pick]), engine_geometry(g), "l2_atom",
                              torch.from_numpy(C).float(), order=2, psf=True)[2]
        assert relerr(H.cpu().numpy()[pick], few.cpu().numpy()) < TOL
        # (supports inside one cell: Hessians that cancel beyond FP32)
        if rdiag[1] < 10:
            assert relerr(H.cpu().numpy()[pick], np.array([o[2] for o in out])) < TOL


@pytest.mark.parametrize("N,A,D", [(3, 3071, 64), (3, 3072, 64), (40, 6143, 20), (40, 6144, 20),
                                   (97, 3103, 50), (97, 3104, 50), (300, 6144, 33)])
def test_forward_with_one_warp_a_tile(eng, cuda_ready, N, A, D):
    """2D: the least tiles of the one-warp form for few atoms and for 97, and one angle less."""
    g = make_geometry("2d", A, D)
    I, x, r = make_atoms(2, N, N + D, rdiag=(2, 8), roff=0.5)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    ref = go.psf_radproj(I, x, r, g)
    R = eng.radproj(atoms, geom, psf=True)
    assert relerr(R.cpu().numpy(), ref) < TOL
    data = torch.from_numpy(1.1 * ref + 0.01 * ref.max()).float().cuda()
    fw = eng.fit_forward(atoms, geom, data, "l2", psf=True)
    assert torch.equal(fw["alpha"], R - data)
    want = 0.5 * (fw["alpha"].double() ** 2).sum().item()
    assert abs(float(fw["loss"]) - want) < 1e-6 * want


@pytest.mark.parametrize("D", [20, 31, 33, 65])
@pytest.mark.parametrize("N", [1, 40])
def test_forward_of_wide_and_narrow_atoms(eng, cuda_ready, N, D):
    """2D: atoms that meet from a few cells of a tile to all of them, about the 20 from which they
    take a lane a cell."""
    g = make_geometry("2d", 7, D)
    rng = np.random.default_rng(N + D)
    step = 3.0 / (D - 1)
    rd = 2.0 / (step * np.exp(rng.uniform(np.log(3), np.log(45), (N, 1))))
    I, x, _r = make_atoms(2, N, N + D)
    r = np.concatenate([rd, rd * rng.uniform(0.8, 1.25, (N, 1)), 0.1 * rd], 1)
    r = r.astype(np.float32).astype(np.float64)
    R = eng.radproj(engine_atoms(I, x, r), engine_geometry(g), psf=True)
    assert relerr(R.cpu().numpy(), go.psf_radproj(I, x, r, g)) < TOL
