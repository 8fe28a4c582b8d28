"""The rounding of the pixel-integrated exponent: the form is scaled by -30 log2 e once.
Bounds: 1.15 times the error of one FP32 evaluation of each point that way, a point at a
time; factors folded into the form's coefficients pass them on these problems."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, make_atoms, make_geometry, relerr

pytestmark = pytest.mark.gpu


def problem(seed):
    """Narrow to wide, sheared atoms."""
    rng = np.random.default_rng(seed)
    A, D, N = int(rng.integers(2, 12)), int(rng.integers(9, 60)), int(rng.integers(1, 60))
    rd = float(np.exp(rng.uniform(np.log(1.0), np.log(30))))
    ro = float(rng.choice([0.1, 0.5, 1.0, 2.0])) * rd
    g = make_geometry(["3d", "2p5d"][seed % 2], A, D)
    I, x, r = make_atoms(3, N, seed, rdiag=(0.7 * rd, 1.4 * rd), roff=ro)
    return g, I, x, r, go.psf_radproj(I, x, r, g)


@pytest.mark.parametrize("seed,bound", [(12, 1.15 * 1.84e-6), (13, 1.15 * 6.46e-7)])
def test_forward(eng, cuda_ready, seed, bound):
    g, I, x, r, ref = problem(seed)
    R = eng.radproj(engine_atoms(I, x, r), engine_geometry(g), psf=True).cpu().numpy()
    assert relerr(R, ref) < bound


@pytest.mark.parametrize("seed,bound", [(35, 1.15 * 6.00e-7), (50, 1.15 * 7.53e-7)])
def test_gradient(eng, cuda_ready, seed, bound):
    g, I, x, r, ref = problem(seed)
    C = (1.1 * ref + 0.001).astype(np.float32).astype(np.float64)
    _f, G, _H = eng.atom_derivs(engine_atoms(I, x, r), engine_geometry(g), "inner",
                                torch.from_numpy(C).float().cuda(), order=1, psf=True)
    n = min(len(I), 5)
    want = np.array([go.psf_atom_derivs("ip", I[j], x[j], r[j], g, C, 1)[1] for j in range(n)])
    assert np.linalg.norm(G.cpu().numpy()[:n] - want) < bound * np.linalg.norm(want)
