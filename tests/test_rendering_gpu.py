"""The 3D point-sampled rendering around its tiles' edges, atom counts around one
and several staging passes, and grids that run backwards, against the FP64 oracle
to the repository's FP32 bar, 1e-5."""
import importlib

import numpy as np
import pytest

from oracle import gauss_oracle as go
from problems import engine_atoms, make_atoms, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-5
vol = importlib.import_module("2018_dictionary_tomography_gb300.volume")


@pytest.mark.parametrize("n,N", [((1, 1, 1), 40), ((8, 16, 16), 256), ((7, 15, 17), 257),
                                 ((9, 17, 33), 600), ((25, 4, 40), 40),
                                 # grids that give a lane 2, 4 and 8 voxels
                                 ((9, 130, 129), 40), ((19, 130, 129), 40), ((21, 161, 176), 40)])
@pytest.mark.parametrize("iso", [False, True])
@pytest.mark.parametrize("back", [False, True])
def test_rendering(eng, cuda_ready, n, N, iso, back):
    I, x, r = make_atoms(3, N, N, iso=iso, rdiag=(2, 9))
    coords = [np.linspace(-1, 1, k).astype(np.float32).astype(np.float64) if k > 1
              else np.array([0.125]) for k in n]
    if back:
        coords = [c[::-1].copy() for c in coords]
    u = vol.volproj(engine_atoms(I, x, r), coords).cpu().numpy()
    ref = go.volproj(I, x, r, coords)
    assert relerr(u, ref) < TOL
