"""3D rendering of small grids: edges of the 4 x 8 x 8 tiles and of a warp's voxels, atom
counts around 32 and the block's 256, wide supports (most of 32 atoms reach a warp) and
narrow ones (few do), descending coordinates; against the oracle at the FP32 bar."""
import importlib

import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, f32, make_atoms, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (4, 8, 8), (5, 9, 7), (3, 4, 17), (13, 1, 8), (17, 23, 31)])
@pytest.mark.parametrize("N,rdiag", [(1, (0.6, 1.0)), (31, (1, 2)), (33, (8, 12)), (255, (1, 2)),
                                     (257, (8, 12)), (600, (0.6, 12))])
def test_small_grids(gr, eng, cuda_ready, shape, N, rdiag):
    volume = importlib.import_module("2018_dictionary_tomography_gb300.volume")
    I, x, r = make_atoms(3, N, N, rdiag=rdiag, roff=0.3)
    ys = [f32(np.linspace(-0.9, 0.9, n)) for n in shape]
    ys[1] = ys[1][::-1].copy()
    u = volume.volproj(engine_atoms(I, x, r), [torch.from_numpy(y).float().cuda() for y in ys])
    assert relerr(u.cpu().numpy(), go.volproj(I, x, r, ys)) < 1e-5
