"""The 2D projection where it can go wrong: detectors around a tile's edges (the
order in which a launch takes the tiles must reach each once), atom counts around
each variant's line and each pass's list, intensities of both signs.  Against the
FP64 oracle to the repository's FP32 bar, 1e-5."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, make_atoms, make_geometry, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("D0", [2, 31, 32, 33, 65, 96, 300])
@pytest.mark.parametrize("N", [1, 255, 256, 1023, 1024, 1100])
def test_project1d(eng, cuda_ready, D0, N):
    g = make_geometry("2d", 5, D0)
    I, x, r = make_atoms(2, N, D0 + N, rdiag=(2.0, 12.0), roff=1.0, box=0.9)
    I[::3] *= -1
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    ref = go.radproj(I, x, r, g)
    size = go.radproj(np.abs(I), x, r, g).max()   # (terms of both signs cancel)
    R = eng.radproj(atoms, geom)
    assert np.abs(R.cpu().numpy() - ref).max() <= TOL * size   # (0 = 0 off the detector)
    data = torch.from_numpy(ref + 0.1 * size).float().cuda()
    fw = eng.fit_forward(atoms, geom, data, "l2")
    assert torch.equal(fw["alpha"], R - data)
    want = 0.5 * (fw["alpha"].double() ** 2).sum().item()
    # a cell's term rounds twice, and 5 ceil(D0 / 32) tiles of at most 32 positive
    # terms are summed in float32 before float64
    assert abs(float(fw["loss"]) - want) <= 40 * 2.0 ** -24 * want
