"""3D binning where a detector has several ranges of tiles: supports across the ranges'
borders, a few wide ones among narrow ones, only wide ones, one atom alone."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, f32, make_geometry, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-5


def mixed_atoms(N, n_wide, seed):
    rng = np.random.default_rng(seed)
    rd = np.where(np.arange(N)[:, None] % max(1, N // max(1, n_wide)) == 0, 0.7, 25.0)
    r = np.concatenate([rd * rng.uniform(0.8, 1.3, (N, 3)), 0.2 * rd * rng.normal(size=(N, 3))], 1)
    return f32(rng.uniform(0.5, 1.5, N)), f32(rng.uniform(-1, 1, (N, 3))), f32(r)


# 40 x 22 tiles of 16 x 32 cells (512 tiles a range, the border inside a row of tiles)
@pytest.mark.parametrize("N,n_wide,D0,D1", [(1, 1, 640, 700), (40, 3, 640, 700), (40, 40, 640, 700),
                                            (300, 20, 640, 700), (70, 5, 33, 8193)])
@pytest.mark.parametrize("form", [1, 2])
def test_ranges_of_tiles(eng, cuda_ready, N, n_wide, D0, D1, form):
    lib = __import__("importlib").import_module("2018_dictionary_tomography_gb300._lib")
    g = make_geometry("2p5d", 2, D0, D1)
    I, x, r = mixed_atoms(N, n_wide, N + n_wide)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    plan = eng.Plan(lib.GR_OP_PROJECT, atoms, geom).set(3, form)
    R = eng.radproj(atoms, geom, plan=plan)
    assert relerr(R.cpu().numpy(), go.radproj_boxed(I, x, r, g)) < TOL


def test_wide_support_on_a_large_detector_is_quick(eng, cuda_ready):
    """Binning and projection of one atom across 2048^2 cells (8192 tiles): 30 to 40 us;
    one thread going through its tiles once per range took 2.3 ms."""
    g = make_geometry("2p5d", 1, 2048)
    atoms, geom = engine_atoms(*mixed_atoms(1, 1, 0)), engine_geometry(g)
    out = torch.empty(geom.shape, device="cuda")
    ms = []
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(4):
            eng.radproj(atoms, geom, out=out)
        b.record()
        b.synchronize()
        ms.append(a.elapsed_time(b) / 4)
    assert min(ms) < 1.0
