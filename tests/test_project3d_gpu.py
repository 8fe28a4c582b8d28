"""The 3D projection where its layout can go wrong: detectors smaller than a
tile and a subtile, ragged edges, more atoms in a tile than a pass (256) or a
list (1024) holds, very elongated and very wide footprints, and workspaces
that hold the pair records of all, some or no angles (which must not change a
bit).  Tolerance: the repository's FP32 bar, 1e-5 of the oracle normwise."""
import ctypes
import importlib

import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, make_atoms, make_geometry, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-5
PKG = "2018_dictionary_tomography_gb300"


@pytest.mark.parametrize("D0,D1,N,kw", [
    (1, 1, 3, {}),                                          # one cell
    (3, 2, 5, {}),                                          # less than a subtile
    (16, 32, 31, {}),                                       # exactly a tile
    (17, 33, 33, {}),                                       # one cell over
    (37, 95, 300, dict(rdiag=(10.0, 50.0), roff=6.0, box=1.2)),
    (20, 20, 1100, dict(rdiag=(3.0, 6.0), box=0.2)),        # a tile's list in rounds
    (64, 48, 60, dict(rdiag=(1.0, 40.0), roff=15.0)),       # elongated footprints
    (48, 64, 40, dict(iso=True, rdiag=(0.5, 60.0))),        # whole detector to below a cell
])
@pytest.mark.parametrize("form", [1, 2])
def test_project3d_edges(eng, cuda_ready, D0, D1, N, kw, form):
    lib = importlib.import_module(PKG + "._lib")
    g = make_geometry("3d", 6, max(D0, 2), max(D1, 2), det_box=1.5 if D0 > 3 else 0.3)
    if D0 == 1:
        g = go.Geometry.from_angles([np.linspace(0.1, 3.0, 3), np.linspace(-1.0, 1.2, 2)],
                                    np.array([0.1]), np.array([-0.2]))
        g = g.cast(np.float32).cast(np.float64)
    I, x, r = make_atoms(3, N, 7 * N + D0, **kw)
    I[::5] *= -1.0
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    plan = eng.Plan(lib.GR_OP_PROJECT, atoms, geom).set(3, form)
    R = eng.radproj(atoms, geom, plan=plan).cpu().numpy()
    ref = go.radproj(I, x, r, g)
    assert np.abs(ref).max() > 0
    assert relerr(R, ref) < TOL
    assert np.count_nonzero(R[ref == 0]) <= 1e-3 * R.size   # cells on the cut-off alone


def test_project3d_workspace_sizes_agree_bitwise(eng, cuda_ready):
    """Records of all angles, of a range of them at a time, and none."""
    lib = importlib.import_module(PKG + "._lib").load()
    g = make_geometry("2p5d", 13, 50, 70)
    I, x, r = make_atoms(3, 200, 5, rdiag=(8.0, 30.0), roff=4.0, box=1.0)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    data = torch.from_numpy(np.random.default_rng(1).normal(size=g.shape)).float().cuda()
    full = int(lib.gr_workspace_bytes(0, ctypes.byref(atoms.struct), ctypes.byref(geom.struct)))
    row = 200 * 32                       # records of one angle
    least = full - (13 * row + 255) // 256 * 256
    outs = []
    for nb in (full, least + 5 * row, least + row, least):
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        R, alpha = torch.empty_like(data), torch.empty_like(data)
        loss = torch.empty((), dtype=torch.float64, device="cuda")
        eng.fit_forward_into(atoms, geom, data, "l2", 0.0, R, alpha, None, loss, ws)
        outs.append((R, alpha, loss))
    for o in outs[1:]:
        assert torch.equal(o[0], outs[0][0]) and torch.equal(o[1], outs[0][1])
        assert abs(o[2].item() - outs[0][2].item()) <= 1e-12 * abs(outs[0][2].item())
    with pytest.raises(Exception):
        ws = torch.empty(least - 256, dtype=torch.uint8, device="cuda")
        eng.fit_forward_into(atoms, geom, data, "l2", 0.0, outs[0][0], None, None, outs[0][2], ws)
