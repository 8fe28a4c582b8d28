"""Hessians where a lane walks its own pair (boxes of at most 24 cells in 2D, 8 x 8 in 3D)
and where groups of lanes do: box widths on both sides of the line, warps of mixed widths,
and in 2D the groups of 2, 4 and 8 lanes.  Tolerance: 1e-5 of the oracle, Hessians per
atom normwise (l2_atom: over all atoms)."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import (atom_normwise_relerr, engine_atoms, engine_geometry, entry_relerr, f32,
                      make_geometry, relerr)

pytestmark = pytest.mark.gpu
TOL = 1e-5


def check(eng, g, I, x, r, mode, beta):
    rng = np.random.default_rng(1)
    C = f32(rng.uniform(0.5, 1.5, g.shape))
    B = f32(rng.uniform(0.5, 1.5, g.shape)) if beta else np.ones(g.shape)
    dev = lambda a: torch.from_numpy(a).float().cuda()
    _f, G, H = eng.atom_derivs(engine_atoms(I, x, r), engine_geometry(g), mode, dev(C),
                               dev(B) if beta else None, 1.0, order=2)
    pick = np.unique(np.linspace(0, len(I) - 1, 10).astype(int))
    kind = "l2" if mode == "l2_atom" else "field"
    out = [go.atom_derivs(kind, I[j], x[j], r[j], g, C, 2, beta=B) for j in pick]
    assert entry_relerr(G.cpu().numpy()[pick], np.array([o[1] for o in out])) < TOL
    # (a single atom's residual I E - C cancels in FP32 for some atoms: l2_atom over all)
    err = relerr if mode == "l2_atom" else atom_normwise_relerr
    assert err(H.cpu().numpy()[pick], np.array([o[2] for o in out])) < TOL


@pytest.mark.parametrize("mode,beta", [("field", False), ("field", True), ("l2_atom", False)])
@pytest.mark.parametrize("kind,D,cells", [("2d", 96, (22, 26)), ("2d", 40, (5, 9)), ("2d", 25, (30, 60)),
                                          ("2p5d", 40, (6, 10)), ("2p5d", 40, (4, 6)),
                                          ("2p5d", 9, (9, 14)), ("2p5d", 40, (3, 14))])
def test_widths_around_the_line(eng, cuda_ready, kind, D, cells, mode, beta):
    N, A = 600, 70                     # (42000 pairs: a lane sets up one pair each)
    g = make_geometry(kind, A, D)
    dim = 2 if kind == "2d" else 3
    rng = np.random.default_rng(D + cells[0])
    step = 3.0 / (D - 1)
    rd = 2.0 / (step * rng.uniform(*cells, (N, 1)))   # a support 2 / r wide
    r = np.concatenate([np.repeat(rd, dim, 1), 0.1 * rd * rng.normal(size=(N, 1 if dim == 2 else 3))], 1)
    check(eng, g, f32(rng.uniform(0.5, 1.5, N)), f32(rng.uniform(-1.2, 1.2, (N, dim))), f32(r), mode, beta)


@pytest.mark.parametrize("mode,beta", [("field", False), ("field", True), ("l2_atom", False)])
@pytest.mark.parametrize("N", [3, 60, 120, 250, 500])
def test_groups_of_every_width_2d(eng, cuda_ready, N, mode, beta):
    """100 angles: 8, 8, 4, 2 and 1 lanes' worth of pairs."""
    g = make_geometry("2d", 100, 130)
    rng = np.random.default_rng(N)
    rd = np.exp(rng.uniform(np.log(1.0), np.log(12), (N, 1)))
    r = np.concatenate([rd, rd, 0.2 * rd * rng.normal(size=(N, 1))], 1)
    check(eng, g, f32(rng.uniform(0.5, 1.5, N)), f32(rng.uniform(-1, 1, (N, 2))), f32(r), mode, beta)
