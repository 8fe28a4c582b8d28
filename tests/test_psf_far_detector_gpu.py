"""Pixel-integrated operator on a detector far from the origin: at 10^4, with cells of
1/128, an atom's centre rounded to float32 lies up to a sixteenth of a cell from its
place.  A cell that the atom's support only just reaches counts all the same (sheared
atoms, whose density does not vanish at the support's end)."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, f32, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("kind,first", [("2d", 1e4), ("2d", 3e4), ("2d", 6e4), ("2p5d", 1e4), ("2p5d", 6e4)])
def test_cells_at_the_supports_end(eng, cuda_ready, kind, first):
    D, step, N = 48, 2.0 ** -7, 300
    p0 = first + step * np.arange(D)
    if kind == "2d":
        g = go.Geometry.from_angles([np.full(1, 0.3)], p0)
    else:
        g = go.Geometry.from_angles([np.full(1, 0.3)], p0, step * np.arange(16))
    g = g.cast(np.float32).cast(np.float64)
    geom = engine_geometry(g)
    rng = np.random.default_rng(D)
    dim = 2 if kind == "2d" else 3
    x = np.zeros((N, dim))
    x[:, :2] = np.asarray(g.w0)[0] * (first + step * D * rng.uniform(0, 1, N))[:, None]
    if dim == 3:
        x[:, 2] = step * 16 * rng.uniform(0, 1, N)
    r = np.concatenate([rng.uniform(15, 40, (N, dim)),
                        rng.normal(0, 60, (N, 3 if dim == 3 else 1))], axis=1)
    I, x, r = f32(rng.uniform(0.5, 1.5, N)), f32(x), f32(r)
    atoms = engine_atoms(I, x, r)
    # one atom at a time: a missing cell is not drowned by the others
    C = np.ones(g.shape)
    f, _g, _H = eng.atom_derivs(atoms, geom, "inner", torch.ones(geom.shape, device="cuda"),
                               order=1, psf=True)
    out = [go.psf_atom_derivs("ip", I[j], x[j], r[j], g, C, 1) for j in range(N)]
    assert relerr(f.cpu().numpy(), np.array([o[0] for o in out])) < TOL
    for j in range(0, N, 6):
        R = eng.radproj(engine_atoms(I[j:j + 1], x[j:j + 1], r[j:j + 1]), geom, psf=True)
        assert relerr(R.cpu().numpy(), go.psf_radproj(I[j:j + 1], x[j:j + 1], r[j:j + 1], g)) < TOL, j
