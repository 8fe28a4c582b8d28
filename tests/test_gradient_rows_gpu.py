"""The 3D gradient's walk of detector rows where it can go wrong: rows shorter than
a load of four cells, rows that begin on a 16-byte boundary or not, a field that
does not itself begin on one, supports clipped at every edge of the detector, one
and several angles per lane.  Tolerance: the repository's FP32 bar, 1e-5 of the
oracle per parameter entry."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, make_atoms, make_geometry, relerr

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _field(a, shift):
    """a on the device, its first element `shift` floats past a 16-byte boundary."""
    buf = torch.full((a.size + 8,), float("nan"), device="cuda")
    out = buf[shift:shift + a.size].view(a.shape)
    out.copy_(torch.from_numpy(a))
    return out


@pytest.mark.parametrize("D0,D1", [(1, 1), (3, 2), (2, 3), (5, 4), (4, 5), (9, 8), (17, 31),
                                   (16, 32), (15, 33), (20, 44)])
@pytest.mark.parametrize("A,N", [(3, 5), (65, 7)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_gradient_rows(eng, cuda_ready, D0, D1, A, N, shift):
    g = make_geometry("2p5d", A, D0, D1, det_box=0.1 * max(1, min(D0, D1) - 1) / 2)
    I, x, r = make_atoms(3, N, 31 * D0 + D1, rdiag=(2.0, 8.0), roff=2.0,
                         box=0.1 + 0.05 * min(D0, D1))
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    rng = np.random.default_rng(D0 * D1)
    al = rng.normal(size=g.shape).astype(np.float32).astype(np.float64)
    F = _field(al.astype(np.float32), shift)
    _f, G, _ = eng.atom_derivs(atoms, geom, "field", F, order=1)
    want = np.array([go.atom_derivs("field", I[j], x[j], r[j], g, al, 2,
                                    beta=np.ones_like(al))[1] for j in range(N)])
    scale = np.abs(want).max(axis=0)
    assert np.all(np.abs(G.cpu().numpy() - want).max(axis=0) <= TOL * np.maximum(scale, 1e-30))
    # the same bits wherever the field begins, unless rows begin on fours there
    if D1 % 4:
        _f, G0, _ = eng.atom_derivs(atoms, geom, "field", _field(al.astype(np.float32), 0), order=1)
        assert relerr(G.cpu().numpy(), G0.cpu().numpy()) < 2 * TOL


def test_values_beyond_the_cut_off_count_for_nothing_in_fours(eng, cuda_ready):
    g = make_geometry("2p5d", 70, 50, 44)
    I, x, r = make_atoms(3, 6, 9, rdiag=(6.0, 20.0), roff=4.0)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    rng = np.random.default_rng(2)
    out = go.radproj(I, x, r * 0.999, g) == 0.0
    al = rng.normal(size=g.shape).astype(np.float32)
    res = [eng.atom_derivs(atoms, geom, "field", _field(np.where(out, np.float32(bad), al), 0),
                           order=1)[1] for bad in (0.0, np.nan, np.inf)]
    assert torch.equal(res[1], res[0]) and torch.equal(res[2], res[0])
