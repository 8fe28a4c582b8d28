"""The derivative kernels' cell walks where they can go wrong: detectors of a
few cells (chunks of cells that would run past the end), supports from one
cell to the whole detector, elongated supports, every number of pairs per warp,
every kind of weight field, and field values that are not finite beyond the
cut-off.  Tolerance: the repository's FP32 bar, 1e-5 of the oracle (gradients
per parameter entry, Hessians per atom normwise)."""
import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import (atom_normwise_relerr, engine_atoms, engine_geometry, entry_relerr,
                      make_atoms, make_geometry, relerr)

pytestmark = pytest.mark.gpu
TOL = 1e-5

CASES = [
    # kind, A, D0, D1, N, atoms  (pairs per warp follow from N A)
    ("2d", 3, 2, None, 2, dict(box=0.05, rdiag=(2.0, 3.0), roff=0.3)),
    ("2d", 7, 5, None, 3, dict(box=0.1, rdiag=(0.5, 2.0), roff=0.3)),
    ("2d", 30, 61, None, 40, dict(rdiag=(2.0, 15.0), roff=2.0)),
    ("2d", 60, 37, None, 400, {}),
    ("3d", 4, 2, 3, 2, dict(box=0.05, rdiag=(2.0, 3.0), roff=0.3)),
    ("3d", 6, 7, 5, 3, dict(box=0.1, rdiag=(0.5, 2.0), roff=0.3)),
    ("2p5d", 9, 41, 30, 30, dict(rdiag=(2.0, 10.0), roff=3.0)),
    ("3d", 36, 24, 33, 300, dict(rdiag=(3.0, 9.0))),
    ("3d", 40, 24, 20, 1700, dict(rdiag=(4.0, 9.0), box=0.7)),
]


@pytest.mark.parametrize("kind,A,D0,D1,N,kw", CASES)
@pytest.mark.parametrize("field", ["alpha", "alpha_beta", "l2_atom"])
def test_walk_matches_oracle(eng, cuda_ready, kind, A, D0, D1, N, kw, field):
    if field == "l2_atom" and kind == "2d" and D0 == 2:
        pytest.skip("six residuals I E - C that cancel: any FP32 walk is near 1e-5 there")
    g = make_geometry(kind, A, D0, D1, det_box=0.15 if D0 < 10 else 1.5)
    I, x, r = make_atoms(2 if kind == "2d" else 3, N, 3 * N + D0, **kw)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    rng = np.random.default_rng(N)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    al, be = f32(rng.normal(size=g.shape)), f32(rng.uniform(0.5, 1.5, size=g.shape))
    t = lambda a: torch.from_numpy(a).float().cuda()
    pick = np.linspace(0, N - 1, min(N, 12)).astype(int)
    if field == "l2_atom":
        f, G, H = eng.atom_derivs(atoms, geom, "l2_atom", t(al), order=2)
        out = [go.atom_derivs("l2", I[j], x[j], r[j], g, al, 2) for j in pick]
        fo = np.array([o[0] for o in out])
        assert relerr(f.cpu().numpy()[pick], fo) < TOL
    else:
        beta = be if field == "alpha_beta" else np.ones_like(be)
        f, G, H = eng.atom_derivs(atoms, geom, "field", t(al),
                                  t(be) if field == "alpha_beta" else None, 1.0, order=2)
        out = [go.atom_derivs("field", I[j], x[j], r[j], g, al, 2, beta=beta) for j in pick]
    go_, Ho = np.array([o[1] for o in out]), np.array([o[2] for o in out])
    assert entry_relerr(G.cpu().numpy()[pick], go_) < TOL
    assert atom_normwise_relerr(H.cpu().numpy()[pick], Ho) < TOL
    # the gradient-only kernels
    _f, G1, _ = eng.atom_derivs(atoms, geom, "l2_atom" if field == "l2_atom" else "field", t(al),
                                order=1)
    assert entry_relerr(G1.cpu().numpy()[pick], go_) < TOL


@pytest.mark.parametrize("kind", ["2d", "2p5d"])
@pytest.mark.parametrize("order", [1, 2])
def test_fields_beyond_the_cut_off_count_for_nothing(eng, cuda_ready, kind, order):
    g = make_geometry(kind, 12, 50, 45)
    I, x, r = make_atoms(2 if kind == "2d" else 3, 6, 9, rdiag=(6.0, 20.0), roff=4.0)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    rng = np.random.default_rng(2)
    # cells that no atom of a support 0.1 % wider meets
    out = go.radproj(I, x, r * 0.999, g) == 0.0
    al, be = rng.normal(size=g.shape), rng.uniform(0.5, 1.5, size=g.shape)
    res = []
    for bad in (0.0, np.nan, np.inf):
        t = lambda a: torch.from_numpy(np.where(out, bad, a)).float().cuda()
        res.append(eng.atom_derivs(atoms, geom, "field", t(al), t(be), 0.0, order=order))
    for o in res[1:]:
        assert torch.equal(o[1], res[0][1])
        if order == 2:
            assert torch.equal(o[2], res[0][2])


@pytest.mark.parametrize("kind", ["2d", "2p5d"])
@pytest.mark.parametrize("A", [1, 7, 8, 9, 65, 300])
def test_chunk_sums(eng, cuda_ready, kind, A):
    """Chunk counts around the batches and shared ranges of the finalize sum,
    and the float32 gradients written straight from it."""
    g = make_geometry(kind, A, 40, 30)
    I, x, r = make_atoms(2 if kind == "2d" else 3, 5, A, rdiag=(3.0, 8.0))
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    C = np.random.default_rng(A).normal(size=g.shape).astype(np.float32).astype(np.float64)
    Ct = torch.from_numpy(C).float().cuda()
    ref = [go.atom_derivs("ip", I[j], x[j], r[j], g, C, 2) for j in range(5)]
    for order in (1, 2):
        _f, G, H = eng.atom_derivs(atoms, geom, "inner", Ct, order=order)
        assert entry_relerr(G.cpu().numpy(), np.array([o[1] for o in ref])) < TOL
    assert atom_normwise_relerr(H.cpu().numpy(), np.array([o[2] for o in ref])) < TOL
    _f, G, _H = eng.atom_derivs(atoms, geom, "inner", Ct, order=1)
    gI, gx, gr_ = eng.atom_grads(atoms, geom, Ct)
    d = 2 if kind == "2d" else 3
    assert torch.equal(gI, G[:, 0].float()) and torch.equal(gx, G[:, 1:1 + d].float())
    assert torch.equal(gr_, G[:, 1 + d:].float())


@pytest.mark.parametrize("iso", [False, True])
def test_atoms_from_host_and_float32_gradients(eng, cuda_ready, iso):
    """Atoms from lists, numpy arrays and tensors are the same, and the adjoint
    of float32 parameters is the rounded adjoint of float64 ones."""
    import importlib
    ag = importlib.import_module("2018_dictionary_tomography_gb300.autograd")
    g = make_geometry("2p5d", 9, 30, 26)
    I, x, r = make_atoms(3, 7, 3, iso=iso)
    geom = engine_geometry(g)
    ref = eng.radproj(engine_atoms(I, x, r), geom)
    dev = lambda a, t: torch.tensor(a, dtype=t, device="cuda")
    for v in ((I.tolist(), x.tolist(), r.tolist()), tuple(torch.from_numpy(a) for a in (I, x, r)),
              tuple(dev(a, torch.float64) for a in (I, x, r)),
              tuple(dev(a, torch.float32) for a in (I, x, r))):
        assert torch.equal(eng.radproj(eng.DeviceAtoms(*v), geom), ref)
    G = torch.randn(geom.shape, device="cuda")
    grads = []
    for t in (torch.float32, torch.float64):
        p = [dev(a, t).requires_grad_(True) for a in (I, x, r)]
        grads.append(torch.autograd.grad(ag.project(*p, geom), p, G))
    for a, b in zip(*grads):
        assert a.shape == b.shape and a.dtype == torch.float32 and torch.equal(a, b.float())


@pytest.mark.parametrize("kind", ["2d", "2p5d", "3d"])
def test_supports_off_the_detector(eng, cuda_ready, kind):
    """Atoms beyond each edge of a small detector, supports reaching over it or
    not, some along one axis only: what the oracle counts, and exactly nothing
    where no support meets the detector."""
    dim = 2 if kind == "2d" else 3
    g = make_geometry(kind, 8, 20, 16, det_box=0.5)
    rng = np.random.default_rng(4)
    x = []
    for r0 in (0.45, 0.55, 0.8, 1.5, 3.0):
        for v in list(np.eye(dim)) + list(-np.eye(dim)) + [np.ones(dim), -np.ones(dim)]:
            x.append(r0 * v + 0.05 * rng.normal(size=dim))
    x = np.array(x).astype(np.float32).astype(np.float64)
    N = len(x)
    I, _x, r = make_atoms(dim, N, 5, rdiag=(2.0, 8.0), roff=1.0)
    al = rng.normal(size=g.shape).astype(np.float32).astype(np.float64)
    for order in (1, 2):
        _f, G, H = eng.atom_derivs(engine_atoms(I, x, r), engine_geometry(g), "field",
                                   torch.from_numpy(al).float().cuda(), order=order)
        G = G.cpu().numpy()
        ref = [go.atom_derivs("field", I[j], x[j], r[j], g, al, 2, beta=np.ones_like(al))
               for j in range(N)]
        assert entry_relerr(G, np.array([o[1] for o in ref])) < TOL
        off = np.array([not np.any(go.radproj(I[j:j + 1], x[j:j + 1], r[j:j + 1] * 0.99, g))
                        for j in range(N)])
        # (in 2D every atom here meets the detector at some angle)
        assert off.sum() == 0 if kind == "2d" else 0 < off.sum() < N
        assert not np.any(G[off])
    H = H.cpu().numpy()
    Ho = np.array([o[2] for o in ref])
    assert np.max(np.abs(H - Ho)) <= TOL * np.max(np.abs(Ho)) and not np.any(H[off])
