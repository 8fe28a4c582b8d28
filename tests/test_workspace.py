"""Workspace sizes of the derivative launches: what gr_workspace_bytes answers holds
the chunk partials of every schedule that launches under it, and a launch refuses less
than its own schedule needs."""
import ctypes
import importlib

import numpy as np
import pytest
import torch

from oracle import gauss_oracle as go
from problems import engine_atoms, engine_geometry, entry_relerr, make_atoms, make_geometry, relerr

LIB = importlib.import_module("2018_dictionary_tomography_gb300._lib")
TOL = 1e-5


def partials_bytes(kdet, n, A, order, atoms_per_warp, split):
    """Bytes of chunk partials under the default tuning, one angle per lane: split
    schedules share a pair among up to 8 lanes where that gives at most 65536."""
    lanes, rs = 32 // atoms_per_warp, 1
    while split and rs < 8 and rs < lanes and n * A * rs * 2 <= 65536:
        rs *= 2
    P = 6 if kdet == 1 else 10
    qn = 1 + P + (P * (P + 1) // 2 if order == 2 else 0)
    return -(-A // (lanes // rs)) * qn * n * 4


def schedules(kdet, n, A, order):
    """(point-sampled, pixel-integrated) partials: one atom a warp for Hessians and
    long series, else four; a 3D point-sampled series is long from 64 angles where they fill
    warps of 32 about as well as eights, or pairs are shared."""
    ag = 1
    while ag < min(n, 4):
        ag *= 2
    one = order == 2 or A >= 1024
    fits = -(-A // 32) * 32 <= -(-A // 8) * 8 * 17 // 16
    one_point = one or (kdet == 2 and A >= 64 and (2 * n * A <= 65536 or fits))
    point = partials_bytes(kdet, n, A, order, 1 if one_point else ag, True)
    pixel = partials_bytes(kdet, n, A, order, 1 if one else ag, False)
    return point, pixel


def host_problem(kdet, n, A, D):
    """Descriptors for host-side checks (their pointers are never followed)."""
    at, g = LIB.GrAtoms(), LIB.GrGeometry()
    at.n_atoms = n
    at.I = at.x = at.r = 256
    g.kdet, g.n_angles, g.frames = kdet, A, 256
    for k in range(kdet):
        g.det[k], g.n_det[k], g.det_inv_step[k] = 256, D, 1.0
    return at, g


@pytest.mark.parametrize("kdet", [1, 2])
@pytest.mark.parametrize("order", [1, 2])
def test_query_covers_both_operators_without_gpu(kdet, order):
    lib = LIB.load()
    for n in (1, 3, 4, 5, 31, 128, 1000, 4096):
        for A in (1, 31, 40, 63, 64, 65, 130, 401, 500, 1023, 1024, 2000):
            need = max(schedules(kdet, n, A, order))
            if need > 1 << 30:
                continue  # (above the one-angle budget: fewer chunks)
            at, g = host_problem(kdet, n, A, 16)
            have = lib.gr_workspace_bytes(LIB.GR_OP_DERIVS_1 if order == 1 else LIB.GR_OP_DERIVS_2,
                                          ctypes.byref(at), ctypes.byref(g))
            assert have >= need, (n, A, have, need)


@pytest.mark.parametrize("n,A", [(128, 401), (1000, 64), (300, 130), (4096, 1023)])
def test_pixel_integrated_gradient_refuses_less_without_gpu(n, A):
    """One byte less than the partials: refused before any launch."""
    lib = LIB.load()
    at, g = host_problem(2, n, A, 16)
    less = schedules(2, n, A, 1)[1] - 1
    rc = lib.gr_psf_atom_derivs(ctypes.byref(at), ctypes.byref(g), LIB.GR_MODE_INNER, 256, None,
                                0.0, 1, 256, 256, None, 256, less, None)
    assert rc == -2, rc  # GR_ERR_WORKSPACE


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["inner", "l2_atom"])
@pytest.mark.parametrize("N,A,order,psf", [(300, 130, 1, True), (600, 64, 1, True),
                                           (20, 130, 1, True), (300, 130, 1, False),
                                           (40, 70, 2, True)])
def test_queried_workspace_is_not_passed(eng, cuda_ready, N, A, order, psf, mode):
    """A workspace of exactly the queried size inside a larger buffer whose tail must
    stay as it was; values against the oracle."""
    g = make_geometry("3d" if A != 70 else "2p5d", A, 9)
    I, x, r = make_atoms(3, N, N + A, rdiag=(2, 4), roff=0.3)
    geom, atoms = engine_geometry(g), engine_atoms(I, x, r)
    fwd = go.psf_radproj if psf else go.radproj
    C = (fwd(I[:1] * 1.1, x[:1], r[:1], g) + 0.001).astype(np.float32).astype(np.float64)
    op = LIB.GR_OP_DERIVS_1 if order == 1 else LIB.GR_OP_DERIVS_2
    need = eng.workspace_bytes(op, atoms, geom)
    whole = torch.full((8 * need + (1 << 20),), 0xA5, dtype=torch.uint8, device="cuda")
    P = atoms.n_params()
    f = torch.zeros(N, dtype=torch.float64, device="cuda")
    G = torch.zeros((N, P), dtype=torch.float64, device="cuda")
    H = torch.zeros((N, P, P), dtype=torch.float64, device="cuda") if order == 2 else None
    eng.atom_derivs_into(atoms, geom, mode, torch.from_numpy(C).float().cuda(), None, 1.0, order,
                         f, G, H, whole[:need], psf=psf)
    torch.cuda.synchronize()
    assert bool((whole[need:] == 0xA5).all())
    derivs = go.psf_atom_derivs if psf else go.atom_derivs
    pick = np.linspace(0, N - 1, min(N, 6)).astype(int)
    out = [derivs({"inner": "ip", "l2_atom": "l2"}[mode], I[j], x[j], r[j], g, C, 2) for j in pick]
    assert relerr(f.cpu().numpy()[pick], np.array([o[0] for o in out])) < TOL
    assert entry_relerr(G.cpu().numpy()[pick], np.array([o[1] for o in out])) < TOL


@pytest.mark.parametrize("n,A,D", [(8192, 20000, 128), (1000000, 64, 64), (40, 60, 32), (8192, 2049, 16)])
def test_records_are_asked_for_where_they_are_used_without_gpu(n, A, D):
    """Up to 512 MB of records of all angles, or of ranges of 32768 items and more."""
    lib = LIB.load()
    at, g = host_problem(2, n, A, D)
    at0, g0 = host_problem(2, n, A, D)
    tiles = -(-D // 16) * -(-D // 32)
    rng = min(A, (512 << 20) // (32 * n))
    want = rng * n * 32 if rng == A or rng * tiles >= 32768 else 0
    have = lib.gr_workspace_bytes(LIB.GR_OP_PROJECT, ctypes.byref(at), ctypes.byref(g))
    least = 256 + 4 * (A * tiles * (-(-n // 32) + 1)) + 12 * A * tiles + 2048   # all but the records
    assert want <= have - least + 4096 and have <= want + least + 4096, (have, want, least)


@pytest.mark.gpu
@pytest.mark.parametrize("angles", [0, 1, 7, 59, 60])
def test_few_records_do_not_split_a_projection(eng, cuda_ready, angles):
    """Room for the records of some angles, too few for the GPU at a time: one launch each of
    binning and projection, the same bits."""
    lib = LIB.load()
    g = make_geometry("2p5d", 60, 64)
    I, x, r = make_atoms(3, 500, 3, rdiag=(4, 20))
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    want = eng.radproj(atoms, geom)
    full = eng.workspace_bytes(LIB.GR_OP_PROJECT, atoms, geom)
    size = full - (60 - angles) * 500 * 32
    ws = torch.empty(full, dtype=torch.uint8, device="cuda")
    R = torch.empty_like(want)
    before = eng.launch_count()
    LIB.check(lib.gr_radproj(ctypes.byref(atoms.struct), ctypes.byref(geom.struct), R.data_ptr(),
                             ws.data_ptr(), size, eng._stream_handle(geom.device)), "gr_radproj")
    assert eng.launch_count() - before == 2
    assert torch.equal(R, want)


@pytest.mark.gpu
@pytest.mark.parametrize("angles,launches", [(32767, 2), (32768, 4), (39999, 4), (40000, 2)])
def test_ranges_of_angles(eng, cuda_ready, angles, launches):
    """A tile an angle: ranges are taken from 32768 items on, and give the same bits."""
    lib = LIB.load()
    A, n = 40000, 9
    g = make_geometry("2p5d", A, 16, 32)
    I, x, r = make_atoms(3, n, 3)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    want = eng.radproj(atoms, geom)
    full = eng.workspace_bytes(LIB.GR_OP_PROJECT, atoms, geom)
    ws = torch.empty(full, dtype=torch.uint8, device="cuda")
    R = torch.empty_like(want)
    before = eng.launch_count()
    LIB.check(lib.gr_radproj(ctypes.byref(atoms.struct), ctypes.byref(geom.struct), R.data_ptr(),
                             ws.data_ptr(), full - (A - angles) * n * 32,
                             eng._stream_handle(geom.device)), "gr_radproj")
    assert eng.launch_count() - before == launches
    assert torch.equal(R, want)


def test_pixel_integrated_forward_asks_for_no_records_without_gpu():
    lib = LIB.load()
    at, g = host_problem(2, 8192, 2000, 64)
    size = lambda op: lib.gr_workspace_bytes(op, ctypes.byref(at), ctypes.byref(g))
    assert size(LIB.GR_OP_PROJECT) - size(LIB.GR_OP_PSF_PROJECT) > 8192 * 2000 * 32 - 4096
    at1, g1 = host_problem(1, 8192, 2000, 64)
    both = [lib.gr_workspace_bytes(op, ctypes.byref(at1), ctypes.byref(g1))
            for op in (LIB.GR_OP_PROJECT, LIB.GR_OP_PSF_PROJECT)]
    assert both[0] == both[1]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["2d", "2p5d"])
def test_pixel_integrated_forward_in_its_own_workspace(eng, cuda_ready, monkeypatch, kind):
    """Projection, fit and a fit step hold no more than the query for them."""
    g = make_geometry(kind, 70, 40)
    I, x, r = make_atoms(2 if kind == "2d" else 3, 300, 3)
    atoms, geom = engine_atoms(I, x, r), engine_geometry(g)
    monkeypatch.setattr(eng, "_workspaces", {})    # (a stream's handle may be an older one's)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        R = eng.radproj(atoms, geom, psf=True)
        eng.fit_forward(atoms, geom, R, "l2", psf=True)
        need = eng.workspace_bytes(LIB.GR_OP_PSF_PROJECT, atoms, geom)
        assert eng.workspace(0, geom.device).numel() == need
    s.synchronize()
    assert relerr(R.cpu().numpy(), go.psf_radproj(I, x, r, g)) < TOL
    derivs = eng.workspace_bytes(LIB.GR_OP_DERIVS_1, atoms, geom)
    step = eng.FitStep(geom, 300, order=1, psf=True)
    assert step.ws.numel() == max(need, derivs)
