"""Performance cases: what users of the engine have it do, from one atom's
derivatives to a fit step over 20 000 images.

Sizes and value distributions are those of the repository's benchmark
configurations (``workloads.py``): 2D isotropic and anisotropic fits, 3D tilt
series, single-particle images at random orientations, and the served range of
16 to 4096 atoms, 30 to 180 angles and 64 to 512 detector cells a side.

Data sinograms are the projection of isotropic atoms (a sum of separable
terms, so a batched matrix product) at jittered centres, plus noise: a fit of
anisotropic atoms to them has the residual of an early fit.  They are made
without the engine, from the seed alone.

Atoms are float32, so a fit carries losses, gradients and Hessians on in
float32: ``run`` returns them so.
"""
import importlib
import math

import numpy as np
import torch

PKG = "2018_dictionary_tomography_gb300"


def _m(name):
    return importlib.import_module(PKG + "." + name)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the reference's per-atom call with host arrays in and out
        dict(name="dropin_atom_2d", kind="dropin", frames="2d", iso=False, N=1, A=180, D0=256,
             D1=1, box=1.5, fit="l2", order=2),
        # one step of the per-atom descent loop: gradient of one atom and trial of its move
        dict(name="atom_step_2d", kind="atomstep", frames="2d", iso=True, N=64, A=60, D0=128,
             D1=1, box=1.5, fit="l2", order=1),
        # the smallest whole fit step
        dict(name="fit_2d_small", kind="fit", frames="2d", iso=True, N=64, A=60, D0=128, D1=1,
             box=1.5, fit="l2", order=1),
        # an ordinary 2D Newton step with Poisson counts
        dict(name="newton_2d_kl", kind="fit", frames="2d", iso=False, N=512, A=180, D0=256, D1=1,
             box=1.5, fit="kl", order=2),
        # a large served 2D request
        dict(name="newton_2d_wide", kind="fit", frames="2d", iso=True, N=2150, A=153, D0=467,
             D1=1, box=1.5, fit="l2", order=2),
        # a training step through autograd on a tilt series: projection and adjoint
        dict(name="tilt_train", kind="train", frames="tilt", iso=False, N=4096, A=121, D0=256,
             D1=256, box=1.5, fit="l2", order=1),
        # a small 3D Newton step on a wide detector, ragged sizes
        dict(name="newton_3d_small", kind="fit", frames="tilt", iso=False, N=146, A=61, D0=301,
             D1=275, box=1.5, fit="l2", order=2),
        # the largest served 3D Newton step
        dict(name="newton_3d_large", kind="fit", frames="tilt", iso=False, N=2936, A=148, D0=493,
             D1=493, box=1.5, fit="l2", order=2),
        # host arrays in, host results out, as one graph
        dict(name="host_step_3d", kind="host", frames="so3", iso=False, N=1000, A=1001, D0=95,
             D1=95, box=1.0, fit="l2", order=1),
        # single-particle refinement over a whole image set
        dict(name="particles", kind="fit", frames="so3", iso=False, N=8192, A=20000, D0=128,
             D1=128, box=1.0, fit="l2", order=1),
        # the pixel-integrated (single-particle) operator
        dict(name="pixel_integrated", kind="psf", frames="so3", iso=False, N=128, A=401, D0=64,
             D1=64, box=1.0, fit="l2", order=1),
        # rendering the atoms on a voxel grid
        dict(name="render_3d", kind="render", frames="vol", iso=False, N=1000, A=1, D0=128,
             D1=120, box=1.0, fit="l2", order=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "atomstep", "fit2d", "fit2d", "train", "fit3d", "fit3d", "host",
                       "particles", "psf", "render"])
    A, D0 = rng.randint(30, 180), rng.randint(64, 512)
    iso = rng.random() < 0.3
    c = dict(kind=kind, frames="2d", iso=iso, N=_log_int(rng, 16, 4096), A=A, D0=D0, D1=1,
             box=1.5, fit=rng.choice(["l2", "l2", "kl"]), order=rng.choice([1, 2]))
    if kind == "dropin":
        c.update(N=1, order=2, fit="l2")
    elif kind == "atomstep":
        c.update(N=rng.randint(16, 512), order=1, fit="l2")
    elif kind == "fit2d":
        c.update(kind="fit")
    elif kind == "train":
        c.update(frames="tilt", D1=rng.randint(64, 512), fit="l2", order=1)
    elif kind == "fit3d":
        c.update(kind="fit", frames="tilt", D1=rng.randint(64, 512))
    elif kind == "host":
        c.update(frames="so3", N=_log_int(rng, 64, 4096), A=_log_int(rng, 100, 3000),
                 D0=rng.randint(48, 160), D1=rng.randint(48, 160), box=1.0, fit="l2")
    elif kind == "particles":
        D = rng.randint(64, 128)
        c.update(kind="fit", frames="so3", iso=False, N=_log_int(rng, 512, 8192),
                 A=_log_int(rng, 1000, 20000), D0=D, D1=D, box=1.0, fit="l2", order=1)
    elif kind == "psf":
        D = rng.randint(32, 80)
        c.update(frames="so3", N=_log_int(rng, 16, 256), A=_log_int(rng, 30, 400), D0=D, D1=D,
                 box=1.0, fit="l2", order=1)
    else:
        c.update(frames="vol", N=_log_int(rng, 16, 4096), A=1, D0=rng.randint(32, 160),
                 D1=rng.randint(32, 160), box=1.0, fit="l2", order=0)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dim(c):
    return 2 if c["frames"] == "2d" else 3


def _frames(c, seed):
    """(T, (w0[, w1])) float32 host arrays in the reference layout."""
    g = _m("geometry")
    if c["frames"] == "2d":
        th = np.linspace(0, np.pi, c["A"], endpoint=False)
        T, w = g.theta_to_vec([th]), g.perp([th])
    elif c["frames"] == "tilt":
        th = np.linspace(-np.pi / 3, np.pi / 3, c["A"])
        T, w = g.theta_to_vec([th]), g.perp([th])
    else:
        R = _m("workloads").random_rotations(np.random.default_rng(seed), c["A"])
        T, w = R[:, :, 2], (R[:, :, 0], R[:, :, 1])
    return T.astype(np.float32), tuple(o.astype(np.float32) for o in w)


def _detector(c):
    f = _m("workloads").cell_centres
    d = (f(-c["box"], c["box"], c["D0"]),)
    if c["frames"] != "2d":
        d += (f(-c["box"], c["box"], c["D1"]),)
    return tuple(a.astype(np.float32) for a in d)


def _atoms(c, gen):
    """(I, x, r) float32 device tensors with the configurations' distributions."""
    N, d = c["N"], _dim(c)
    U = lambda lo, hi, *s: lo + (hi - lo) * torch.rand(*s, generator=gen, device="cuda")
    half = {"2d": 0.6, "tilt": 1.0}.get(c["frames"], 0.7)
    x = U(-half, half, N, d)
    I = U(0.5, 1.5, N) if d == 2 else U(0.2, 2.0, N)
    if c["iso"]:
        r = 1.0 / (math.sqrt(60.0) * U(0.02, 0.08, N, 1)) if d == 2 else U(10.0, 50.0, N, 1)
    else:
        lo, hi, sd = (8.0, 40.0, 5.0) if d == 2 else (10.0, 50.0, 6.0)
        off = torch.randn(N, 1 if d == 2 else 3, generator=gen, device="cuda") * sd
        r = torch.cat([U(lo, hi, N, d), off], 1)
    return I, x, r.contiguous()


def _clean(c, I, x, r, T, w, det):
    """Projection of isotropic atoms of the same size, FP32."""
    d = _dim(c)
    s = r[:, 0] if c["iso"] else torch.exp(torch.log(r[:, :d]).mean(1))
    p = [torch.from_numpy(a).cuda() for a in det]
    amp = (I / s).reshape(1, -1)
    out = torch.empty((c["A"],) + tuple(a.numel() for a in p), device="cuda")
    wt = [torch.from_numpy(a).cuda() for a in w]
    if c["frames"] == "tilt":
        wt = [torch.cat([wt[0], torch.zeros(c["A"], 1, device="cuda")], 1),
              torch.tensor([[0.0, 0.0, 1.0]], device="cuda").expand(c["A"], 3)]
    step = max(1, int(2e8 / (c["N"] * max(c["D0"], c["D1"]))))
    for a in range(0, c["A"], step):
        u = []
        for k in range(d - 1):
            q = wt[k][a:a + step] @ x.T
            u.append(torch.exp(-30.0 * (s.reshape(1, -1, 1) * (p[k] - q[:, :, None])) ** 2))
        if d == 2:
            out[a:a + step] = (amp @ u[0])[:, 0]
        else:
            out[a:a + step] = (u[0] * amp[:, :, None]).transpose(1, 2) @ u[1]
    return out


BACKGROUND = 1.0


def _problem(c, seed):
    """Atoms to fit, geometry arrays and data."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 13)
    T, w = _frames(c, seed)
    det = _detector(c)
    I, x, r = _atoms(c, gen)
    N = c["N"]
    if c["A"] * c["D0"] * c["D1"] * N > 1e12:
        # whole image sets: noise of ten times the signal's power hides what
        # the images show of the atoms, so the noise alone stands for the data
        # (signal: about N in-support sums of amplitude I / s)
        sd = math.sqrt(10.0) * 0.02 * math.sqrt(N / 512.0)
        data = sd * torch.randn((c["A"], c["D0"], c["D1"]), generator=gen, device="cuda")
        return I, x, r, T, w, det, data
    sd = 0.1 / (math.sqrt(60.0) * r[:, :1 if c["iso"] else _dim(c)].amax(1, keepdim=True))
    xt = x + torch.randn(x.shape, generator=gen, device="cuda") * sd
    It = I * (0.9 + 0.2 * torch.rand(N, generator=gen, device="cuda"))
    clean = _clean(c, It, xt, r, T, w, det)
    if c["fit"] == "kl":
        scale = 1e4 / clean.max()
        I = I * scale
        data = torch.poisson(clean * scale + BACKGROUND, generator=gen)
    else:
        data = clean + torch.randn(clean.shape, generator=gen, device="cuda") * (0.01 * clean.max())
    return I.contiguous(), x, r, T, w, det, data.contiguous()


def _coords(c):
    n = (c["D0"], c["D1"], (c["D0"] + c["D1"]) // 2)
    return [np.linspace(-1, 1, k).astype(np.float32) for k in n]


class _Radon:
    def __init__(self, space):
        self.range = space


def _moved(c, I, x, r, j):
    """The trial parameters of atom j of a per-atom step (host arrays)."""
    return I[j:j + 1] * np.float32(1.03), x[j:j + 1] + np.float32(0.004), \
        r[j:j + 1] * np.float32(0.99)


def prepare(case, seed):
    c = case
    eng, geo = _m("engine"), _m("geometry")
    s = dict(case=c)
    if c["kind"] == "render":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed) * 7919 + 13)
        s.update(atoms=eng.DeviceAtoms(*_atoms(c, gen)), coords=_coords(c))
        return s
    I, x, r, T, w, det, data = _problem(c, seed)
    if c["kind"] == "dropin":
        sp = _m("spaces")
        space = sp.ProjSpace(orientations=T, ortho=w, detector=det)
        atom = sp.AtomSpace(2, isotropic=c["iso"]).element(x.cpu(), r.cpu(), I.cpu())
        s.update(Radon=_Radon(space), atom=atom, C=data.cpu().numpy())
        return s
    geom = geo.DeviceGeometry(T, w, det)
    s.update(geom=geom, data=data)
    if c["kind"] == "train":
        s.update(p=[t.clone().requires_grad_(True) for t in (I, x, r)])
    elif c["kind"] == "host":
        s.update(step=eng.FitStep(geom, c["N"], iso=c["iso"], fit=c["fit"], order=c["order"]))
        s["step"].set_inputs(I.cpu(), x.cpu(), r.cpu(), data.cpu())
    elif c["kind"] == "atomstep":
        R = _Exact(c, I, x, r, T, w, det).forward().float()
        s.update(host=[t.cpu().numpy() for t in (I, x, r)], R=R, alpha=R - data, j=seed % c["N"])
    else:
        s.update(atoms=eng.DeviceAtoms(I, x, r))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    c = s["case"]
    eng = _m("engine")
    kind = c["kind"]
    if kind == "render":
        return [_m("volume").volproj(s["atoms"], s["coords"])]
    if kind == "dropin":
        f, Df, DDf = _m("NewtonBases2D").L2derivs_RadProj(s["atom"], s["Radon"], s["C"], order=2)
        return [np.float32(f), Df.astype(np.float32), DDf.astype(np.float32)]
    if kind == "train":
        R = _m("autograd").project(*s["p"], s["geom"])
        return [R.detach()] + list(torch.autograd.grad(R, s["p"], R.detach() - s["data"]))
    if kind == "host":
        loss, g, H = s["step"].run()
        return [np.float32(loss), g.float()] + ([H.float()] if H is not None else [])
    if kind == "atomstep":
        I, x, r = s["host"]
        j = s["j"]
        old = eng.DeviceAtoms(I[j:j + 1], x[j:j + 1], r[j:j + 1])
        _f, g, _H = eng.atom_derivs(old, s["geom"], "field", s["alpha"], None, 1.0, 1)
        new = eng.DeviceAtoms(*_moved(c, I, x, r, j))
        d = eng.atom_step(old, new, s["geom"], "l2", False, s["R"], s["data"], s["alpha"])
        return [g.float(), d.float()]
    if kind == "psf":
        fw = eng.fit_forward(s["atoms"], s["geom"], s["data"], "l2", psf=True)
        _f, g, _H = eng.atom_derivs(s["atoms"], s["geom"], "field", fw["alpha"], None, 1.0, 1,
                                    psf=True)
        return [fw["loss"].float(), fw["alpha"], g.float()]
    if c["fit"] == "kl":
        loss, g, H = eng.kl_fit_derivs(s["atoms"], s["geom"], s["data"], BACKGROUND, c["order"])
    else:
        loss, g, H = eng.l2_fit_derivs(s["atoms"], s["geom"], s["data"], c["order"])
    return [loss.float(), g.float()] + ([H.float()] if H is not None else [])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _evaluations(c):
    """Expected number of in-support (atom, angle, cell) evaluations."""
    rng = np.random.default_rng(0)
    d, n = _dim(c), 512
    if c["iso"]:
        s = 1 / (math.sqrt(60.0) * rng.uniform(0.02, 0.08, n)) if d == 2 else rng.uniform(10, 50, n)
        M = s[:, None, None] * np.eye(d)
    else:
        lo, hi, sd = (8.0, 40.0, 5.0) if d == 2 else (10.0, 50.0, 6.0)
        M = np.zeros((n, d, d))
        for i in range(d):
            M[:, i, i] = rng.uniform(lo, hi, n)
            for j in range(i + 1, d):
                M[:, i, j] = rng.normal(0, sd, n)
    if c["frames"] == "vol":
        cell = np.prod([2.0 / (k.size - 1) for k in _coords(c)])
        return c["N"] * float(np.mean(4 / 3 * np.pi / np.abs(np.linalg.det(M)))) / cell
    B = np.linalg.qr(rng.normal(size=(n, d, d)))[0]
    K = M @ B
    Q = np.einsum("nac,nad->ncd", K, K)
    G = Q[:, :-1, :-1] - Q[:, :-1, -1:] * Q[:, -1:, :-1] / Q[:, -1:, -1:]
    cell = 2 * c["box"] / c["D0"] * (1.0 if d == 2 else 2 * c["box"] / c["D1"])
    area = (2.0 if d == 2 else np.pi) / np.sqrt(np.linalg.det(G))
    return c["N"] * c["A"] * float(np.mean(area)) / cell


def work(case):
    c = case
    d = _dim(c)
    P = (2 + d) if c["iso"] else (1 + d + (3 if d == 2 else 6))
    ev = _evaluations(c)
    if c["kind"] == "render":
        return {"bytes": 4.0 * np.prod([k.size for k in _coords(c)]) + 4.0 * c["N"] * P,
                "flops": 16.0 * ev}
    cells = float(c["A"]) * c["D0"] * c["D1"]
    # per evaluation: quadratic form, exponential and sum (forward), the
    # weighted moments (gradient: degree 2, Hessian: degree 4, twice)
    grad = {1: 16.0, 2: 48.0}[c["order"]]
    out = 4.0 * c["N"] * (1 + P + (P * P if c["order"] == 2 else 0))
    flops, nbytes = (12.0 + grad) * ev, 4.0 * cells + out + 4.0 * c["N"] * P
    if c["kind"] == "dropin":
        flops = grad * ev
    elif c["kind"] == "atomstep":
        # one atom's gradient and the change of the fit over its support
        flops, nbytes = (grad + 24.0) * ev / c["N"], 8.0 * ev / c["N"] + 8.0 * (1 + P)
    elif c["kind"] == "train":
        nbytes += 4.0 * cells
    elif c["kind"] == "psf":
        flops, nbytes = 121 * (8.0 + 10.0) * ev, nbytes + 4.0 * cells
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
class _Exact:
    """The operator of the reference in float64: per (atom, angle) the
    projected Gaussian I n exp(-30 (q - q*)^T G (q - q*)) where the form is
    at most 1, on windows of cells around q*."""

    SLOTS = 1 << 24

    def __init__(self, c, I, x, r, T, w, det):
        f = lambda a: torch.as_tensor(a).cuda().double()
        self.c, self.d = c, _dim(c)
        A = c["A"]
        T, w = f(T), [f(o) for o in w]
        if c["frames"] == "tilt":
            z = torch.zeros(A, 1, dtype=torch.float64, device="cuda")
            T, w = torch.cat([T, z], 1), [torch.cat([w[0], z], 1),
                                          torch.tensor([[0.0, 0.0, 1.0]], device="cuda",
                                                       dtype=torch.float64).expand(A, 3)]
        self.B = torch.stack(w + [T], 2)                       # columns w0 (w1) T
        self.Binv = torch.linalg.inv(self.B)
        self.p = [f(a) for a in det]
        self.first = [float(a[0]) for a in self.p]
        self.h = [float((a[-1] - a[0]) / (a.numel() - 1)) for a in self.p]
        self.theta = torch.cat([f(I).reshape(-1, 1), f(x), f(r).reshape(c["N"], -1)], 1)

    def pair(self, th, a):
        """(I, ln n, G (list), q (list)) of parameter rows th at angles a."""
        d, k = self.d, self.d - 1
        r = th[:, 1 + d:]
        z = torch.zeros_like(r[:, 0])
        if self.c["iso"]:
            rows = [[r[:, 0] if i == j else z for j in range(d)] for i in range(d)]
        elif d == 2:
            rows = [[r[:, 0], r[:, 2]], [z, r[:, 1]]]
        else:
            rows = [[r[:, 0], r[:, 3], r[:, 5]], [z, r[:, 1], r[:, 4]], [z, z, r[:, 2]]]
        M = torch.stack([torch.stack(v, 1) for v in rows], 1)
        K = M @ self.B[a]
        Q = K.transpose(1, 2) @ K
        qt = Q[:, k, k]
        G = [Q[:, i, j] - Q[:, i, k] * Q[:, j, k] / qt for i in range(k) for j in range(i, k)]
        q = (self.Binv[a][:, :k] @ th[:, 1:1 + d, None])[:, :, 0]
        return th[:, 0], -0.5 * torch.log(qt), G, [q[:, i] for i in range(k)]

    def blocks(self, slots, extra=None):
        """(angles, atoms, first cells, window) lists covering every pair, of
        at most ``slots`` window cells each."""
        c, k = self.c, self.d - 1
        step = max(1, int(2 ** 21 // c["N"]))
        for a0 in range(0, c["A"], step):
            na = min(step, c["A"] - a0)
            a = torch.arange(a0, a0 + na, device="cuda").repeat_interleave(c["N"])
            j = torch.arange(c["N"], device="cuda").repeat(na)
            with torch.no_grad():
                _I, _l, G, q = self.pair(self.theta[j], a)
                if extra is not None:
                    hw = [extra[j] for _ in range(k)]
                elif k == 1:
                    hw = [G[0] ** -0.5]
                else:
                    det = G[0] * G[2] - G[1] ** 2
                    hw = [torch.sqrt(G[2] / det), torch.sqrt(G[0] / det)]
                lo, n, key = [], [], torch.zeros_like(j)
                for i in range(k):
                    D = self.p[i].numel()
                    cc, hh = (q[i] - self.first[i]) / self.h[i], hw[i] / self.h[i] + 0.01
                    l = torch.ceil(cc - hh).clamp(0, D).long()
                    u = torch.floor(cc + hh).clamp(-1, D - 1).long()
                    m = (u - l + 1).clamp(min=0)
                    lo.append(l)
                    n.append(m)
                    # windows rounded up to a few sizes
                    key = key * 64 + torch.ceil(2 * torch.log2(m.double().clamp(min=0.5)) + 2).long()
                live = torch.ones_like(j, dtype=torch.bool)
                for m in n:
                    live &= m > 0
            for v in torch.unique(key[live]).tolist():
                at = torch.nonzero(live & (key == v))[:, 0]
                W = [int(m[at].max()) for m in n]
                per = max(1, slots // int(np.prod(W)))
                for b in range(0, at.numel(), per):
                    t = at[b:b + per]
                    yield a[t], j[t], [l[t] for l in lo], W

    def window(self, a, lo, W):
        """(flat cell index, inside mask, cell coordinates per axis)."""
        idx, ok, p = [], True, []
        for i, (l, n) in enumerate(zip(lo, W)):
            D = self.p[i].numel()
            e = l[:, None] + torch.arange(n, device="cuda")
            inside = e < D
            e = e.clamp(max=D - 1)
            sh = (-1, n, 1) if (i == 0 and len(W) == 2) else ((-1, 1, n) if i else (-1, n))
            idx.append(e.reshape(sh))
            p.append(self.p[i][e].reshape(sh))
            ok = ok & inside.reshape(sh)
        flat = idx[0] if len(W) == 1 else idx[0] * self.p[1].numel() + idx[1]
        cells = int(np.prod([t.numel() for t in self.p]))
        return a.reshape((-1,) + (1,) * len(W)) * cells + flat, ok, p

    def form(self, G, q, p):
        e = lambda t: t.reshape((-1,) + (1,) * len(p))
        dd = [p[i] - e(q[i]) for i in range(len(p))]
        if len(p) == 1:
            return e(G[0]) * dd[0] ** 2, dd
        return e(G[0]) * dd[0] ** 2 + 2 * e(G[1]) * dd[0] * dd[1] + e(G[2]) * dd[1] ** 2, dd

    def shape(self):
        return (self.c["A"],) + tuple(t.numel() for t in self.p)

    def forward(self):
        R = torch.zeros(self.shape(), dtype=torch.float64, device="cuda")
        with torch.no_grad():
            for a, j, lo, W in self.blocks(self.SLOTS):
                I, ln, G, q = self.pair(self.theta[j], a)
                at, ok, p = self.window(a, lo, W)
                m, _d = self.form(G, q, p)
                e = lambda t: t.reshape((-1,) + (1,) * len(p))
                v = torch.where(ok & (m <= 1), e(I) * torch.exp(e(ln) - 30.0 * m), 0.0)
                R.view(-1).index_add_(0, at.reshape(-1), v.reshape(-1))
        return R

    def linear(self, th, a, A0, M):
        """The function of the parameters whose gradient is that of
        sum alpha R, given the (fixed) moments of alpha E."""
        I, ln, G, q = self.pair(th, a)
        I0, Gd = I.detach(), [g.detach() for g in G]
        if len(q) == 1:
            s = A0 * ln - 30.0 * M[1] * G[0] + 60.0 * Gd[0] * M[0] * q[0]
        else:
            s = (A0 * ln - 30.0 * (M[2] * G[0] + 2 * M[3] * G[1] + M[4] * G[2])
                 + 60.0 * ((Gd[0] * M[0] + Gd[1] * M[1]) * q[0]
                           + (Gd[1] * M[0] + Gd[2] * M[1]) * q[1]))
        return (A0 * I + I0 * s).sum()

    @staticmethod
    def moments(wE, dd):
        ax = tuple(range(1, wE.dim()))
        if len(dd) == 1:
            return wE.sum(ax), [(wE * dd[0]).sum(ax), (wE * dd[0] ** 2).sum(ax)]
        return wE.sum(ax), [(wE * dd[0]).sum(ax), (wE * dd[1]).sum(ax), (wE * dd[0] ** 2).sum(ax),
                            (wE * dd[0] * dd[1]).sum(ax), (wE * dd[1] ** 2).sum(ax)]

    def gradient(self, alpha):
        g = torch.zeros_like(self.theta)
        alpha = alpha.reshape(-1)
        for a, j, lo, W in self.blocks(self.SLOTS):
            with torch.no_grad():
                _I, ln, G, q = self.pair(self.theta[j], a)
                at, ok, p = self.window(a, lo, W)
                m, dd = self.form(G, q, p)
                e = lambda t: t.reshape((-1,) + (1,) * len(p))
                wE = torch.where(ok & (m <= 1), torch.exp(e(ln) - 30.0 * m), 0.0) * alpha[at]
                A0, M = self.moments(wE, dd)
            th = self.theta[j].requires_grad_(True)
            g.index_add_(0, j, torch.autograd.grad(self.linear(th, a, A0, M), th)[0])
        return g

    def hessian(self, alpha, beta):
        """Gradient and per-atom Hessian of sum alpha R + beta (R - R0)^2 / 2."""
        n, P = self.theta.shape
        g = torch.zeros_like(self.theta)
        H = torch.zeros(n, P, P, dtype=torch.float64, device="cuda")
        alpha = alpha.reshape(-1)
        beta = None if beta is None else beta.reshape(-1)
        for a, j, lo, W in self.blocks(self.SLOTS // 4):
            th = self.theta[j].requires_grad_(True)
            I, ln, G, q = self.pair(th, a)
            at, ok, p = self.window(a, lo, W)
            m, _d = self.form(G, q, p)
            e = lambda t: t.reshape((-1,) + (1,) * len(p))
            R = torch.where(ok & (m <= 1), e(I) * torch.exp(e(ln) - 30.0 * m), 0.0)
            b = 1.0 if beta is None else beta[at]
            S = (alpha[at] * R + 0.5 * b * (R - R.detach()) ** 2).sum()
            gp = torch.autograd.grad(S, th, create_graph=True)[0]
            for k in range(P):
                h = torch.autograd.grad(gp[:, k].sum(), th, retain_graph=k + 1 < P)[0]
                H[:, k].index_add_(0, j, h)
            g.index_add_(0, j, gp.detach())
        return g, H

    def integrated(self, data):
        """Loss, residual and gradient of the pixel-integrated operator (11 x
        11 points a cell at lo + t (hi - lo) / 10, t = 1..11, of the cell
        clipped to +-rr around the centre, rr = 1 / min(diag r))."""
        d = self.d
        s = 0.5 * self.h[0]
        r = self.theta[:, 1 + d:]
        rr = 1.0 / (r[:, 0] if self.c["iso"] else r[:, :d].amin(1))
        t = torch.arange(1, 12, dtype=torch.float64, device="cuda")
        R = torch.zeros(self.shape(), dtype=torch.float64, device="cuda")
        alpha, g = None, torch.zeros_like(self.theta)
        for gradient in (False, True):
            for a, j, lo, W in self.blocks(self.SLOTS // 128, rr + s * 1.5):
                with torch.no_grad():
                    I, ln, G, q = self.pair(self.theta[j], a)
                    at, ok, p = self.window(a, lo, W)
                    e = lambda v: v.reshape(-1, 1, 1)
                    dc = [p[i] - e(q[i]) for i in range(2)]
                    ok = ok & (torch.sqrt(dc[0] ** 2 + dc[1] ** 2) - e(rr[j]) <= s)
                    st, pt = [], []
                    for i in range(2):
                        l = torch.maximum(-dc[i] - e(rr[j]), torch.tensor(-s, device="cuda").double())
                        u = torch.minimum(-dc[i] + e(rr[j]), torch.tensor(s, device="cuda").double())
                        st.append((u - l) / 10)
                        v = (dc[i] + l)[..., None] + t * st[i][..., None]
                        pt.append(v[..., :, None] if i == 0 else v[..., None, :])
                    f = lambda v: v.reshape(-1, 1, 1, 1, 1)
                    m = f(G[0]) * pt[0] ** 2 + 2 * f(G[1]) * pt[0] * pt[1] + f(G[2]) * pt[1] ** 2
                    E = torch.exp(f(ln) - 30.0 * m) * (100.0 / 121.0 * st[0] * st[1]
                                                       * ok)[..., None, None]
                    if not gradient:
                        v = e(I) * E.sum((3, 4))
                        R.view(-1).index_add_(0, at.reshape(-1), v.reshape(-1))
                        continue
                    A0, M = self.moments(E * alpha.reshape(-1)[at][..., None, None], pt)
                th = self.theta[j].requires_grad_(True)
                g.index_add_(0, j, torch.autograd.grad(self.linear(th, a, A0, M), th)[0])
            if alpha is None:
                alpha = R - data.double()
        return 0.5 * (alpha ** 2).sum(), alpha, g


def _volume64(c, I, x, r):
    d = 3
    y = [torch.from_numpy(a).cuda().double() for a in _coords(c)]
    I, x, r = I.double(), x.double(), r.double()
    if c["iso"]:
        r = torch.cat([r.reshape(-1, 1).expand(-1, d), torch.zeros(r.shape[0], 3, device="cuda")], 1)
    u = torch.zeros([t.numel() for t in y], dtype=torch.float64, device="cuda")
    for j in range(c["N"]):
        M = r[j].tolist()
        X = x[j].tolist()
        rad = 1.0 / float(np.linalg.svd(np.array([[M[0], M[3], M[5]], [0, M[1], M[4]],
                                                  [0, 0, M[2]]]), compute_uv=False)[-1])
        sl, Y = [], []
        for i in range(d):
            h = 2.0 / (y[i].numel() - 1)
            a = max(0, int((X[i] - rad + 1) / h) - 1)
            b = min(y[i].numel(), int((X[i] + rad + 1) / h) + 3)
            sl.append(slice(a, b))
            Y.append((y[i][a:b] - X[i]).reshape([-1 if k == i else 1 for k in range(d)]))
        nn = ((M[0] * Y[0] + M[3] * Y[1] + M[5] * Y[2]) ** 2 + (M[1] * Y[1] + M[4] * Y[2]) ** 2
              + (M[2] * Y[2]) ** 2)
        u[tuple(sl)] += torch.where(nn <= 1, float(I[j]) * math.sqrt(30.0 / math.pi)
                                    * torch.exp(-30.0 * nn), 0.0)
    return u


def exact(case, seed):
    c = case
    if c["kind"] == "render":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed) * 7919 + 13)
        return [_volume64(c, *_atoms(c, gen))]
    I, x, r, T, w, det, data = _problem(c, seed)
    X = _Exact(c, I, x, r, T, w, det)
    D = data.double()
    if c["kind"] == "psf":
        return list(X.integrated(data))
    if c["kind"] == "dropin":
        R = X.forward()
        g, H = X.hessian(R - D, None)
        return [0.5 * ((R - D) ** 2).sum(), g[0], H[0]]
    if c["kind"] == "atomstep":
        R = X.forward().float()
        alpha = (R - data).double()
        hI, hx, hr = (t.cpu().numpy() for t in (I, x, r))
        j = seed % c["N"]
        one = dict(c, N=1)
        old = _Exact(one, hI[j:j + 1], hx[j:j + 1], hr[j:j + 1], T, w, det)
        new = _Exact(one, *_moved(c, hI, hx, hr, j), T, w, det)
        delta = new.forward() - old.forward()
        return [old.gradient(alpha), (delta * (alpha + 0.5 * delta)).sum()]
    R = X.forward()
    if c["kind"] == "train":
        g, d = X.gradient(R - D), X.d
        return [R, g[:, 0], g[:, 1:1 + d], g[:, 1 + d:]]
    if c["fit"] == "kl":
        G = R + BACKGROUND
        loss = (torch.where(D > 0, D * torch.log(D.clamp(min=1e-30) / G), 0.0) - D + G).sum()
        alpha, beta = 1.0 - D / G, D / G ** 2
    else:
        alpha, beta = R - D, None
        loss = 0.5 * (alpha ** 2).sum()
    del R, D
    if c["order"] == 1:
        return [loss, X.gradient(alpha)]
    return [loss] + list(X.hessian(alpha, beta))
