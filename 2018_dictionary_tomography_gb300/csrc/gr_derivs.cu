// Per-atom derivatives of data fits (sm_103a).
//
// Replaces the reference's one-atom-per-launch kernels
// __L2derivs_RadProj_aniso (GaussDictCode/bin/NewtonBases2D.py:331-401),
// __derivs_RadProj_aniso (NewtonBases2D.py:446-515) and their 3D twins
// (GaussDictCode/bin/NewtonBases.py:794-870, :995-1069), which evaluate a
// 6x6 / 10x10 per-cell Hessian of one atom at every detector cell.
//
// For one (atom, angle) pair the projection is R(q) = I E(q),
// E = n exp(-30 (q - q*)^T G (q - q*)) (see gr_common.cuh), so
//   ln E = ln n - 30 d^T G d,   d = q - q*,
// is linear in psi = (ln n, G, q*) up to the quadratic dependence on q*.
// Every derivative sum over cells of a weight field w times a polynomial in d
// is therefore a combination of a few cell moments  M_ij = sum w d0^i d1^j
// (degree <= 2 for gradients, <= 4 for Hessians), and the chain rule from psi
// to (I, x, r) is done once per pair:
//   psi -> Q = (r B)^T (r B) -> r   and   q* = (B^{-1} x)[0:K].
// Per cell the kernel evaluates one exp2 and a handful of FMAs; moments are
// accumulated per detector row and folded with powers of d0 at row end.
//
// Work layout: a warp's lanes are the (atom, angle) pairs of one atom (or a
// few) and a chunk of angles.  A lane sets its pair up and does its chain-rule
// assembly; in between, for Hessians, groups of lanes walk the pairs' cells
// together (gr_hess_kernel); for gradients (gr_grad_kernel) a lane walks alone.  Gradients are
// accumulated per lane with compensated FP32 sums, Hessians in FP32; lanes
// sharing an atom are combined by a fixed-order butterfly; chunk partials are
// summed in FP64 in chunk order by gr_deriv_finalize_kernel, which also applies
// the isotropic chain rule.  No float atomics anywhere: results are bitwise
// reproducible.
#include <type_traits>

#include "gr_assembly.cuh"

namespace gr {

inline int next_pow2(int v) {
  int p = 1;
  while (p < v && p < 32) p <<= 1;
  return p;
}

// resident warps per SM asked of the Hessian kernels
__host__ __device__ constexpr int hess_min_warps(int K, bool one) {
  return one ? (K == 1 ? 24 : 16) : 4;
}

// Work split of the derivative kernels (Tuning, gr_set_tuning / gr_plan_set):
// about deriv_target_warps warps in total, each angle chunk holding at least
// deriv_min_angles angles per lane group.
// deriv_atoms_per_warp (power of two up to 32; 0 = automatic): with fewer
// atoms per warp the lanes of a warp take different angles of one atom, whose
// support boxes are of similar size, so fewer lanes idle.  Automatic: one
// atom per warp for Hessians and for long angle series, else four (so each
// lane still has a few angles to amortise the warp's closing reduction).  A 3D
// gradient has a cheap closing reduction for one atom, so there a series is long
// from 64 angles on if rounding it up to a warp's 32 angles leaves few more lanes
// idle than rounding to eight, or if pairs are shared among lanes anyway (us, one and
// four atoms a warp, 8192 atoms x 64^2: 32 angles 33.7, 33.7; 33: 51.7, 40.6; 48: 53.4,
// 46.8; 64: 56.5, 57.8; 65: 74.8, 64.2; 80: 77.3, 71.0; 96: 78.7, 82.4; 97: 97.7, 86.2; 128:
// 101.2, 106.4; 300: 237, 240; 700: 508, 538; 100 atoms, shared: 64: 8.6, 10.1; 65: 9.4,
// 10.7; 300: 11.6, 12.7).  (The pixel-integrated kernel keeps the longer line: 66 us
// with four, 76 with one at 128 x 401 x 64^2.)
// deriv_split_lanes: problems with few (atom, angle) pairs give a warp 32 / rs
// of them, rs the largest power of two up to 8 with pairs * rs <=
// deriv_split_lanes, so that the pairs spread over more warps (a 3D gradient's
// pair then has its rows split over rs lanes).  0: never split.
// deriv_one_mb: take as many angle chunks as give every lane at most one
// angle (the ONE kernel variant: fewer registers, no spills) whenever the
// chunk partials then fit in this many MB; 0: keep the target-warps split.
// On 8192 atoms x 20000 orientations the one-angle split (625 chunks, 225 MB
// of partials) runs the gradient kernel in 23.6 ms against 25.7 ms for 16
// chunks.
DerivCfg deriv_cfg(int K, int n_atoms, int n_angles, int order, const Tuning &t, bool split) {
  DerivCfg c;
  c.ag = next_pow2(n_atoms < 1 ? 1 : n_atoms);
  const long long pairs = (long long)(n_atoms < 1 ? 1 : n_atoms) * (n_angles < 1 ? 1 : n_angles);
  bool one_atom = order > 1 || n_angles >= 1024;
  if (K == 2 && split && n_angles >= 64)
    one_atom = one_atom || 2 * pairs <= (long long)t.deriv_split_lanes ||
               32 * ((n_angles + 31) / 32) <= 8 * ((n_angles + 7) / 8) * 17 / 16;
  const int ag_cap = t.deriv_atoms_per_warp > 0 ? t.deriv_atoms_per_warp : one_atom ? 1 : 4;
  if (c.ag > ag_cap) c.ag = ag_cap;
  c.sg = 32 / c.ag;
  c.rs = 1;
  while (split && t.deriv_split_lanes > 0 && c.rs < 8 && c.rs < c.sg &&
         pairs * c.rs * 2 <= (long long)t.deriv_split_lanes)
    c.rs <<= 1;
  const int warps_atoms = (n_atoms + c.ag - 1) / c.ag;
  int nch = (t.deriv_target_warps + warps_atoms - 1) / warps_atoms;
  const int per = (c.sg / c.rs) * (t.deriv_min_angles < 1 ? 1 : t.deriv_min_angles);
  const int max_ch = (n_angles + per - 1) / per;
  if (nch > max_ch) nch = max_ch;
  const int P0 = 1 + (K + 1) + (K == 1 ? 3 : 6);
  const size_t qn0 = 1 + P0 + (order > 1 ? P0 * (P0 + 1) / 2 : 0);
  if (t.deriv_one_mb > 0 && t.deriv_min_angles == 1 && nch < max_ch &&
      (size_t)max_ch * qn0 * (size_t)(n_atoms < 1 ? 1 : n_atoms) * sizeof(float) <=
          ((size_t)t.deriv_one_mb << 20))
    nch = max_ch;
  if (nch < 1) nch = 1;
  c.ch = (n_angles + nch - 1) / nch;
  if (c.ch < 1) c.ch = 1;
  c.nchunks = (n_angles + c.ch - 1) / c.ch;
  const int P = 1 + (K + 1) + (K == 1 ? 3 : 6);
  c.qn = 1 + P + (order > 1 ? P * (P + 1) / 2 : 0);
  return c;
}

// ---- the cell walk -----------------------------------------------------------
// A warp's pairs are set up one per lane and staged in shared memory; groups of
// GL lanes then walk one pair each, lane l the cells of columns l, l + GL, ..
// of its support (3D) or the cells l, l + GL, .. (2D), so that a load of the
// weight field covers GL neighbouring cells, and the lanes' moment sums are
// combined and handed back to the pair's lane, which does the chain-rule
// assembly.  The groups walk rows (3D) in step, so that their loads share
// sectors, and two cells at a time in packed FP32 pairs.
// What bounds it: issue (51 % of the slots in 3D, 60 % in 2D) and the 128 registers
// of the 3D assembly (16 warps an SM; 168 registers and 12 warps: 363 against 301 us,
// 96 registers 310 us with four rows a lane).  A lane walking a wide pair alone
// waited on 32 lines of the field per load with 12 warps an SM and 124
// registers of moment sums; a group's lane keeps 20.  2936 atoms x 148 x 493^2
// (3D, 120 cells a pair): 401 -> 277 us; 146 x 61 x 301 x 275: 18.7 -> 15.5 us;
// 2150 x 153 x 467 (2D): 85.5 -> 58.6 us.  Cells a lane loads together: 2D, 2 lanes:
// 4, 6, 8: 60.0, 58.6, 56.8 us there, 11.5, 11.8, 11.8 us on 512 x 180 x 256 (9 cells a
// pair); 3D, 4 lanes: 2, 4, 6, 8: 397, 301, 277, 290 us.  4 lanes in 2D: 61.9 and 11.2
// us.  Narrow pairs: walk_narrow_of.
// cells of a lane loaded together (even)
template <int K>
__host__ __device__ constexpr int walk_cells_of() { return 6; }
// Where all pairs of a warp have boxes of at most this many cells along each axis, a
// lane walks its own pair, two cells at a time: groups would give most of their lanes
// nothing and pay for the exchange of 16 or 32 sums (us, own lane up to 0, 4, 5, 6, 8,
// 10, 12, 16 cells: 3364 atoms x 751 x 41^2, r = 30: 432, 307, 307, 307, 307, 307, 307,
// 307; 7599 x 63 x 24^2, 5 cells: 123, 129, 126, 113, 101, 100, 100, 100; 1000 x 100 x
// 128^2, r = 7: -, -, -, -, 82, 82, 84, 92; 2D, up to 0, 8, 12, 16, 24, 32, 48, 64 cells:
// 7293 x 106 x 55: 54, 44, 43, 43, 43, 43, 43, 43; 2150 x 153 x 467, r = 8: 37, -, -, -,
// 37, 37, 39, 40).
template <int K>
__host__ __device__ constexpr int walk_narrow_of() { return K == 1 ? 24 : 8; }
// lanes of a group (8 where a warp has four pairs; in 2D 4 where it has eight)
template <int K>
__host__ __device__ constexpr int walk_lanes_of() { return K == 1 ? 2 : 4; }
template <int K>
__host__ __device__ constexpr int n_sums() {   // moments (alpha, beta), sum E C, sum E^2
  return (2 * n_mom<K, 4>() + 2 + 7) / 8 * 8;   // (up to 8 lanes share them out)
}

// What the weight fields are: a kernel of its own for each (a test in the cell
// loop cost the Hessian kernels 10 to 20 %), one for all where a lane takes
// several angles.
enum FieldKind : int { kFieldPlain = 0, kFieldBeta = 1, kFieldL2Atom = 2, kFieldAny = 3 };

struct WalkPair {
  float4 q;      // -qh0, -ql0, -qh1, -ql1
  float4 v;      // G00, 2 G01, G11, log2 n
  float4 r;      // centre row, its drift per unit of d1, half-height per unit, I (walk_stage)
  float4 e;      // det G, d1 of the support's lowest row
  int4 box;      // first and last cell along each axis
};

template <int K>
struct WalkSmem {
  static constexpr int NV = n_sums<K>();
  WalkPair pair[32];
  float sum[32][NV + 1];
};

template <int K>
__device__ __forceinline__ void walk_stage(const Pair<K> &p, const Geom &g, float I, WalkPair &w) {
  w.q = make_float4(-p.qh[0], -p.ql[0], K == 2 ? -p.qh[K - 1] : 0.f, K == 2 ? -p.ql[K - 1] : 0.f);
  w.v = make_float4(p.G[0], 2.f * p.G[1], p.G[2], lg2_approx(p.n));
  const DetAxis &x0 = g.ax[0];
  // 3D: at column offset d1 the support's rows are r.x - r.y d1 -+ r.z
  // sqrt(G00 - e.x d1^2); its lowest row is at d1 = e.y, its highest at -e.y
  const float iG0 = 1.f / p.G[0], det = p.G[0] * p.G[2] - p.G[1] * p.G[1];
  w.r = make_float4((p.qh[0] - x0.first) * x0.inv_step, p.G[1] * iG0 * x0.inv_step,
                    iG0 * x0.inv_step, I);
  w.e = make_float4(det, K == 2 && p.G[1] != 0.f ? p.G[1] * rsqrtf(p.G[2] * det) : 0.f,
                    0.f, 0.f);
  // a support off the detector along either axis has no cells (the walk's rows
  // and columns are clipped to the box, not to the detector)
  const bool live = p.lo[0] <= p.hi[0] && p.lo[K - 1] <= p.hi[K - 1];
  w.box = live ? make_int4(p.lo[0], p.hi[0], p.lo[K - 1], p.hi[K - 1]) : make_int4(1, 0, 1, 0);
}

__device__ __forceinline__ F2 f2_keep(const F2 &v, bool k0, bool k1) {
  float x, y;
  f2_get(v, x, y);
  return f2(k0 ? x : 0.f, k1 ? y : 0.f);
}

// Two cells' terms: m their form, d0 their offsets along axis 0, c and b their
// field values.
// Sa, Sb: sums over alpha E and beta E^2 times powers of d0.
__device__ __forceinline__ void walk_cells(F2 m, F2 d0, bool in0, bool in1, F2 c, F2 b, float l2n,
                                           float I, const bool l2atom, const bool bfield,
                                           F2 (&Sa)[5], F2 (&Sb)[5], F2 &X0, F2 &Y0) {
  constexpr int DEG = 4;
  float m0, m1;
  f2_get(m, m0, m1);
  in0 = in0 && m0 <= 1.f;
  in1 = in1 && m1 <= 1.f;
  float e0, e1;
  f2_get(f2_fma(m, f2(kNegThirtyLog2e, kNegThirtyLog2e), f2(l2n, l2n)), e0, e1);
  const F2 E = f2(ex2_approx(e0), ex2_approx(e1));
  F2 al = c;
  if (l2atom) al = f2_fma(f2(I, I), E, f2_mul(c, f2(-1.f, -1.f)));
  // the products, not their factors, are cut off: a field value beyond the
  // cut-off counts for nothing, also one that is not finite
  const F2 w = f2_keep(f2_mul(al, E), in0, in1);
  F2 pw[DEG + 1];
  pw[1] = d0;
#pragma unroll
  for (int q = 2; q <= DEG; ++q) pw[q] = f2_mul(pw[q - 1], d0);
  Sa[0] = f2_add(Sa[0], w);
#pragma unroll
  for (int q = 1; q <= DEG; ++q) Sa[q] = f2_fma(w, pw[q], Sa[q]);
  // a constant beta scales the moments once per pair instead
  F2 wb = f2_mul(E, E);
  if (bfield) wb = f2_mul(wb, b);
  wb = f2_keep(wb, in0, in1);
  Sb[0] = f2_add(Sb[0], wb);
#pragma unroll
  for (int q = 1; q <= DEG; ++q) Sb[q] = f2_fma(wb, pw[q], Sb[q]);
  if (l2atom) {
    X0 = f2_add(X0, f2_keep(f2_mul(E, c), in0, in1));
    Y0 = f2_add(Y0, f2_keep(f2_mul(E, E), in0, in1));
  }
}

__device__ __forceinline__ float f2_sum(const F2 &a) {
  float x, y;
  f2_get(a, x, y);
  return x + y;
}

// The sums of one pair over this lane's share of its cells (v: moments of
// alpha, of beta, then sum E C and sum E^2).  R: cells of a column loaded
// together before any is used (even); they may lie past the support's end
// (their terms are cut off), not past the detector's.
template <int K, int GL, int R, int FK>
__device__ __forceinline__ void walk_pair(const WalkPair &w, const Geom &g, const DerivIn &in, int a,
                                          int sub, float (&v)[n_sums<K>()]) {
  constexpr int DEG = 4;
  constexpr int NM = n_mom<K, DEG>();
  constexpr int NV = n_sums<K>();
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = 0.f;
  const float4 q = w.q, u = w.v;
  const int4 box = w.box;
  const float I = w.r.w;
  const bool l2atom = FK == kFieldAny ? in.mode == kModeL2Atom : FK == kFieldL2Atom;
  const bool bfield = FK == kFieldAny ? in.beta != nullptr : FK == kFieldBeta;
  const int D0 = g.ax[0].n, D1 = K == 2 ? g.ax[1].n : 1;
  const float *__restrict__ x0 = g.ax[0].coords;
  const F2 nqh = f2(q.x, q.x), nql = f2(q.y, q.y), g00 = f2(u.x, u.x);
  F2 X0 = f2(0.f, 0.f), Y0 = X0;
  if constexpr (K == 1) {
    const float *__restrict__ fa = in.alpha + (size_t)a * D0;
    const float *__restrict__ fb = bfield ? in.beta + (size_t)a * D0 : fa;
    F2 Sa[DEG + 1], Sb[DEG + 1];
#pragma unroll
    for (int e = 0; e <= DEG; ++e) {
      Sa[e] = f2(0.f, 0.f);
      Sb[e] = f2(0.f, 0.f);
    }
    auto cells = [&](float xa, float xb, float ca, float cb, float ba, float bb, bool two) {
      const F2 d0 = f2_add(f2_add(f2(xa, xb), nqh), nql);
      walk_cells(f2_mul(f2_mul(g00, d0), d0), d0, true, two, f2(ca, cb), f2(ba, bb), u.w, I, l2atom,
                          bfield, Sa, Sb, X0, Y0);
    };
    for (int k = box.x + sub; k <= box.y; k += GL * R) {
      if (k + (R - 1) * GL < D0) {
        float c[R], b[R], x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          c[i] = __ldg(fa + k + i * GL);
          x[i] = __ldg(x0 + k + i * GL);
          b[i] = bfield ? __ldg(fb + k + i * GL) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < R; i += 2)
          cells(x[i], x[i + 1], c[i], c[i + 1], b[i], b[i + 1], true);
      } else {
        for (int kk = k; kk <= box.y; kk += GL) {
          const float c = __ldg(fa + kk), x = __ldg(x0 + kk), b = bfield ? __ldg(fb + kk) : 0.f;
          cells(x, x, c, c, b, b, false);
        }
      }
    }
#pragma unroll
    for (int e = 0; e <= DEG; ++e) {
      v[e] = f2_sum(Sa[e]);
      v[NM + e] = f2_sum(Sb[e]);
    }
  } else {
    const size_t abase = (size_t)a * D0 * D1;
    for (int c0 = box.z; c0 <= box.w; c0 += GL) {
      // rows that the ellipse reaches in columns c0 .. c0 + GL - 1, the same
      // for every lane of the group so that its loads share sectors: the
      // row range at the column nearest to the ellipse's lowest (highest)
      // point, widened like the support box
      const int cz = min(c0 + GL - 1, box.w), col = min(c0 + sub, box.w);
      const float da = (__ldg(g.ax[1].coords + c0) + q.z) + q.w;
      const float db = (__ldg(g.ax[1].coords + cz) + q.z) + q.w;
      const float d1 = (__ldg(g.ax[1].coords + col) + q.z) + q.w;
      const float low = w.e.y;
      const float dh = fminf(fmaxf(-low, da), db), dl = fminf(fmaxf(low, da), db);
      const float hh = sqrtf(fmaxf(fmaf(-w.e.x * dh, dh, u.x), 0.f));
      const float hl = sqrtf(fmaxf(fmaf(-w.e.x * dl, dl, u.x), 0.f));
      const float rhi = fmaf(hh * w.r.z, 1.0001f, fmaf(-w.r.y, dh, w.r.x)) + 0.02f;
      const float rlo = fmaf(hl * w.r.z, -1.0001f, fmaf(-w.r.y, dl, w.r.x)) - 0.02f;
      const int r_lo = (int)fminf(fmaxf(ceilf(rlo), (float)box.x), (float)box.y + 1.f);
      const int r_hi = (int)fmaxf(fminf(floorf(rhi), (float)box.y), (float)box.x - 1.f);
      const bool mine = c0 + sub <= box.w;
      // (a lane past the last column repeats it, cut off)
      const float c1 = u.y * d1, b1 = mine ? u.z * d1 * d1 : 4.f + u.z * d1 * d1 + c1 * c1 / u.x;
      const F2 c1p = f2(c1, c1), b1p = f2(b1, b1);
      const float *__restrict__ fa = in.alpha + abase + (size_t)r_lo * D1 + col;
      const float *__restrict__ fb = bfield ? in.beta + abase + (size_t)r_lo * D1 + col : fa;
      F2 Sa[DEG + 1], Sb[DEG + 1];
#pragma unroll
      for (int e = 0; e <= DEG; ++e) {
        Sa[e] = f2(0.f, 0.f);
        Sb[e] = f2(0.f, 0.f);
      }
      auto cells = [&](float xa, float xb, float ca, float cb, float ba, float bb, bool two) {
        const F2 d0 = f2_add(f2_add(f2(xa, xb), nqh), nql);
        walk_cells(f2_fma(d0, f2_fma(g00, d0, c1p), b1p), d0, true, two, f2(ca, cb), f2(ba, bb), u.w, I, l2atom,
                            bfield, Sa, Sb, X0, Y0);
      };
      for (int k = r_lo; k <= r_hi; k += R) {
        if (k + R <= D0) {
          float c[R], b[R], x[R];
#pragma unroll
          for (int i = 0; i < R; ++i) {
            c[i] = __ldg(fa);
            b[i] = bfield ? __ldg(fb) : 0.f;
            x[i] = __ldg(x0 + k + i);
            fa += D1;
            if (bfield) fb += D1;
          }
#pragma unroll
          for (int i = 0; i < R; i += 2)
            cells(x[i], x[i + 1], c[i], c[i + 1], b[i], b[i + 1], true);
        } else {
          for (int kk = k; kk <= r_hi; ++kk) {
            const float c = __ldg(fa), x = __ldg(x0 + kk), b = bfield ? __ldg(fb) : 0.f;
            cells(x, x, c, c, b, b, false);
            fa += D1;
            if (bfield) fb += D1;
          }
        }
      }
      // fold the column's sums with powers of d1
      float pw = 1.f;
#pragma unroll
      for (int e = 0; e <= DEG; ++e) {
#pragma unroll
        for (int i = 0; i <= DEG - e; ++i) {
          v[mi(i, e)] = fmaf(pw, f2_sum(Sa[i]), v[mi(i, e)]);
          v[NM + mi(i, e)] = fmaf(pw, f2_sum(Sb[i]), v[NM + mi(i, e)]);
        }
        pw *= d1;
      }
    }
  }
  v[NV - 2] = f2_sum(X0);
  v[NV - 1] = f2_sum(Y0);
}

// ONE: the work split gives every lane at most one angle of its atom (every
// Hessian split of up to ~32 angles per chunk, which covers the tilt series
// and the served fits): the angle loop runs at most once, so the per-lane
// accumulators need not live across the whole pair computation.
// The body of one block whose first warp is warp0 of the launch's warps
// (warp w takes the w-th (atom group, angle chunk); a multi-problem launch
// maps its blocks to (problem, first warp)).  What a warp computes depends on
// its warp index only, so the block size changes no result.
// smem: the warp's own staging area.
template <int K, bool ONE, int GL, int R, int FK>
__device__ __forceinline__ void hess_body(const Atoms &at, const Geom &g, const DerivIn &in,
                                           const DerivCfg &cfg, float *part, int warp0,
                                           WalkSmem<K> &sm) {
  constexpr int PR = n_rparam<K>();
  constexpr int P = n_par<K>();
  constexpr int NPSI = n_psi<K>();
  constexpr int DEG = 4;
  constexpr int NM = n_mom<K, DEG>();
  constexpr int NV = n_sums<K>();
  constexpr int NH = P * (P + 1) / 2;
  constexpr int NG = 32 / GL;                    // groups of a warp
  const int gw = warp0 + ((int)threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int warps_atoms = (at.n + cfg.ag - 1) / cfg.ag;
  if (gw >= warps_atoms * cfg.nchunks) return;
  const int chunk = gw / warps_atoms, wa = gw - chunk * warps_atoms;
  const int j = wa * cfg.ag + (lane & (cfg.ag - 1));   // slot
  const int sub = lane / cfg.ag;
  const bool valid = j < at.n;
  const int jj = valid ? (at.order ? at.order[j] : j) : 0;  // atom of the slot
  const float I = at.I[jj];
  const int a_lo = chunk * cfg.ch;
  const int a_hi = min(g.n_angles, a_lo + cfg.ch);

  float f = 0.f;
  CAcc gacc[P];
  float hacc[NH];
#pragma unroll
  for (int i = 0; i < P; ++i) gacc[i].zero();
#pragma unroll
  for (int i = 0; i < NH; ++i) hacc[i] = 0.f;

  // the warp's first 32 / rs lanes have a pair each (atom lane % ag, angle
  // a0 + lane / ag); small problems give a warp fewer pairs than lanes
  const int npairs = 32 / cfg.rs, astep = cfg.sg / cfg.rs;
  for (int a0 = a_lo; a0 < a_hi; a0 += astep) {
    const int a = a0 + sub;
    const bool mine = valid && lane < npairs && a < a_hi;
    Frame<K> fr;
    Pair<K> p;
    if (mine) {
      load_frame<K>(g.frames, a, fr);
      pair_setup<K>(at, jj, fr, g, p);
      walk_stage<K>(p, g, I, sm.pair[lane]);
    } else {
      sm.pair[lane].box = make_int4(1, 0, 1, 0);
    }
    __syncwarp();
    const bool narrow =
        cfg.rs == 1 && __all_sync(0xffffffffu, !mine || (p.hi[0] - p.lo[0] < walk_narrow_of<K>() &&
                                                         p.hi[K - 1] - p.lo[K - 1] < walk_narrow_of<K>()));
    if (narrow) {
      float v[NV];
      walk_pair<K, 1, 2, FK>(sm.pair[lane], g, in, a, 0, v);
#pragma unroll
      for (int k = 0; k < NV; ++k) sm.sum[lane][k] = v[k];
    }
    for (int s0 = narrow ? npairs : 0; s0 < npairs; s0 += NG) {
      const int s = s0 + lane / GL, gl = lane % GL;
      float v[NV];
      walk_pair<K, GL, R, FK>(sm.pair[s < 32 ? s : 31], g, in, a0 + s / cfg.ag, gl, v);
      __syncwarp();
      // the group's lanes: each ends with the sums of NV / GL of the values
      int n = NV, first = 0;
#pragma unroll
      for (int m = GL / 2; m >= 1; m >>= 1) {
        n /= 2;
        const bool up = (gl & m) != 0;
        if (up) first += n;
#pragma unroll
        for (int k = 0; k < NV / 2; ++k)
          if (k < n) {
            const float keep = up ? v[k + n] : v[k];
            const float give = up ? v[k] : v[k + n];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, give, m);
          }
      }
#pragma unroll
      for (int k = 0; k < NV / GL; ++k) sm.sum[s < 32 ? s : 31][first + k] = v[k];
    }
    __syncwarp();
    if (mine) {
      float Ma[NM], Mb[NM];
#pragma unroll
      for (int q = 0; q < NM; ++q) {
        Ma[q] = sm.sum[lane][q];
        Mb[q] = in.beta ? sm.sum[lane][NM + q] : in.beta_const * sm.sum[lane][NM + q];
      }
      float Aa[NPSI];
      first_psi<K, NM>(Ma, p.G, Aa);
      // value
      if (in.mode == kModeInner) f += I * Ma[0];
      else if (in.mode == kModeL2Atom)
        f += I * (0.5f * I * sm.sum[lane][NV - 1] - sm.sum[lane][NV - 2]);
      float Ba[NPSI][NPSI], Bb[NPSI][NPSI];
      psi_gram<K, true>(Ma, p.G, Ba);
      psi_gram<K, false>(Mb, p.G, Bb);
      accumulate_pair<K, 2>(p, fr, I, Aa, Ba, Bb, gacc, hacc);
    }
    if constexpr (ONE) break;
    __syncwarp();
  }

  // combine lanes sharing an atom, then write
  float vals_f = f;
  float gv[P];
#pragma unroll
  for (int i = 0; i < P; ++i) gv[i] = gacc[i].get();
  if (cfg.ag == 1) {
    // one atom per warp: a reduce-scatter leaves the warp sum of value
    // 32 c + lane of the atom's qn values in lane `lane` (chunk c), so every
    // lane stores one value; a full butterfly of every value on every lane
    // would cost qn * 5 shuffles per lane instead of 31 per 32 values
    constexpr int QN = 1 + P + NH;
    constexpr int NC = (QN + 31) / 32;
    float *dst = part + (size_t)chunk * cfg.qn * at.n + j;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      float v[32];
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        const int q = 32 * c + k;
        v[k] = q == 0 ? vals_f : (q <= P ? gv[q - 1] : (q < QN ? hacc[q - 1 - P] : 0.f));
      }
      warp_reduce_scatter32(v, lane);
      const int q = 32 * c + lane;
      if (valid && q < QN) dst[(size_t)q * at.n] = v[0];
    }
    return;
  }
  for (int off = cfg.ag; off < 32; off <<= 1) {
    vals_f += __shfl_xor_sync(0xffffffffu, vals_f, off);
#pragma unroll
    for (int i = 0; i < P; ++i) gv[i] += __shfl_xor_sync(0xffffffffu, gv[i], off);
#pragma unroll
    for (int i = 0; i < NH; ++i) hacc[i] += __shfl_xor_sync(0xffffffffu, hacc[i], off);
  }
  if (!valid || sub != 0) return;
  const size_t N = at.n;
  float *dst = part + (size_t)chunk * cfg.qn * N + j;
  dst[0] = vals_f;
#pragma unroll
  for (int i = 0; i < P; ++i) dst[(1 + i) * N] = gv[i];
#pragma unroll
  for (int i = 0; i < NH; ++i) dst[(1 + P + i) * N] = hacc[i];
}

// One-warp blocks: a warp that finishes frees its slot at once; with four, a
// block holds its slot until its slowest warp (the one with the widest
// supports) is done, which lowers the resident warps of the register-limited
// Hessian kernels.
template <int K, bool ONE, int GL, int R, int FK>
__global__ void __launch_bounds__(32, hess_min_warps(K, ONE))
    gr_hess_kernel(Atoms at, Geom g, DerivIn in, DerivCfg cfg, float *part) {
  __shared__ WalkSmem<K> sm;
  hess_body<K, ONE, GL, R, FK>(at, g, in, cfg, part, (int)blockIdx.x, sm);
}

// ---- gradients: a lane per pair ------------------------------------------------
// A lane walks its pair's support alone: in 2D its cells, in 3D the rows of its
// ellipse.  A 3D pair holds 20 to 40 cells, which groups of 2, 4 or 8 lanes per
// pair, as the Hessians use, pad to 56 to 87 lane steps: 21.4, 21.2 and 24.5
// against 17.4 ms on 8192 atoms x 20000 orientations of 128^2.
//
// 2D: cells in chunks of CH, whose field values are loaded together.
template <int CH>
__device__ __forceinline__ void lane_cells(const Pair<1> &p, const Geom &g, const DerivIn &in, int a,
                                           float I, float (&Ma)[n_mom<1, 2>()], float &X0,
                                           float &Y0, int phase, int rs) {
  constexpr int NM = n_mom<1, 2>();
#pragma unroll
  for (int i = 0; i < NM; ++i) Ma[i] = 0.f;
  X0 = 0.f;
  Y0 = 0.f;
  if (p.lo[0] > p.hi[0]) return;
  const float l2n = lg2_approx(p.n);
  const float *__restrict__ field = in.alpha + (size_t)a * g.ax[0].n;
  // a cell's term: m its form, d its offset, c its field value
  auto cell = [&](float m, float d, float c) {
    if (m <= 1.f) {
      const float E = ex2_approx(fmaf(m, kNegThirtyLog2e, l2n));
      const float al = (in.mode == kModeL2Atom) ? fmaf(I, E, -c) : c;
      const float w = al * E;
      Ma[0] += w;
      Ma[1] = fmaf(w, d, Ma[1]);
      Ma[2] = fmaf(w, d * d, Ma[2]);
      if (in.mode == kModeL2Atom) {
        X0 = fmaf(E, c, X0);
        Y0 = fmaf(E, E, Y0);
      }
    }
  };
  const int c_hi = p.hi[0];
  for (int kb = p.lo[0] + phase * CH; kb <= c_hi; kb += rs * CH) {
    float cv[CH], pv[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      const int k0 = min(kb + i, c_hi);
      cv[i] = __ldg(field + k0);
      pv[i] = __ldg(g.ax[0].coords + k0);
    }
#pragma unroll
    for (int i = 0; i < CH; ++i) {
      if (kb + i > c_hi) break;
      const float d0 = (pv[i] - p.qh[0]) - p.ql[0];
      cell(p.G[0] * d0 * d0, d0, cv[i]);
    }
  }
}

// 3D: a row's cells in aligned fours of the field, in packed FP32 pairs.  The
// loads bound it: 32 lanes touch 32 lines of the field, one L1 tag each, so a load
// takes 16 bytes a lane (a four of 4-byte loads took four times the tags: 17.4 ms
// where this takes 12.7; a row's first four loaded a row ahead costs registers:
// 15.4 to 16.3).  The m <= 1 test decides every cell of a four.
//
// Rows that begin anywhere: fours are aligned in the whole field, two cells of a
// four at a time; a four that crosses an end of its row loads the row's cells one
// by one.
template <bool L2ATOM>
__device__ __forceinline__ void lane_rows(const Pair<2> &p, const Geom &g, const DerivIn &in, int a,
                                          float I, float (&Ma)[n_mom<2, 2>()], float &X0,
                                          float &Y0, int phase, int rs) {
  constexpr int NM = n_mom<2, 2>();
#pragma unroll
  for (int i = 0; i < NM; ++i) Ma[i] = 0.f;
  X0 = 0.f;
  Y0 = 0.f;
  if (p.lo[0] > p.hi[0] || p.lo[1] > p.hi[1]) return;
  const float l2n = lg2_approx(p.n);
  const int D0 = g.ax[0].n, D1 = g.ax[1].n;
  const float *__restrict__ x0 = g.ax[0].coords, *__restrict__ x1 = g.ax[1].coords;
  const float *__restrict__ field = in.alpha + (size_t)a * D0 * D1;
  const F2 nqh = f2(-p.qh[1], -p.qh[1]), nql = f2(-p.ql[1], -p.ql[1]);
  const F2 g2 = f2(p.G[2], p.G[2]), amp = f2(l2n, l2n);
  // per row, m <= 1 holds for d1 within hw(d0) = sqrt(G2 - d0^2 det)/G2 of
  // -G1 d0/G2: the walk visits that range (widened like the support box)
  // instead of the whole box; the m <= 1 test still decides every cell
  const float det = p.G[0] * p.G[2] - p.G[1] * p.G[1];
  const float iG2 = 1.f / p.G[2];
  const float rc0 = (p.qh[1] - g.ax[1].first) * g.ax[1].inv_step;
  const float rcd = p.G[1] * iG2 * g.ax[1].inv_step;
  const float rhs = iG2 * g.ax[1].inv_step * 1.0001f;
  for (int k0 = p.lo[0] + phase; k0 <= p.hi[0]; k0 += rs) {
    const float d0 = (__ldg(x0 + k0) - p.qh[0]) - p.ql[0];
    const float t0 = p.G[0] * d0 * d0, u = 2.f * p.G[1] * d0;
    const float rc = fmaf(-rcd, d0, rc0);
    const float rh = fmaf(sqrt_approx(fmaxf(fmaf(-d0 * d0, det, p.G[2]), 0.f)), rhs, 1e-3f);
    const int c_lo = (int)fminf(fmaxf(ceilf(rc - rh), (float)p.lo[1]), (float)p.hi[1] + 1.f);
    const int c_hi = (int)fmaxf(fminf(floorf(rc + rh), (float)p.hi[1]), (float)p.lo[1] - 1.f);
    if (c_lo > c_hi) continue;
    const float *__restrict__ row = field + (size_t)k0 * D1;
    const F2 t0p = f2(t0, t0), up = f2(u, u);
    F2 S0 = f2(0.f, 0.f), S1 = S0, S2 = S0, X = S0, Y = S0;
    // two cells: coordinates, field values, whether they are cells of the row
    auto cells = [&](F2 x, F2 c, bool in0, bool in1) {
      const F2 d = f2_add(f2_add(x, nqh), nql);
      const F2 m = f2_fma(d, f2_fma(g2, d, up), t0p);
      float m0, m1, e0, e1;
      f2_get(m, m0, m1);
      in0 = in0 && m0 <= 1.f;
      in1 = in1 && m1 <= 1.f;
      f2_get(f2_fma(m, f2(kNegThirtyLog2e, kNegThirtyLog2e), amp), e0, e1);
      const F2 E = f2(ex2_approx(e0), ex2_approx(e1));
      F2 al = c;
      if (L2ATOM) al = f2_fma(f2(I, I), E, f2_mul(c, f2(-1.f, -1.f)));
      // the product is cut off: a field value beyond the cut-off counts for
      // nothing, also one that is not finite
      const F2 w = f2_keep(f2_mul(al, E), in0, in1);
      S0 = f2_add(S0, w);
      const F2 wd = f2_mul(w, d);
      S1 = f2_add(S1, wd);
      S2 = f2_fma(wd, d, S2);
      if (L2ATOM) {
        X = f2_add(X, f2_keep(f2_mul(E, c), in0, in1));
        Y = f2_add(Y, f2_keep(f2_mul(E, E), in0, in1));
      }
    };
    // cells before c_lo down to a 16-byte boundary
    const int back = (int)((reinterpret_cast<size_t>(row + c_lo) >> 2) & 3);
    for (int kb = c_lo - back; kb <= c_hi; kb += 4) {
      if (kb >= 0 && kb + 4 <= D1) {
        const float4 c = __ldg(reinterpret_cast<const float4 *>(row + kb));
        const float *x = x1 + kb;
        cells(f2(__ldg(x), __ldg(x + 1)), f2(c.x, c.y), true, true);
        cells(f2(__ldg(x + 2), __ldg(x + 3)), f2(c.z, c.w), true, true);
      } else {
        // a four that crosses an end of the row: the row's cells only
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const int ka = kb + i, ia = min(max(ka, 0), D1 - 1), ib = min(max(ka + 1, 0), D1 - 1);
          cells(f2(__ldg(x1 + ia), __ldg(x1 + ib)), f2(__ldg(row + ia), __ldg(row + ib)),
                ka == ia, ka + 1 == ib);
        }
      }
    }
    const float S[3] = {f2_sum(S0), f2_sum(S1), f2_sum(S2)};
    if (L2ATOM) {
      X0 += f2_sum(X);
      Y0 += f2_sum(Y);
    }
    float pw = 1.f;
#pragma unroll
    for (int i = 0; i <= 2; ++i) {
#pragma unroll
      for (int j = 0; j <= 2 - i; ++j) Ma[mi(i, j)] = fmaf(pw, S[j], Ma[mi(i, j)]);
      pw *= d0;
    }
  }
}

// Rows that begin on fours (D1 a multiple of four, field and coordinates on 16
// bytes): two rows at a time, a row per half of a register pair, over the union of
// their ranges, so that coordinates and a load's latency are shared by two (8192
// atoms x 20000 x 128^2: 12.7 ms, 13.5 a row at a time; 4096 x 121 x 256^2: 59 and
// 64 us).
template <bool L2ATOM>
__device__ __forceinline__ void lane_row_pairs(const Pair<2> &p, const Geom &g, const DerivIn &in,
                                               int a, float I, float (&Ma)[n_mom<2, 2>()],
                                               float &X0, float &Y0, int phase, int rs) {
  constexpr int NM = n_mom<2, 2>();
#pragma unroll
  for (int i = 0; i < NM; ++i) Ma[i] = 0.f;
  X0 = 0.f;
  Y0 = 0.f;
  if (p.lo[0] > p.hi[0] || p.lo[1] > p.hi[1]) return;
  const float l2n = lg2_approx(p.n);
  const int D1 = g.ax[1].n;
  const float *__restrict__ x0 = g.ax[0].coords, *__restrict__ x1 = g.ax[1].coords;
  const float *__restrict__ field = in.alpha + (size_t)a * g.ax[0].n * D1;
  const F2 K2 = f2(kNegThirtyLog2e, kNegThirtyLog2e), amp = f2(l2n, l2n);
  // (the rows' ranges as in lane_rows)
  const float det = p.G[0] * p.G[2] - p.G[1] * p.G[1];
  const float iG2 = 1.f / p.G[2];
  const float rc0 = (p.qh[1] - g.ax[1].first) * g.ax[1].inv_step;
  const float rcd = p.G[1] * iG2 * g.ax[1].inv_step;
  const float rhs = iG2 * g.ax[1].inv_step * 1.0001f;
  const float c_min = (float)p.lo[1], c_max = (float)p.hi[1];
  for (int k0 = p.lo[0] + 2 * phase; k0 <= p.hi[0]; k0 += 2 * rs) {
    const bool two = k0 < p.hi[0];
    const float da = (__ldg(x0 + k0) - p.qh[0]) - p.ql[0];
    const float db = (__ldg(x0 + k0 + (two ? 1 : 0)) - p.qh[0]) - p.ql[0];
    const float ra = fmaf(-rcd, da, rc0), rb = fmaf(-rcd, db, rc0);
    const float ha = fmaf(sqrt_approx(fmaxf(fmaf(-da * da, det, p.G[2]), 0.f)), rhs, 1e-3f);
    const float hb = fmaf(sqrt_approx(fmaxf(fmaf(-db * db, det, p.G[2]), 0.f)), rhs, 1e-3f);
    const int c_lo = (int)fmaxf(ceilf(fminf(ra - ha, rb - hb)), c_min);
    const int c_hi = (int)fminf(floorf(fmaxf(ra + ha, rb + hb)), c_max);
    // (a row past the support: no cell of it is within)
    const F2 t0 = f2(p.G[0] * da * da, two ? p.G[0] * db * db : 4.f);
    const F2 u = f2(2.f * p.G[1] * da, two ? 2.f * p.G[1] * db : 0.f);
    const float *__restrict__ row = field + (size_t)k0 * D1;
    const int to_b = two ? D1 : 0;
    F2 S0 = f2(0.f, 0.f), S1 = S0, S2 = S0, X = S0, Y = S0;
    for (int kb = c_lo & ~3; kb <= c_hi; kb += 4) {
      const float4 ca = __ldg(reinterpret_cast<const float4 *>(row + kb));
      const float4 cb = __ldg(reinterpret_cast<const float4 *>(row + kb + to_b));
      const float4 xv = __ldg(reinterpret_cast<const float4 *>(x1 + kb));
      auto column = [&](float x, float fa, float fb) {
        const float d = (x - p.qh[1]) - p.ql[1];
        const float gd = p.G[2] * d;
        const F2 D = f2(d, d);
        const F2 m = f2_fma(D, f2_add(f2(gd, gd), u), t0);
        float m0, m1, e0, e1;
        f2_get(m, m0, m1);
        f2_get(f2_fma(m, K2, amp), e0, e1);
        const F2 E = f2(ex2_approx(e0), ex2_approx(e1)), c = f2(fa, fb);
        const bool in0 = m0 <= 1.f, in1 = m1 <= 1.f;
        F2 al = c;
        if (L2ATOM) al = f2_fma(f2(I, I), E, f2_mul(c, f2(-1.f, -1.f)));
        const F2 w = f2_keep(f2_mul(al, E), in0, in1);
        S0 = f2_add(S0, w);
        const F2 wd = f2_mul(w, D);
        S1 = f2_add(S1, wd);
        S2 = f2_fma(wd, D, S2);
        if (L2ATOM) {
          X = f2_add(X, f2_keep(f2_mul(E, c), in0, in1));
          Y = f2_add(Y, f2_keep(f2_mul(E, E), in0, in1));
        }
      };
      column(xv.x, ca.x, cb.x);
      column(xv.y, ca.y, cb.y);
      column(xv.z, ca.z, cb.z);
      column(xv.w, ca.w, cb.w);
    }
    if (L2ATOM) {
      X0 += f2_sum(X);
      Y0 += f2_sum(Y);
    }
    float s0a, s0b, s1a, s1b;
    f2_get(S0, s0a, s0b);
    f2_get(S1, s1a, s1b);
    Ma[mi(0, 0)] += s0a + s0b;
    Ma[mi(0, 1)] += s1a + s1b;
    Ma[mi(0, 2)] += f2_sum(S2);
    Ma[mi(1, 1)] += fmaf(da, s1a, db * s1b);
    const float w0a = da * s0a, w0b = db * s0b;
    Ma[mi(1, 0)] += w0a + w0b;
    Ma[mi(2, 0)] += fmaf(da, w0a, db * w0b);
  }
}

template <int K>
struct FramesOf { using type = FrameSmem; };
template <>
struct FramesOf<1> { using type = int; };  // (2D: not used)

// ONE, one-warp blocks: as gr_hess_kernel.  QUAD, L2ATOM: 3D only (2D reads the
// mode from `in`).  Row pairs take 28 warps an SM (72 registers: tilt series of 4096
// x 121 x 256^2 59.3 us, 63.0 with 32 warps), single rows 32 (1000 x 1001 x 95^2:
// 88.4 us, 91.0 with 28).
template <int K, bool ONE, bool QUAD, bool L2ATOM>
__global__ void __launch_bounds__(32, QUAD ? 28 : 32)
    gr_grad_kernel(Atoms at, Geom g, DerivIn in, DerivCfg cfg, float *part) {
  constexpr int P = n_par<K>();
  constexpr int NM = n_mom<K, 2>();
  constexpr int NPSI = n_psi<K>();
  __shared__ typename FramesOf<K>::type s_frames;
  const int gw = blockIdx.x, lane = threadIdx.x;
  const int warps_atoms = (at.n + cfg.ag - 1) / cfg.ag;
  const int chunk = gw / warps_atoms, wa = gw - chunk * warps_atoms;
  const int j = wa * cfg.ag + (lane % cfg.ag);   // slot
  const int sub = lane / cfg.ag;
  const bool valid = j < at.n;
  const int jj = valid ? (at.order ? at.order[j] : j) : 0;  // atom of the slot
  const float I = at.I[jj];
  const int a_lo = chunk * cfg.ch;
  const int a_hi = min(g.n_angles, a_lo + cfg.ch);
  float f = 0.f, none[1];
  CAcc gacc[P];
#pragma unroll
  for (int i = 0; i < P; ++i) gacc[i].zero();
  // lanes sharing a pair (cfg.rs of them, sub = s rs + phase) walk its rows
  // (2D: chunks) phase, phase + rs, ... and combine their moment sums
  const int phase = sub & (cfg.rs - 1);
  unsigned gmask = 0u;
  for (int o = 0; o < cfg.rs; ++o) gmask |= 1u << (lane + (o - phase) * cfg.ag);
  // angle a (3D: frame i of the staged)
  auto add_pair = [&](int a, int i) {
    Frame<K> fr;
    if constexpr (K == 2) load_frame(s_frames, i, fr);
    else load_frame<K>(g.frames, a, fr);
    Pair<K> p;
    pair_setup<K, K == 2>(at, jj, fr, g, p);
    float Ma[NM], X0, Y0;
    if constexpr (K == 1) lane_cells<8>(p, g, in, a, I, Ma, X0, Y0, phase, cfg.rs);
    else if constexpr (QUAD) lane_row_pairs<L2ATOM>(p, g, in, a, I, Ma, X0, Y0, phase, cfg.rs);
    else lane_rows<L2ATOM>(p, g, in, a, I, Ma, X0, Y0, phase, cfg.rs);
    for (int o = 1; o < cfg.rs; o <<= 1) {
#pragma unroll
      for (int q = 0; q < NM; ++q) Ma[q] += __shfl_xor_sync(gmask, Ma[q], o * cfg.ag);
      X0 += __shfl_xor_sync(gmask, X0, o * cfg.ag);
      Y0 += __shfl_xor_sync(gmask, Y0, o * cfg.ag);
    }
    if (phase == 0) {
      if constexpr (K == 2) {  // (read again rather than held over the walk)
        asm volatile("" ::: "memory");
        load_frame(s_frames, i, fr);
      }
      float Aa[NPSI], Z[NPSI][NPSI];
      first_psi<K, NM>(Ma, p.G, Aa);
      if (in.mode == kModeInner) f += I * Ma[0];
      else if (in.mode == kModeL2Atom) f += I * (0.5f * I * Y0 - X0);
      accumulate_pair<K, 1>(p, fr, I, Aa, Z, Z, gacc, none);
    }
  };
  const int astep = cfg.sg / cfg.rs;
  if constexpr (K == 1) {
    for (int a = a_lo + sub / cfg.rs; a < a_hi && valid; a += astep) {
      add_pair(a, 0);
      if constexpr (ONE) break;
    }
  } else {
    for (int a0 = a_lo; a0 < a_hi; a0 += astep) {
      stage_frames(s_frames, g.frames + (size_t)a0 * kFrameStride3D, min(astep, a_hi - a0));
      __syncwarp();
      const int i = sub / cfg.rs;
      if (valid && a0 + i < a_hi) add_pair(a0 + i, i);
      if constexpr (ONE) break;
      __syncwarp();
    }
  }
  // combine lanes sharing an atom, then write
  float gv[P];
#pragma unroll
  for (int i = 0; i < P; ++i) gv[i] = gacc[i].get();
  if constexpr (K == 2) {
    if (cfg.ag == 1) {
      // one atom per warp: halve the 16 values held over four exchanges, then one
      // more sums each (16 shuffles, not five for each of the 11 values)
      float v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = k == 0 ? f : (k <= P ? gv[k - 1] : 0.f);
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) {
        const bool up = lane & (2 * w);
#pragma unroll
        for (int k = 0; k < w; ++k) {
          const float keep = up ? v[w + k] : v[k], give = up ? v[k] : v[w + k];
          v[k] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * w);
        }
      }
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
      const int q = lane >> 1;
      if (valid && (lane & 1) == 0 && q <= P) part[((size_t)chunk * cfg.qn + q) * at.n + j] = v[0];
      return;
    }
  }
  for (int off = cfg.ag; off < 32; off <<= 1) {
    f += __shfl_xor_sync(0xffffffffu, f, off);
#pragma unroll
    for (int i = 0; i < P; ++i) gv[i] += __shfl_xor_sync(0xffffffffu, gv[i], off);
  }
  if (!valid || sub != 0) return;
  const size_t N = at.n;
  float *dst = part + (size_t)chunk * cfg.qn * N + j;
  dst[0] = f;
#pragma unroll
  for (int i = 0; i < P; ++i) dst[(1 + i) * N] = gv[i];
}

// Pixel-integrated operator: per cell, the quadrature points' moments give
// the cell's value R = I s sum E and its psi-space derivative sums
// A_cell = s first_psi(M), BC_cell = s psi_gram(M) (the quadrature points
// are fixed, as in the reference's __drf2/__drf3, which also give the
// "total mass" cells zero derivatives).  The pair's sums
//   Sa = sum alpha A_cell, Ta = sum alpha BC_cell, Ub = sum beta A_cell A_cell^T
// feed the same chain-rule assembly as the point-sampled kernel.
// A block's 32 pairs: the sums over an atom's pairs, in angle order, as FP32 pairs
// (a Hessian's 28 or 66 values in FP64 held the SM's FP64 pipe for half of the time
// of 2154 x 736 narrow pairs: 243 and 119 us).
template <int QN>
__device__ __forceinline__ void psf_close(const float (*vals)[QN + 1], int n_atoms,
                                          const DerivCfg &cfg, int chunk, int wa, float *part) {
  for (int e = threadIdx.x; e < cfg.ag * QN; e += blockDim.x) {
    const int t = e / QN, q = e - t * QN;
    if (wa * cfg.ag + t >= n_atoms) continue;
    float v = 0.f, c = 0.f;
    for (int k = 0; k < cfg.sg; ++k) pair_add(v, c, vals[t + k * cfg.ag][q], 0.f);
    part[((size_t)chunk * cfg.qn + q) * n_atoms + wa * cfg.ag + t] = v + c;
  }
}

// 2D: a block takes 32 (atom, angle) pairs at a time (as a warp of the other
// kernels does), L lanes each, which share the pair's few cells (11 points
// each); a pair's first lane assembles, and the block adds its pairs' values per
// atom.
template <int ORDER, int L>
__global__ void __launch_bounds__(32 * L)
    gr_psf_deriv1d_kernel(Atoms at, Geom g, DerivIn in, DerivCfg cfg, float *part, float s) {
  constexpr int K = 1;
  constexpr int P = n_par<K>();
  constexpr int NPSI = n_psi<K>();
  constexpr int DEG = ORDER == 1 ? 2 : 4;
  constexpr int NM = n_mom<K, DEG>();
  constexpr int NH = P * (P + 1) / 2;
  constexpr int QN = 1 + P + (ORDER > 1 ? NH : 0);
  constexpr int NT = ORDER > 1 ? NPSI * (NPSI + 1) / 2 : 1;   // upper triangles
  __shared__ float vals[32][QN + 1];
  const int gw = blockIdx.x;
  const int pr = threadIdx.x / L, gl = threadIdx.x % L;
  const unsigned gmask = ((1u << L) - 1u) << ((threadIdx.x & 31) & ~(L - 1));
  const int warps_atoms = (at.n + cfg.ag - 1) / cfg.ag;
  const int chunk = gw / warps_atoms, wa = gw - chunk * warps_atoms;
  const int j = wa * cfg.ag + (pr % cfg.ag);   // slot
  const int sub = pr / cfg.ag;
  const bool valid = j < at.n;
  const int jj = valid ? (at.order ? at.order[j] : j) : 0;  // atom of the slot
  const float I = at.I[jj];
  const int a_lo = chunk * cfg.ch;
  const int a_hi = min(g.n_angles, a_lo + cfg.ch);
  const int D0 = g.ax[0].n;

  float f = 0.f;
  CAcc gacc[P];
  float hacc[ORDER > 1 ? NH : 1];
#pragma unroll
  for (int i = 0; i < P; ++i) gacc[i].zero();
#pragma unroll
  for (int i = 0; i < (ORDER > 1 ? NH : 1); ++i) hacc[i] = 0.f;

  for (int a = a_lo + sub; a < a_hi && valid; a += cfg.sg) {
    Frame<K> fr;
    load_frame<K>(g.frames, a, fr);
    Pair<K> p;
    const bool ok = pair_setup<K>(at, jj, fr, g, p);
    PsfPair<K> q;
    psf_setup<K>(at, jj, g, p, ok, s, q);
    const float l2n = lg2_approx(p.n);
    float Sa[NPSI], Tt[NT], Ut[NT], fa = 0.f;
#pragma unroll
    for (int k = 0; k < NPSI; ++k) Sa[k] = 0.f;
#pragma unroll
    for (int k = 0; k < NT; ++k) Tt[k] = Ut[k] = 0.f;
    for (int k0 = q.lo[0] + gl; k0 <= q.hi[0]; k0 += L) {
      float dc[K], base[K], step[K];
      dc[0] = (__ldg(g.ax[0].coords + k0) - p.qh[0]) - p.ql[0];
      const int kind = psf_cell_kind<K>(q, dc, s, base, step);
      if (kind == 0) continue;
      const size_t gi = (size_t)a * D0 + k0;
      const float c = __ldg(in.alpha + gi);
      if (kind == 1) {
        const float R = q.total;
        if (in.mode == kModeInner) fa = fmaf(c, R, fa);
        else if (in.mode == kModeL2Atom) fa += R * (0.5f * R - c);
        continue;
      }
      float M[NM];
#pragma unroll
      for (int i = 0; i < NM; ++i) M[i] = 0.f;
#pragma unroll
      for (int t = 1; t <= 11; ++t) {
        const float d = fmaf((float)t, step[0], base[0]);
        float w = ex2_approx(fmaf(p.G[0] * d * d, kNegThirtyLog2e, l2n));
#pragma unroll
        for (int i = 0; i < NM; ++i) {
          M[i] += w;
          w *= d;
        }
      }
      const float scale = 10.f * step[0] / 11.f;
      const float R = I * scale * M[0];
      float al, be;
      if (in.mode == kModeInner) {
        al = c;
        be = 0.f;
        fa = fmaf(c, R, fa);
      } else if (in.mode == kModeL2Atom) {
        al = R - c;
        be = 1.f;
        fa += R * (0.5f * R - c);
      } else {
        al = c;
        be = in.beta ? __ldg(in.beta + gi) : in.beta_const;
      }
      float A[NPSI];
      first_psi<K, NM>(M, p.G, A);
#pragma unroll
      for (int k = 0; k < NPSI; ++k) {
        A[k] *= scale;
        Sa[k] = fmaf(al, A[k], Sa[k]);
      }
      if constexpr (ORDER > 1) {
        float BC[NPSI][NPSI];
        psi_gram<K, true>(M, p.G, BC);
        const float as = al * scale;
        int o = 0;
#pragma unroll
        for (int k = 0; k < NPSI; ++k)
#pragma unroll
          for (int l = k; l < NPSI; ++l, ++o) {
            Tt[o] = fmaf(as, BC[k][l], Tt[o]);
            Ut[o] = fmaf(be * A[k], A[l], Ut[o]);
          }
      }
    }
    __syncwarp(gmask);
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      fa += __shfl_xor_sync(gmask, fa, o);
#pragma unroll
      for (int k = 0; k < NPSI; ++k) Sa[k] += __shfl_xor_sync(gmask, Sa[k], o);
      if constexpr (ORDER > 1) {
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          Tt[k] += __shfl_xor_sync(gmask, Tt[k], o);
          Ut[k] += __shfl_xor_sync(gmask, Ut[k], o);
        }
      }
    }
    if (gl == 0) {
      f += fa;
      float Ta[NPSI][NPSI], Ub[NPSI][NPSI];
      if constexpr (ORDER > 1) {
        int o = 0;
#pragma unroll
        for (int k = 0; k < NPSI; ++k)
#pragma unroll
          for (int l = k; l < NPSI; ++l, ++o) {
            Ta[k][l] = Ta[l][k] = Tt[o];
            Ub[k][l] = Ub[l][k] = Ut[o];
          }
      }
      accumulate_pair<K, ORDER>(p, fr, I, Sa, Ta, Ub, gacc, hacc);
    }
  }

  if (gl == 0) {
    vals[pr][0] = f;
#pragma unroll
    for (int i = 0; i < P; ++i) vals[pr][1 + i] = gacc[i].get();
    if constexpr (ORDER > 1) {
#pragma unroll
      for (int i = 0; i < NH; ++i) vals[pr][1 + P + i] = hacc[i];
    }
  }
  __syncthreads();
  psf_close<QN>(vals, at.n, cfg, chunk, wa, part);
}

// 3D: a block takes 32 (atom, angle) pairs at a time, a warp PW of them.  The
// warp's lanes look over a pair's cell box and queue the cells it reaches; 32
// queued cells at a time, of as many pairs as that takes, are summed over their
// 121 points, two to a register pair (this bounds it), and reduced into shared
// memory.  A lane per pair sets up and assembles, and the block adds its pairs'
// values per atom.  128 atoms x 401 x 64^2, gradient: 163 us with a lane
// per pair, which walked some 40 cells in series on 10 warps an SM; 143 us with
// eight lanes a pair, 12 of 32 lanes at work; with the queue and PW = 8 69 us.
// Narrow supports are set-up and assembly above all, of which PW = 8 does four
// times the instructions (start_psf).

// From PW = 16 on: pairs whose boxes all have at most this many cells are looked over by their
// own lanes, all at a time, not one after the other (2366 atoms x 572 x 29^2, one or
// two cells a pair: gradient 410 -> 216 us; 1412 x 907 x 78^2, r = 35: 644 -> 414).
constexpr int kPsfNarrow = 16;
struct PsfWalk {
  float4 a, b;        // qh0 ql0 qh1 ql1; G00 G01 G11 log2 n
  float rr, total, I;
  int angle;
  int lo0, lo1, bw, ncell;
};

template <int ORDER, int PW>
__global__ void __launch_bounds__(1024 / PW, (ORDER == 1 ? 16 : 8) * PW / 32)
    gr_psf_deriv_kernel(Atoms at, Geom g, DerivIn in, DerivCfg cfg, float *part, float s) {
  constexpr int K = 2;
  constexpr int NW = 32 / PW;
  constexpr int P = n_par<K>();
  constexpr int NPSI = n_psi<K>();
  constexpr int DEG = ORDER == 1 ? 2 : 4;
  constexpr int NM = n_mom<K, DEG>();
  constexpr int NH = P * (P + 1) / 2;
  constexpr int QN = 1 + P + (ORDER > 1 ? NH : 0);
  constexpr int NT = ORDER > 1 ? NPSI * (NPSI + 1) / 2 : 0;   // upper triangles
  // a cell's sums: f, first order, second order against alpha and against beta
  constexpr int NV = (1 + NPSI + 2 * NT + 7) / 8 * 8;
  __shared__ PsfWalk s_walk[NW][PW];
  __shared__ int2 s_queue[NW][64];
  __shared__ float s_sum[NW][PW][NV + 1];
  __shared__ float vals[32][QN + 1];
  const int gw = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  PsfWalk *walk = s_walk[warp];
  int2 *queue = s_queue[warp];
  float(*sum)[NV + 1] = s_sum[warp];
  const int pr = warp * PW + (lane & (PW - 1));
  const int warps_atoms = (at.n + cfg.ag - 1) / cfg.ag;
  const int chunk = gw / warps_atoms, wa = gw - chunk * warps_atoms;
  const int j = wa * cfg.ag + (pr % cfg.ag);   // slot
  const int sub = pr / cfg.ag;
  const bool valid = lane < PW && j < at.n;
  const int jj = valid ? (at.order ? at.order[j] : j) : 0;  // atom of the slot
  const float I = at.I[jj];
  const int a_lo = chunk * cfg.ch;
  const int a_hi = min(g.n_angles, a_lo + cfg.ch);
  const int D0 = g.ax[0].n, D1 = g.ax[1].n;

  float f = 0.f;
  CAcc gacc[P];
  float hacc[ORDER > 1 ? NH : 1];
#pragma unroll
  for (int i = 0; i < P; ++i) gacc[i].zero();
#pragma unroll
  for (int i = 0; i < (ORDER > 1 ? NH : 1); ++i) hacc[i] = 0.f;

  // the first n queued cells
  auto add_cells = [&](int n) {
    const bool on = lane < n;
    const int2 it = queue[on ? lane : n - 1];
    const int slot = it.x & (PW - 1), k0 = it.x >> 5, k1 = it.y;
    const float4 wa4 = walk[slot].a, wb4 = walk[slot].b;
    const float Ij = walk[slot].I;
    float V[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) V[i] = 0.f;
    if (on) {
      Pair<K> p;
      p.G[0] = wb4.x;
      p.G[1] = wb4.y;
      p.G[2] = wb4.z;
      const float l2n = wb4.w;
      PsfPair<K> q;
      q.rr = walk[slot].rr;
      float dc[K], base[K], step[K];
      dc[0] = (__ldg(g.ax[0].coords + k0) - wa4.x) - wa4.y;
      dc[1] = (__ldg(g.ax[1].coords + k1) - wa4.z) - wa4.w;
      const int kind = psf_cell_kind<K>(q, dc, s, base, step);
      const size_t gi = ((size_t)walk[slot].angle * D0 + k0) * D1 + k1;
      const float c = __ldg(in.alpha + gi);
      if (kind == 1) {
        const float R = walk[slot].total;
        if (in.mode == kModeInner) V[0] = c * R;
        else if (in.mode == kModeL2Atom) V[0] = R * (0.5f * R - c);
      } else {
        // a row's points two at a time (packed FP32)
        float M[NM];
#pragma unroll
        for (int i = 0; i < NM; ++i) M[i] = 0.f;
        const PsfRow row(base[1], step[1], p.G[2], l2n);
#pragma unroll 1
        for (int t = 1; t <= 11; ++t) {
          const float d0 = fmaf((float)t, step[0], base[0]);
          const float t0 = p.G[0] * d0 * d0, u = 2.f * p.G[1] * d0;
          const F2 tp = f2(t0, t0), up = f2(u, u);
          F2 S2[DEG + 1];
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            F2 w = row.pair(v, up, tp);
#pragma unroll
            for (int i = 0; i <= DEG; ++i) {
              S2[i] = v == 0 ? w : f2_add(S2[i], w);
              if (i < DEG) w = f2_mul(w, row.d[v]);
            }
          }
          float w = row.end(u, t0);
          float S[DEG + 1];
#pragma unroll
          for (int i = 0; i <= DEG; ++i) {
            float x, y;
            f2_get(S2[i], x, y);
            S[i] = (x + y) + w;
            w *= row.last;
          }
          float pw = 1.f;
#pragma unroll
          for (int i = 0; i <= DEG; ++i) {
#pragma unroll
            for (int jx = 0; jx <= DEG - i; ++jx) M[mi(i, jx)] = fmaf(pw, S[jx], M[mi(i, jx)]);
            pw *= d0;
          }
        }
        const float scale = 100.f * step[0] * step[1] / 121.f;
        const float R = Ij * scale * M[0];
        float al, be;
        if (in.mode == kModeInner) {
          al = c;
          be = 0.f;
          V[0] = c * R;
        } else if (in.mode == kModeL2Atom) {
          al = R - c;
          be = 1.f;
          V[0] = R * (0.5f * R - c);
        } else {
          al = c;
          be = in.beta ? __ldg(in.beta + gi) : in.beta_const;
        }
        float A[NPSI];
        first_psi<K, NM>(M, p.G, A);
#pragma unroll
        for (int k = 0; k < NPSI; ++k) {
          A[k] *= scale;
          V[1 + k] = al * A[k];
        }
        if constexpr (ORDER > 1) {
          float BC[NPSI][NPSI];
          psi_gram<K, true>(M, p.G, BC);
          const float as = al * scale;
          int o = 1 + NPSI;
#pragma unroll
          for (int k = 0; k < NPSI; ++k)
#pragma unroll
            for (int l = k; l < NPSI; ++l, ++o) {
              V[o] = as * BC[k][l];
              V[NT + o] = be * A[k] * A[l];
            }
        }
      }
    }
    // into the pairs' sums: pair by pair, eight values at a time, the values held
    // halved over three exchanges, then the four lanes that hold the same one
    // summed.  More pairs than a pair has cells: the pairs' cells in turn, each lane
    // its own values (gradients with PW = 8 lose by the test, 116 and 122 us on
    // 128 x 401 x 64^2).
    int first, last;
    if constexpr (PW >= 16) {   // (the pairs of a batch may come in any order)
      first = __reduce_min_sync(0xffffffffu, slot);
      last = __reduce_max_sync(0xffffffffu, slot);
    } else {
      first = __shfl_sync(0xffffffffu, slot, 0);
      last = __shfl_sync(0xffffffffu, slot, 31);
    }
    if ((ORDER > 1 || PW >= 16) && last - first > 1) {
      const unsigned same = __match_any_sync(0xffffffffu, on ? slot : -1 - lane);
      const int rank = __popc(same & ((1u << lane) - 1u));
      const int turns = __reduce_max_sync(0xffffffffu, rank) + 1;
      if (turns <= last - first) {
        for (int k = 0; k < turns; ++k) {
          if (on && rank == k) {
#pragma unroll
            for (int i = 0; i < 1 + NPSI + 2 * NT; ++i) sum[slot][i] += V[i];
          }
          __syncwarp();
        }
        return;
      }
    }
    for (int sl = first; sl <= last; ++sl) {
      const bool mine = on && slot == sl;
      if (!__any_sync(0xffffffffu, mine)) continue;
#pragma unroll
      for (int v0 = 0; v0 < NV; v0 += 8) {
        float h[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = mine ? V[v0 + i] : 0.f;
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) {
          const bool up = lane & (4 * w);
#pragma unroll
          for (int i = 0; i < w; ++i) {
            const float keep = up ? h[w + i] : h[i], give = up ? h[i] : h[w + i];
            h[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * w);
          }
        }
        h[0] += __shfl_xor_sync(0xffffffffu, h[0], 2);
        h[0] += __shfl_xor_sync(0xffffffffu, h[0], 1);
        if ((lane & 3) == 0) sum[sl][v0 + (lane >> 2)] += h[0];
      }
    }
    __syncwarp();
  };

  const int steps = (a_hi - a_lo + cfg.sg - 1) / cfg.sg;
  for (int st = 0; st < steps; ++st) {
    const int a = a_lo + sub + st * cfg.sg;
    const bool on = valid && a < a_hi;
    Frame<K> fr;
    Pair<K> p;
    int ncell = 0;
    for (int i = lane; i < PW * (NV + 1); i += 32) (&sum[0][0])[i] = 0.f;
    if (on) {
      load_frame<K>(g.frames, a, fr);
      const bool ok = pair_setup<K>(at, jj, fr, g, p);
      PsfPair<K> q;
      psf_setup<K>(at, jj, g, p, ok, s, q);
      PsfWalk w;
      w.a = make_float4(p.qh[0], p.ql[0], p.qh[1], p.ql[1]);
      w.b = make_float4(p.G[0], p.G[1], p.G[2], lg2_approx(p.n));
      w.rr = q.rr;
      w.total = q.total;
      w.I = I;
      w.angle = a;
      w.lo0 = q.lo[0];
      w.lo1 = q.lo[1];
      w.bw = max(q.hi[1] - q.lo[1] + 1, 0);
      w.ncell = ncell = max(q.hi[0] - q.lo[0] + 1, 0) * w.bw;
      walk[lane] = w;
    }
    __syncwarp();
    int queued = 0;
    // the queued cells of all lanes, 32 at a time
    auto push = [&](bool hit, int2 cell) {
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) queue[queued + __popc(m & ((1u << lane) - 1u))] = cell;
      queued += __popc(m);
      __syncwarp();
      if (queued >= 32) {
        add_cells(32);
        queued -= 32;
        const int2 left = queue[32 + lane];
        __syncwarp();
        if (lane < queued) queue[lane] = left;
        __syncwarp();
      }
    };
    // narrow supports: a lane looks over its own pair's few cells
    const bool narrow = PW >= 16 && __reduce_max_sync(0xffffffffu, ncell) <= kPsfNarrow;
    if (narrow) {
      const int most = __reduce_max_sync(0xffffffffu, ncell);
      const PsfWalk w = walk[lane & (PW - 1)];
      PsfPair<K> q;
      q.rr = w.rr;
      int k0 = w.lo0, k1 = w.lo1;
      for (int e = 0; e < most; ++e) {
        bool hit = false;
        if (e < ncell) {
          float dc[K], base[K], step[K];
          dc[0] = (__ldg(g.ax[0].coords + k0) - w.a.x) - w.a.y;
          dc[1] = (__ldg(g.ax[1].coords + k1) - w.a.z) - w.a.w;
          hit = psf_cell_kind<K>(q, dc, s, base, step) != 0;
        }
        push(hit, make_int2(k0 << 5 | lane, k1));
        if (++k1 == w.lo1 + w.bw) {
          k1 = w.lo1;
          ++k0;
        }
      }
    }
    for (int sl = narrow ? PW : 0; sl < PW; ++sl) {
      const int nc = __shfl_sync(0xffffffffu, ncell, sl);
      if (nc == 0) continue;
      const PsfWalk w = walk[sl];
      PsfPair<K> q;
      q.rr = w.rr;
      const float inv_bw = 1.f / (float)w.bw;
      for (int e0 = 0; e0 < nc; e0 += 32) {
        const int e = e0 + lane;
        // (the estimate is within one for boxes below 2^23 cells a row)
        int row = (int)(((float)e + 0.5f) * inv_bw);
        if (row * w.bw > e) --row;
        if ((row + 1) * w.bw <= e) ++row;
        const int k0 = w.lo0 + row, k1 = w.lo1 + (e - row * w.bw);
        bool hit = false;
        if (e < nc) {
          float dc[K], base[K], step[K];
          dc[0] = (__ldg(g.ax[0].coords + k0) - w.a.x) - w.a.y;
          dc[1] = (__ldg(g.ax[1].coords + k1) - w.a.z) - w.a.w;
          hit = psf_cell_kind<K>(q, dc, s, base, step) != 0;
        }
        push(hit, make_int2(k0 << 5 | sl, k1));
      }
    }
    if (queued) add_cells(queued);
    if (on) {
      const float *v = sum[lane];
      f += v[0];
      float Sa[NPSI], Ta[NPSI][NPSI], Ub[NPSI][NPSI];
#pragma unroll
      for (int k = 0; k < NPSI; ++k) Sa[k] = v[1 + k];
      if constexpr (ORDER > 1) {
        int o = 1 + NPSI;
#pragma unroll
        for (int k = 0; k < NPSI; ++k)
#pragma unroll
          for (int l = k; l < NPSI; ++l, ++o) {
            Ta[k][l] = Ta[l][k] = v[o];
            Ub[k][l] = Ub[l][k] = v[NT + o];
          }
      }
      accumulate_pair<K, ORDER>(p, fr, I, Sa, Ta, Ub, gacc, hacc);
    }
    __syncwarp();
  }

  if (lane < PW) {
    vals[pr][0] = f;
#pragma unroll
    for (int i = 0; i < P; ++i) vals[pr][1 + i] = gacc[i].get();
    if constexpr (ORDER > 1) {
#pragma unroll
      for (int i = 0; i < NH; ++i) vals[pr][1 + P + i] = hacc[i];
    }
  }
  __syncthreads();
  psf_close<QN>(vals, at.n, cfg, chunk, wa, part);
}

// Sum chunk partials (FP64), expand the packed Hessian and apply the isotropic
// chain rule r_aniso = (s, .., s, 0, ..).  A block covers kFinAtoms atoms, 64
// threads each; few atoms per block spread the FP64 adds over many SMs' FP64
// pipes (16 cycles per warp instruction each).  Where an atom has fewer than
// 64 values, S threads share one, each summing a contiguous range of chunks in
// chunk order (a dependent FP64 add takes 64 cycles), and the ranges are added
// in order; a thread loads kFinBatch partials before it adds any.  Ranges of less
// than kFinBatch / 2 chunks gain nothing (fin_shares), and an atom whose values fill half
// of the threads has half of them (fin_threads: 6298 atoms x 1 chunk 5.4 -> 3.0 us, 3.3 before ranges).  8192 atoms x
// 625 chunks: 357 -> 244 us (conversions and adds on the FP64 pipe), 1000 x 126:
// 21.7 -> 13.7 us, 64 x 60: 10.2 -> 5.9 us (one thread per value with four loads
// in flight before).
constexpr int kFinAtoms = 4;
constexpr int kFinPer = 64;            // threads per atom
constexpr int kFinThreads = kFinPer * kFinAtoms;
constexpr int kFinBatch = 8;
// threads that share a value of an atom
__host__ __device__ __forceinline__ int fin_shares(const DerivCfg &cfg) {
  int S = 1;
  while (2 * S * cfg.qn <= kFinPer && S < 8 && cfg.nchunks >= S * kFinBatch) S *= 2;
  return S;
}
// threads of a block
__host__ __device__ __forceinline__ int fin_threads(const DerivCfg &cfg) {
  return fin_shares(cfg) * cfg.qn <= kFinPer / 2 ? kFinThreads / 2 : kFinThreads;
}
// Gradients as float32 arrays per parameter kind (gr_atom_grads); q = 0 is the
// value, 1 the intensity.
template <int D>
__device__ __forceinline__ void grad_out(const DerivOut &out, int j, int q, int P, double v) {
  if (q == 1) out.gI[j] = (float)v;
  else if (q > 1 && q <= 1 + D) out.gx[(size_t)j * D + q - 2] = (float)v;
  else if (q > 1 + D) out.gr[(size_t)j * (P - 1 - D) + q - 2 - D] = (float)v;
}

// The body of one block of the finalize launch (the launch's block; a
// multi-problem launch maps its blocks to (problem, block)).
template <int K>
__device__ __forceinline__ void finalize_body(const float *part, const DerivCfg &cfg, int n,
                                              int deriv_order, int r_iso, const DerivOut &out,
                                              const double *f_extra, const int *order, int block) {
  constexpr int D = K + 1;
  constexpr int P = n_par<K>();
  constexpr int QN = 1 + P + P * (P + 1) / 2;
  __shared__ double vs[QN][kFinAtoms];
  __shared__ double ps[kFinPer][kFinAtoms];   // ranges of shared values
  const int tx = threadIdx.x % kFinAtoms, ty = threadIdx.x / kFinAtoms;
  const int slot = block * kFinAtoms + tx;
  const int S = fin_shares(cfg), per = (int)blockDim.x / kFinAtoms;
  for (int e = ty; slot < n && e < cfg.qn * S; e += per) {
    // value q over the s-th of S ranges of chunks
    const int sh = 31 - __clz(S), q = e >> sh, s = e & (S - 1);
    int c = (int)((unsigned)cfg.nchunks * s >> sh);   // (8 times the chunks: 32 bits)
    const int hi = (int)((unsigned)cfg.nchunks * (s + 1) >> sh);
    const size_t step = (size_t)cfg.qn * n;
    const float *src = part + (size_t)q * n + slot + c * step;
    double t = 0.0;
    auto add = [&](auto batch) {
      constexpr int B = decltype(batch)::value;
      float v[B];
#pragma unroll
      for (int i = 0; i < B; ++i) v[i] = __ldcs(src + i * step);
#pragma unroll
      for (int i = 0; i < B; ++i) t += (double)v[i];
      c += B;
      src += B * step;
    };
    while (c + kFinBatch <= hi) add(std::integral_constant<int, kFinBatch>());
    if constexpr (K == 2) {
      // (66 values an atom keep the loads coming: 2936 x 5 chunks 7.5 us, 9.2 as below)
      for (; c < hi; ++c, src += step) t += (double)__ldcs(src);
    } else {
      if (c + 4 <= hi) add(std::integral_constant<int, 4>());
      if (c < hi) {
        float v[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) v[i] = c + i < hi ? __ldcs(src + i * step) : 0.f;
#pragma unroll
        for (int i = 0; i < 3; ++i)
          if (c + i < hi) t += (double)v[i];
      }
    }
    if (S == 1) vs[q][tx] = t;
    else ps[e][tx] = t;
  }
  if (S > 1) {
    __syncthreads();
    if (slot < n && ty < cfg.qn) {
      double t = ps[ty * S][tx];
      for (int k = 1; k < S; ++k) t += ps[ty * S + k][tx];
      vs[ty][tx] = t;
    }
  }
  __syncthreads();
  // outputs of the block's atoms, written by all threads from the sums
  // (consecutive threads write consecutive entries of an atom's block)
  const int nb = min(kFinAtoms, n - (int)block * kFinAtoms);
  auto atom_of = [&](int t) {
    const int sl = block * kFinAtoms + t;
    return order ? order[sl] : sl;
  };
  // entry (a, b) of the full Hessian from the packed upper triangle
  auto hv = [&](int a, int b, int t) -> double {
    const int lo = a < b ? a : b, hi = a < b ? b : a;
    return vs[1 + P + lo * P - lo * (lo - 1) / 2 + (hi - lo)][t];
  };
  const double fx = f_extra ? f_extra[0] : 0.0;
  if (!r_iso) {
    for (int e = threadIdx.x; e < nb * (1 + P); e += blockDim.x) {
      const int t = e / (1 + P), q = e - t * (1 + P);
      const int j = atom_of(t);
      if (out.gI) grad_out<D>(out, j, q, P, vs[q][t]);
      else if (q == 0) out.f[j] = vs[0][t] + fx;
      else out.g[(size_t)j * P + q - 1] = vs[q][t];
    }
    if (deriv_order > 1)
      for (int e = threadIdx.x; e < nb * P * P; e += blockDim.x) {
        const int t = e / (P * P), ab = e - t * (P * P), a = ab / P, b = ab - a * P;
        out.H[(size_t)atom_of(t) * P * P + ab] = hv(a, b, t);
      }
    return;
  }
  // isotropic: parameters (I, x, s); s maps to the D diagonal r entries
  // (r_aniso = (s, .., s, 0, ..)), so its derivatives sum those entries'
  constexpr int PI = 2 + D;
  auto src = [](int a, int q) { return a < 1 + D ? a : 1 + D + q; };
  for (int e = threadIdx.x; e < nb * (1 + PI); e += blockDim.x) {
    const int t = e / (1 + PI), q = e - t * (1 + PI);
    const int j = atom_of(t);
    if (q == 0) {
      if (!out.gI) out.f[j] = vs[0][t] + fx;
    } else {
      const int a = q - 1;
      double gsum = 0.0;
      if (a <= D) {
        gsum = vs[1 + a][t];
      } else {
#pragma unroll
        for (int qq = 0; qq < D; ++qq) gsum += vs[1 + 1 + D + qq][t];
      }
      if (out.gI) grad_out<D>(out, j, q, PI, gsum);
      else out.g[(size_t)j * PI + a] = gsum;
    }
  }
  if (deriv_order > 1)
    for (int e = threadIdx.x; e < nb * PI * PI; e += blockDim.x) {
      const int t = e / (PI * PI), ab = e - t * (PI * PI), a = ab / PI, b = ab - a * PI;
      const int na = a < 1 + D ? 1 : D, nbb = b < 1 + D ? 1 : D;
      double hs = 0.0;
      for (int qa = 0; qa < na; ++qa)
        for (int qb = 0; qb < nbb; ++qb) hs += hv(src(a, qa), src(b, qb), t);
      out.H[(size_t)atom_of(t) * PI * PI + ab] = hs;
    }
}

template <int K>
__global__ void __launch_bounds__(kFinThreads)
    gr_deriv_finalize_kernel(const float *part, DerivCfg cfg, int n, int deriv_order,
                             int r_iso, DerivOut out, const double *f_extra,
                             const int *order) {
  finalize_body<K>(part, cfg, n, deriv_order, r_iso, out, f_extra, order, blockIdx.x);
}

// 1/2 sum C^2 helper: block partial sums (FP32 compensated per thread, FP64
// across the block), then a fixed-order FP64 finalize.
__global__ void gr_sumsq_kernel(const float *C, size_t n, double *part) {
  __shared__ double sh[256];
  CAcc acc;
  acc.zero();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const float c = C[i];
    acc.add(c * c);
  }
  sh[threadIdx.x] = (double)acc.s + (double)acc.c;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// (one thread's chain of n dependent FP64 adds took 16 us)
__global__ void __launch_bounds__(256)
    gr_sumsq_finalize_kernel(const double *part, int n, double scale, double *out) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = scale * sh[0];
}

constexpr int kSumSqBlocks = 304;

int launch_sum_squares(const float *C, size_t n, double *out, void *ws,
                       size_t ws_bytes, cudaStream_t stream) {
  if (ws_bytes < align_up(kSumSqBlocks * sizeof(double))) return kErrWorkspace;
  double *part = static_cast<double *>(ws);
  gr_sumsq_kernel<<<kSumSqBlocks, 256, 0, stream>>>(C, n, part);
  gr_sumsq_finalize_kernel<<<1, 256, 0, stream>>>(part, kSumSqBlocks, 0.5, out);
  note_launches(2);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

Tuning g_tuning;

int tuning_set(Tuning &t, int key, int value) {
  if (key == 0 && value >= 32 && value <= (1 << 26)) {
    t.deriv_target_warps = value;
    return kOk;
  }
  if (key == 1 && value >= 1 && value <= 65536) {
    t.deriv_min_angles = value;
    return kOk;
  }
  if (key == 2 && (value == 0 || (value >= 1 && value <= 32 && (value & (value - 1)) == 0))) {
    t.deriv_atoms_per_warp = value;
    return kOk;
  }
  if (key == 3 && value >= 1 && value <= 3) {
    t.proj_form = value;
    return kOk;
  }
  if (key == 4 && value >= 0) {
    t.proj_split_cells = value;
    return kOk;
  }
  if (key == 6 && value >= 0) {
    t.deriv_split_lanes = value;
    return kOk;
  }
  if (key == 7 && value >= 0) {
    t.deriv_one_mb = value;
    return kOk;
  }
  if (key == 8 && (value == 0 || value == 1)) {
    t.deriv_wide_rows = value;
    return kOk;
  }
  if (key == 9 && (value == 1 || value == 4)) {
    t.deriv_block_warps = value;
    return kOk;
  }
  return kErrArg;
}

int tuning_get(const Tuning &t, int key) {
  return key == 0 ? t.deriv_target_warps : key == 1 ? t.deriv_min_angles
         : key == 2 ? t.deriv_atoms_per_warp : key == 3 ? t.proj_form
         : key == 4 ? t.proj_split_cells
         : key == 6 ? t.deriv_split_lanes : key == 7 ? t.deriv_one_mb
         : key == 8 ? t.deriv_wide_rows : key == 9 ? t.deriv_block_warps : -1;
}

// Workspace of a launch under the split c.
static size_t derivs_bytes(const DerivCfg &c, int n_atoms) {
  size_t b = align_up((size_t)c.nchunks * c.qn * (size_t)n_atoms * sizeof(float));
  b += align_up(kSumSqBlocks * sizeof(double)) + align_up(sizeof(double));
  return b;
}

// The query names no operator: the larger of the point-sampled and the
// pixel-integrated kernels' splits (either can have more chunks: the second never
// shares a pair among lanes, but gives a warp four atoms up to longer series).
size_t derivs_workspace_bytes(int K, int n_atoms, int n_angles, int order, const Tuning &t) {
  const size_t point = derivs_bytes(deriv_cfg(K, n_atoms, n_angles, order, t, true), n_atoms);
  const size_t pixel = derivs_bytes(deriv_cfg(K, n_atoms, n_angles, order, t, false), n_atoms);
  return point > pixel ? point : pixel;
}

struct DerivArgs {
  const Atoms &at;
  const Geom &g;
  const DerivIn &in;
  const DerivCfg &cfg;
  float *part;
  int warps;
  bool one;
  cudaStream_t stream;
};

template <int K, bool QUAD, bool L2ATOM>
static void start_grad(const DerivArgs &d) {
  if (d.one)
    gr_grad_kernel<K, true, QUAD, L2ATOM><<<d.warps, 32, 0, d.stream>>>(d.at, d.g, d.in, d.cfg, d.part);
  else
    gr_grad_kernel<K, false, QUAD, L2ATOM><<<d.warps, 32, 0, d.stream>>>(d.at, d.g, d.in, d.cfg, d.part);
}

static void start_grad3(const DerivArgs &d) {
  const bool l2atom = d.in.mode == kModeL2Atom;
  const size_t at16 = reinterpret_cast<size_t>(d.in.alpha) | reinterpret_cast<size_t>(d.g.ax[1].coords);
  if (d.g.ax[1].n % 4 == 0 && at16 % 16 == 0)
    l2atom ? start_grad<2, true, true>(d) : start_grad<2, true, false>(d);
  else
    l2atom ? start_grad<2, false, true>(d) : start_grad<2, false, false>(d);
}

template <int K, int GL, int FK>
static void start_one(const DerivArgs &d) {
  gr_hess_kernel<K, true, GL, walk_cells_of<K>(), FK><<<d.warps, 32, 0, d.stream>>>(
      d.at, d.g, d.in, d.cfg, d.part);
}

template <int K>
static void start_hess(const DerivArgs &d) {
  const bool beta = d.in.beta != nullptr, l2atom = d.in.mode == kModeL2Atom;
  if (!d.one || (beta && l2atom)) {
    gr_hess_kernel<K, false, walk_lanes_of<K>(), walk_cells_of<K>(), kFieldAny>
        <<<d.warps, 32, 0, d.stream>>>(d.at, d.g, d.in, d.cfg, d.part);
  } else if (d.cfg.rs == 8) {
    // a warp with four pairs has eight lanes walk each
    if (l2atom) start_one<K, 8, kFieldL2Atom>(d);
    else if (beta) start_one<K, 8, kFieldBeta>(d);
    else start_one<K, 8, kFieldPlain>(d);
  } else if (K == 1 && d.cfg.rs == 4) {
    // (64 atoms x 180 x 512, supports of 230 cells, with the closing sums: 23.3 us by
    // two lanes a pair, half of the warp idle, 17.3 by four)
    if (l2atom) start_one<K, 4, kFieldL2Atom>(d);
    else if (beta) start_one<K, 4, kFieldBeta>(d);
    else start_one<K, 4, kFieldPlain>(d);
  } else {
    constexpr int GL = walk_lanes_of<K>();
    if (l2atom) start_one<K, GL, kFieldL2Atom>(d);
    else if (beta) start_one<K, GL, kFieldBeta>(d);
    else start_one<K, GL, kFieldPlain>(d);
  }
}

// Pixel-integrated derivatives.  2D, lanes a pair: as many as keep the blocks'
// warps to 32 an SM (gradients; Hessians 16), since wide supports want lanes and
// narrow ones are mostly set-up and assembly, which L lanes do once for 32 / L
// pairs (us with 4, 2 and 1; gradients, 200 atoms x 100 angles x 467 cells, r = 4:
// 25, 31, 46; 500 x 130 x 300, r = 4: 38, 41, 43, x 64, r = 30: 15, 13.5, 11.4; 2154
// x 736 x 75, r = 30: 152, 104, 72; Hessians there: 282, 183, 119).  3D, pairs a
// warp: all 32 from some four full waves of such blocks on, half from 20 blocks an SM
// on, for the same reason; wide supports lose by their last wave, a tenth or, in few
// blocks, a fifth, and narrow ones gain as much there, so the line of the Hessians keeps
// the long calls from losing (us, 8, 16 and 32 a warp; gradients, 128 x 401 x 64^2, 11
// blocks an SM, r = 8 and 20: 122, 145, 161 and 52, 50, 54; 300 x 401, 25 blocks: 246,
// 265, 295 and 104, 89, 90; 600 x 401, 50 blocks, r = 8 and 30: 476, 493, 520 and 160,
// 101, 89; 1412 x 907 x 78^2, 265 blocks, r = 12 and 35: 1894, 1869, 1835 and 804, 510,
// 414; Hessians 234, 247, 306 and 110, 92, 103; 497, 501, 535 and 229, 185, 172; 961, 949,
// 978 and 366, 242, 197; 3866, 3652, 3654 and 1845, 1231, 975; with 8 and 16 alone, 651 x
// 86 x 57^2, whole detectors, 13 blocks: 1939, 2335, of six-parameter atoms 2473, 2856).
constexpr int kPsfSms = 152;
template <int ORDER>
static void start_psf(const DerivArgs &d, float s) {
  auto go = [&](auto kernel, int threads) {
    kernel<<<d.warps, threads, 0, d.stream>>>(d.at, d.g, d.in, d.cfg, d.part, s);
  };
  if (d.g.K == 1) {
    // lanes that the pairs of short series leave idle count as free
    const long long room = kPsfSms * 32 * (ORDER == 1 ? 32 : 16);
    const long long pairs = (long long)d.at.n * d.g.n_angles, slots = 32ll * d.warps;
    if (4 * pairs <= room || 4 * pairs <= slots) go(gr_psf_deriv1d_kernel<ORDER, 4>, 128);
    else if (2 * pairs <= room || 2 * pairs <= slots) go(gr_psf_deriv1d_kernel<ORDER, 2>, 64);
    else go(gr_psf_deriv1d_kernel<ORDER, 1>, 32);
  } else if (d.warps < kPsfSms * 20) {
    go(gr_psf_deriv_kernel<ORDER, 8>, 128);
  } else if (d.warps < kPsfSms * (ORDER == 1 ? 60 : 40)) {
    go(gr_psf_deriv_kernel<ORDER, 16>, 64);
  } else {
    go(gr_psf_deriv_kernel<ORDER, 32>, 32);
  }
}
template <int ORDER>
static int preload_psf() {
  return preload_fn(gr_psf_deriv1d_kernel<ORDER, 1>) + preload_fn(gr_psf_deriv1d_kernel<ORDER, 2>) +
         preload_fn(gr_psf_deriv1d_kernel<ORDER, 4>) + preload_fn(gr_psf_deriv_kernel<ORDER, 8>) +
         preload_fn(gr_psf_deriv_kernel<ORDER, 16>) + preload_fn(gr_psf_deriv_kernel<ORDER, 32>);
}

int launch_derivs(const Atoms &at, const Geom &g, const DerivIn &in,
                  const DerivOut &out, void *ws, size_t ws_bytes,
                  cudaStream_t stream, const Tuning &t) {
  const int K = g.K;
  if (at.n <= 0) return kOk;
  if (in.order < 1 || in.order > 2) return kErrArg;
  // (the pixel-integrated kernels do not share a pair's cells out by rs)
  const DerivCfg c = deriv_cfg(K, at.n, g.n_angles, in.order, t, !in.psf);
  if (ws == nullptr || ws_bytes < derivs_bytes(c, at.n)) return kErrWorkspace;
  char *wp = static_cast<char *>(ws);
  float *part = reinterpret_cast<float *>(wp);
  wp += align_up((size_t)c.nchunks * c.qn * (size_t)at.n * sizeof(float));
  double *sumsq_part = reinterpret_cast<double *>(wp);
  wp += align_up(kSumSqBlocks * sizeof(double));
  double *f_extra = reinterpret_cast<double *>(wp);
  const double *fe = nullptr;
  if (in.mode == kModeL2Atom) {
    const size_t cells = (size_t)g.n_angles * g.ax[0].n * (K == 2 ? g.ax[1].n : 1);
    int rc = launch_sum_squares(in.alpha, cells, f_extra, sumsq_part,
                                align_up(kSumSqBlocks * sizeof(double)), stream);
    if (rc != kOk) return rc;
    fe = f_extra;
  }
  const int warps = ((at.n + c.ag - 1) / c.ag) * c.nchunks;
  const float s = 0.5f / g.ax[0].inv_step;  // cell half-width (pixel-integrated operator)
  timer_mark(2, 0, stream);
  if (in.psf) {
    const DerivArgs d{at, g, in, c, part, warps, false, stream};
    if (in.order == 1) start_psf<1>(d, s);
    else start_psf<2>(d, s);
  } else {
    // at most one angle per lane: a lane's angles a_lo + sub + k sg lie
    // below a_lo + ch
    const bool one = c.ch <= c.sg / c.rs;
    const DerivArgs d{at, g, in, c, part, warps, one, stream};
    if (in.order == 2) K == 1 ? start_hess<1>(d) : start_hess<2>(d);
    else if (K == 1) start_grad<1, false, false>(d);
    else start_grad3(d);
  }
  timer_mark(2, 1, stream);
  const int fblocks = (at.n + kFinAtoms - 1) / kFinAtoms;
  if (K == 1)
    gr_deriv_finalize_kernel<1><<<fblocks, fin_threads(c), 0, stream>>>(
        part, c, at.n, in.order, at.r_iso, out, fe, at.order);
  else
    gr_deriv_finalize_kernel<2><<<fblocks, fin_threads(c), 0, stream>>>(
        part, c, at.n, in.order, at.r_iso, out, fe, at.order);
  note_launches(2);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

// ---- multi-problem launches (2D Hessians, one angle per lane) ------------
// The derivatives of a problem run only on its first iteration or after an
// accepted trial (a rejected trial leaves its atoms and fields unchanged),
// and not once its fit has stopped.
__device__ __forceinline__ bool batch_derivs_wanted(const BatchProb &B, int active) {
  if (!active) return false;
  const int c = *B.counter;
  return !(c > 0 && c <= B.hist_len && !B.hist_acc[c - 1]);
}

__global__ void __launch_bounds__(128, hess_min_warps(1, true) / 4)
    gr_batch_deriv_kernel(const BatchProb *__restrict__ probs, const int *__restrict__ off,
                          int n, const int *__restrict__ active) {
  __shared__ WalkSmem<1> sm[4];
  const int p = batch_find(off, n, blockIdx.x);
  const BatchProb &B = probs[p];
  if (!batch_derivs_wanted(B, active[p])) return;
  const int warp0 = ((int)blockIdx.x - off[p]) * 4;
  WalkSmem<1> &w = sm[threadIdx.x >> 5];
  if (B.cfg.rs == 8)
    hess_body<1, true, 8, walk_cells_of<1>(), kFieldPlain>(
        B.cur, B.g, B.din, B.cfg, B.part, warp0, w);
  else if (B.cfg.rs == 4)
    hess_body<1, true, 4, walk_cells_of<1>(), kFieldPlain>(
        B.cur, B.g, B.din, B.cfg, B.part, warp0, w);
  else
    hess_body<1, true, walk_lanes_of<1>(), walk_cells_of<1>(), kFieldPlain>(
        B.cur, B.g, B.din, B.cfg, B.part, warp0, w);
}

__global__ void __launch_bounds__(kFinThreads)
    gr_batch_finalize_kernel(const BatchProb *__restrict__ probs, const int *__restrict__ off,
                             int n, const int *__restrict__ active) {
  const int p = batch_find(off, n, blockIdx.x);
  const BatchProb &B = probs[p];
  if (!batch_derivs_wanted(B, active[p])) return;
  finalize_body<1>(B.part, B.cfg, B.cur.n, 2, B.cur.r_iso, B.dout, nullptr, nullptr,
                   blockIdx.x - off[p]);
}

int finalize_blocks(int n_atoms) { return (n_atoms + kFinAtoms - 1) / kFinAtoms; }

int launch_batch_derivs(const BatchLaunch &b, cudaStream_t stream) {
  if (b.grid_deriv <= 0) return kOk;
  gr_batch_deriv_kernel<<<b.grid_deriv, 128, 0, stream>>>(b.probs, b.off_deriv, b.n, b.active);
  gr_batch_finalize_kernel<<<b.grid_fin, kFinThreads, 0, stream>>>(b.probs, b.off_fin, b.n,
                                                                   b.active);
  note_launches(2);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

template <int K, int GL>
static int preload_one() {
  return preload_fn(gr_hess_kernel<K, true, GL, walk_cells_of<K>(), kFieldPlain>) +
         preload_fn(gr_hess_kernel<K, true, GL, walk_cells_of<K>(), kFieldBeta>) +
         preload_fn(gr_hess_kernel<K, true, GL, walk_cells_of<K>(), kFieldL2Atom>);
}
template <int K>
static int preload_walk() {
  return preload_one<K, walk_lanes_of<K>()>() + preload_one<K, 8>() +
         (K == 1 ? preload_one<K, 4>() : 0) +
         preload_fn(gr_hess_kernel<K, false, walk_lanes_of<K>(), walk_cells_of<K>(), kFieldAny>) +
         preload_fn(gr_grad_kernel<K, true, false, false>) +
         preload_fn(gr_grad_kernel<K, false, false, false>);
}

int preload_derivs() {
  return preload_walk<1>() + preload_walk<2>() +
         preload_fn(gr_grad_kernel<2, true, true, false>) + preload_fn(gr_grad_kernel<2, false, true, false>) +
         preload_fn(gr_grad_kernel<2, true, true, true>) + preload_fn(gr_grad_kernel<2, false, true, true>) +
         preload_fn(gr_grad_kernel<2, true, false, true>) + preload_fn(gr_grad_kernel<2, false, false, true>) +
         
         preload_psf<1>() + preload_psf<2>() +
         preload_fn(gr_deriv_finalize_kernel<1>) + preload_fn(gr_deriv_finalize_kernel<2>) +
         preload_fn(gr_sumsq_kernel) + preload_fn(gr_sumsq_finalize_kernel) +
         preload_fn(gr_batch_deriv_kernel) + preload_fn(gr_batch_finalize_kernel);
}

}  // namespace gr
