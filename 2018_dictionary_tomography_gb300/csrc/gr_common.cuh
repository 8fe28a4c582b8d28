// Shared device helpers for the Gaussian-atom Radon kernels (sm_103a).
//
// Model (reference GaussDictCode/bin/NewtonBases2D.py:39-72 and
// GaussDictCode/bin/NewtonBases.py:262-310): an atom (I, x, r) projects to
//     R(y) = I / |r T| * exp(-30 m),   m = |(1 - t t^T) r (y - x)|^2,
//     t = r T / |r T|,   R = 0 where m > 1,
// for detector points y = sum_i q_i w_i.  With the frame B = [w_0 .. w_{K-1}, T]
// and K_c = r B_c, Q = K^T K, the projection of the atom is the Gaussian
//     m(q) = (q - q*)^T G (q - q*),  G = Q_ww - Q_wT Q_wT^T / Q_TT,
//     q* = (B^{-1} x)[0:K],          1/|r T| = Q_TT^{-1/2},
// i.e. a K-dimensional Gaussian whose precision is the Schur complement of
// the atom precision in the frame.  Per (atom, angle) "pair" the kernels
// compute G, q*, the amplitude and the support box once, and per detector
// cell only the quadratic form and one exp2.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gr {

constexpr int kMaxK = 2;                          // detector dimensions
constexpr float kNegThirtyLog2e = -43.28085122666891f;  // -30 / ln 2
constexpr int kFrameStride2D = 8;   // T(2) w0(2) wt0(2) wl0(2)
constexpr int kFrameStride3D = 24;  // T(3) w0(3) w1(3) wt0(3) wt1(3) wl0(3) wl1(3) pad(3)

// Error codes shared with the C ABI.
enum Status : int {
  kOk = 0,
  kErrArg = -1,
  kErrWorkspace = -2,
  kErrLaunch = -3,
  kErrShape = -4,
};

__device__ __forceinline__ float ex2_approx(float v) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
  return y;
}

__device__ __forceinline__ float sqrt_approx(float v) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
  return y;
}

__device__ __forceinline__ float lg2_approx(float v) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
  return y;
}

// Two FP32 values in one register pair (sm_100 and later): one instruction
// adds, multiplies or fuses both, each half rounded as the scalar operation.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_get(const F2 &a, float &x, float &y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 f2_add(const F2 &a, const F2 &b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(const F2 &a, const F2 &b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(const F2 &a, const F2 &b, const F2 &c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// a - b (the product with -1 is exact, so this rounds as a subtraction)
__device__ __forceinline__ F2 f2_sub(const F2 &a, const F2 &b) {
  return f2_fma(b, f2(-1.f, -1.f), a);
}

// Error-free transforms (Knuth TwoSum, FMA TwoProduct) used for the
// compensated projection centre and compensated accumulators.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

__device__ __forceinline__ void two_prod(float a, float b, float &p, float &e) {
  p = __fmul_rn(a, b);
  e = __fmaf_rn(a, b, -p);
}

// Compensated dot product of length n <= 3 (Ogita-Rump-Oishi Dot2): the
// result hi + lo carries roughly twice the working precision.
template <int N>
__device__ __forceinline__ void dot2(const float *a, const float *b, float &hi,
                                     float &lo) {
  float s, c;
  two_prod(a[0], b[0], s, c);
#pragma unroll
  for (int i = 1; i < N; ++i) {
    float p, pe, t, te;
    two_prod(a[i], b[i], p, pe);
    two_sum(s, p, t, te);
    s = t;
    c += pe + te;
  }
  two_sum(s, c, hi, lo);
}

// Kahan-style compensated accumulator (Neumaier variant, exact when |v|>|s|).
struct CAcc {
  float s, c;
  __device__ __forceinline__ void zero() { s = 0.f; c = 0.f; }
  __device__ __forceinline__ void add(float v) {
    float t = s + v;
    c += (fabsf(s) >= fabsf(v)) ? ((s - t) + v) : ((v - t) + s);
    s = t;
  }
  __device__ __forceinline__ float get() const { return s + c; }
};

// Uniform detector grid: the coordinate of cell k is coords[k]; first and
// inverse step locate the support box, the stored coordinates are what the
// cell values use.
struct DetAxis {
  const float *coords;
  int n;
  float first;
  float inv_step;
};

// Geometry of one problem in device memory.
struct Geom {
  int K;                 // 1: 2D sinogram (A, D0); 2: 3D / 2.5D (A, D0, D1)
  int n_angles;
  const float *frames;   // n_angles x stride, see kFrameStride*
  DetAxis ax[kMaxK];
};

// Atoms in device memory: r is packed upper-triangular (2D: r00 r11 r01;
// 3D: r00 r11 r22 r01 r12 r02) or, when r_iso, one radius per atom.
struct Atoms {
  int n;
  const float *I;
  const float *x;
  const float *r;
  int r_iso;
  const int *order;  // optional processing order of the derivative kernels
};

template <int K>
struct Frame {
  float T[K + 1];
  float w[K][K + 1];
  float wt[K][K + 1];  // rows 0..K-1 of B^{-1} (rounded to FP32)
  const float *wl;     // their rounding residues (B^{-1} rows = wt + wl), read
                       // from the record only when a pair is set up
};

template <int K>
__device__ __forceinline__ void load_frame(const float *frames, int a,
                                           Frame<K> &f) {
  constexpr int D = K + 1;
  const float *p = frames + (size_t)a * (K == 1 ? kFrameStride2D : kFrameStride3D);
#pragma unroll
  for (int i = 0; i < D; ++i) f.T[i] = p[i];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int i = 0; i < D; ++i) f.w[k][i] = p[D * (1 + k) + i];
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll
    for (int i = 0; i < D; ++i) f.wt[k][i] = p[D * (1 + K + k) + i];
  f.wl = p + D * (1 + 2 * K);
}

// A warp's 3D frames in shared memory: lanes of a warp take different angles, and
// a lane's own 24 loads, 96 bytes from its neighbour's, touch 24 lines each; the
// records are one run of memory, so the warp copies them 16 bytes a lane.
struct FrameSmem {
  static constexpr int kStride = kFrameStride3D + 4;  // 8 lanes' 16-byte reads: all banks
  float4 v[32][kStride / 4];
};

// the n <= 32 records from `frames` on (the caller synchronises the warp)
__device__ __forceinline__ void stage_frames(FrameSmem &sm, const float *frames, int n) {
  constexpr int Q = kFrameStride3D / 4;
  const int lane = threadIdx.x & 31;
  if ((reinterpret_cast<size_t>(frames) & 15) == 0) {
    for (int i = lane; i < n * Q; i += 32)
      sm.v[i / Q][i % Q] = __ldg(reinterpret_cast<const float4 *>(frames) + i);
  } else {
    for (int i = lane; i < n * kFrameStride3D; i += 32)
      reinterpret_cast<float *>(sm.v[i / kFrameStride3D])[i % kFrameStride3D] = __ldg(frames + i);
  }
}

__device__ __forceinline__ void load_frame(const FrameSmem &sm, int i, Frame<2> &f) {
  const float4 a = sm.v[i][0], b = sm.v[i][1], c = sm.v[i][2], d = sm.v[i][3];
  f.T[0] = a.x, f.T[1] = a.y, f.T[2] = a.z;
  f.w[0][0] = a.w, f.w[0][1] = b.x, f.w[0][2] = b.y;
  f.w[1][0] = b.z, f.w[1][1] = b.w, f.w[1][2] = c.x;
  f.wt[0][0] = c.y, f.wt[0][1] = c.z, f.wt[0][2] = c.w;
  f.wt[1][0] = d.x, f.wt[1][1] = d.y, f.wt[1][2] = d.z;
  f.wl = reinterpret_cast<const float *>(sm.v[i]) + 15;
}

// Upper-triangular r as a dense (K+1)x(K+1) matrix.
template <int K>
__device__ __forceinline__ void load_r(const Atoms &at, int j,
                                       float (&M)[K + 1][K + 1]) {
  constexpr int D = K + 1;
#pragma unroll
  for (int a = 0; a < D; ++a)
#pragma unroll
    for (int b = 0; b < D; ++b) M[a][b] = 0.f;
  if (at.r_iso) {
    float s = at.r[j];
#pragma unroll
    for (int a = 0; a < D; ++a) M[a][a] = s;
  } else if constexpr (K == 1) {
    const float *r = at.r + 3 * (size_t)j;
    M[0][0] = r[0];
    M[1][1] = r[1];
    M[0][1] = r[2];
  } else {
    const float *r = at.r + 6 * (size_t)j;
    M[0][0] = r[0];
    M[1][1] = r[1];
    M[2][2] = r[2];
    M[0][1] = r[3];
    M[1][2] = r[4];
    M[0][2] = r[5];
  }
}

// Packed r index p -> (row, col).
template <int K>
__host__ __device__ constexpr int rrow(int p) {
  return K == 1 ? (p == 0 ? 0 : p == 1 ? 1 : 0)
                : (p == 0 ? 0 : p == 1 ? 1 : p == 2 ? 2 : p == 3 ? 0 : p == 4 ? 1 : 0);
}
template <int K>
__host__ __device__ constexpr int rcol(int p) {
  return K == 1 ? (p == 0 ? 0 : p == 1 ? 1 : 1)
                : (p == 0 ? 0 : p == 1 ? 1 : p == 2 ? 2 : p == 3 ? 1 : p == 4 ? 2 : 2);
}
template <int K>
__host__ __device__ constexpr int n_rparam() { return K == 1 ? 3 : 6; }

// Per (atom, angle) projection data.
template <int K>
struct Pair {
  float qh[K], ql[K];  // projection centre q* = hi + lo
  float G[3];          // G00, G01, G11 (K == 1: G00)
  float n;             // 1 / |r T|
  float l2amp;         // log2(|I| n)
  float sgn;           // sign of I (+1 or -1)
  int lo[K], hi[K];    // inclusive support box in cell indices (empty: lo > hi)
  // quantities kept for the derivative assembly
  float Kc[K + 1][K + 1];  // Kc[c][a] = (r B_c)_a, c = 0..K-1 detector axes, K = T
  float Q[K + 1][K + 1];   // Q[c][d] = Kc[c] . Kc[d]
};

// STAGED: the frame was read from shared memory (load_frame of a FrameSmem).
template <int K, bool STAGED = false>
__device__ __forceinline__ bool pair_setup(const Atoms &at, int j,
                                           const Frame<K> &f, const Geom &g,
                                           Pair<K> &p) {
  constexpr int D = K + 1;
  float M[D][D];
  load_r<K>(at, j, M);
  // K_c = r B_c for the detector axes and the ray direction
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const float *B = (c < K) ? f.w[c] : f.T;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      float s = 0.f;
#pragma unroll
      for (int b = a; b < D; ++b) s = fmaf(M[a][b], B[b], s);
      p.Kc[c][a] = s;
    }
  }
#pragma unroll
  for (int c = 0; c < D; ++c)
#pragma unroll
    for (int d = c; d < D; ++d) {
      float s = 0.f;
#pragma unroll
      for (int a = 0; a < D; ++a) s = fmaf(p.Kc[c][a], p.Kc[d][a], s);
      p.Q[c][d] = s;
      p.Q[d][c] = s;
    }
  const float qtt = p.Q[K][K];
  const float iqtt = 1.f / qtt;
  p.n = rsqrtf(qtt);
  // G = U^T U with U_i = K_i - t (t . K_i), t = K_T / |K_T| (the projected
  // detector axes); this Gram form stays positive semi-definite in FP32.
  float U[K][D];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const float c = p.Q[i][K] * iqtt;
#pragma unroll
    for (int a = 0; a < D; ++a) U[i][a] = fmaf(-c, p.Kc[K][a], p.Kc[i][a]);
  }
  if constexpr (K == 1) {
    p.G[0] = U[0][0] * U[0][0] + U[0][1] * U[0][1];
    p.G[1] = 0.f;
    p.G[2] = 0.f;
  } else {
    float g00 = 0.f, g01 = 0.f, g11 = 0.f;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      g00 = fmaf(U[0][a], U[0][a], g00);
      g01 = fmaf(U[0][a], U[1][a], g01);
      g11 = fmaf(U[1][a], U[1][a], g11);
    }
    p.G[0] = g00;
    p.G[1] = g01;
    p.G[2] = g11;
  }
  const float I = at.I[j];
  p.l2amp = lg2_approx(fabsf(I) * p.n);
  p.sgn = I < 0.f ? -1.f : 1.f;
  float xv[D];
#pragma unroll
  for (int a = 0; a < D; ++a) xv[a] = at.x[(size_t)D * j + a];
#pragma unroll
  // q* = (B^{-1} x)[k] with B^{-1} carried as wt + wl: a dual row rounded to
  // FP32 alone moves the centre by up to ~4e-8, which for the sharpest atoms
  // (r ~ 50) is a 2e-5 relative change of the basis at half its peak
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float hi, lo;
    dot2<D>(f.wt[k], xv, hi, lo);
#pragma unroll
    for (int a = 0; a < D; ++a) {
      // (a staged frame's residues lie in shared memory: no read-only load)
      float w;
      if constexpr (STAGED) w = f.wl[k * D + a];
      else w = __ldg(f.wl + k * D + a);
      lo = fmaf(w, xv[a], lo);
    }
    two_sum(hi, lo, p.qh[k], p.ql[k]);
  }

  // support box of m <= 1: |d_i| <= sqrt((G^{-1})_ii)
  float hw[K];
  bool ok;
  if constexpr (K == 1) {
    ok = p.G[0] > 0.f && qtt > 0.f;
    hw[0] = rsqrtf(p.G[0]);
  } else {
    float det = p.G[0] * p.G[2] - p.G[1] * p.G[1];
    ok = p.G[0] > 0.f && det > 0.f && qtt > 0.f;
    float idet = 1.f / det;
    hw[0] = sqrtf(p.G[2] * idet);
    hw[1] = sqrtf(p.G[0] * idet);
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const DetAxis &ax = g.ax[k];
    // coordinates increase with the cell index (checked on the host)
    float c = (p.qh[k] - ax.first) * ax.inv_step;
    float h = hw[k] * ax.inv_step * 1.0001f + 1e-3f;
    float lo = ceilf(c - h), hi = floorf(c + h);
    bool fin = ok && (lo == lo) && (hi == hi) && fabsf(c) < 1e8f && h < 1e8f;
    p.lo[k] = fin ? max(0, (int)lo) : 1;
    p.hi[k] = fin ? min(ax.n - 1, (int)hi) : 0;
  }
  return ok;
}

// Squared Mahalanobis distance of cell offsets d from the centre.
template <int K>
__device__ __forceinline__ float quad(const Pair<K> &p, const float *d) {
  if constexpr (K == 1) return p.G[0] * d[0] * d[0];
  else return fmaf(d[0], fmaf(p.G[0], d[0], 2.f * p.G[1] * d[1]), p.G[2] * d[1] * d[1]);
}

// ---- pixel-integrated ("point spread") operator -------------------------
// Reference: GaussDictCode/bin/point_spread_functions.py.  A cell's value is
// the integral of the projection over the square cell of half-width s, by an
// 11-point (2D) or 11 x 11 (3D) rule over the cell clipped to the box
// +-rr around the atom centre, rr = 1 / min(diag r) (__Radius :24); the
// points sit at lo + t (hi - lo)/10, t = 1..11 (__rf2 :413, __rf3 :462) and
// the point values carry no m > 1 cut-off (__Rf :386).  A cell farther than
// rr + s from the centre is 0; an atom within s - rr of the cell centre gives
// the total mass I sqrt(pi/30)/(r00 r11) or I (pi/30)/(r00 r11 r22) (__total
// :60) with zero derivatives (__drf2 :924).  Distances are measured in the
// detector plane (orthonormal frames).
template <int K>
struct PsfPair {
  float rr, total;
  int lo[K], hi[K];  // cells that can be non-zero
};

template <int K>
__device__ __forceinline__ void psf_setup(const Atoms &at, int j, const Geom &g,
                                          const Pair<K> &p, bool ok, float s,
                                          PsfPair<K> &q) {
  constexpr int D = K + 1;
  float M[D][D];
  load_r<K>(at, j, M);
  float mn = fminf(M[0][0], M[1][1]);
  float prod = M[0][0] * M[1][1];
  if constexpr (K == 2) {
    mn = fminf(mn, M[2][2]);
    prod *= M[2][2];
  }
  q.rr = 1.f / mn;
  const float I = at.I[j];
  q.total = K == 1 ? I / prod * 0.32360019f : I / prod * 0.10471976f;  // sqrt(pi/30), pi/30
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const DetAxis &ax = g.ax[k];
    const float c = (p.qh[k] - ax.first) * ax.inv_step;
    // (no cell beyond rr + s counts; the slack covers how far an axis accepted as
    // uniform, to 1e-4 of a step a cell, strays from first + k / inv_step, and the
    // rounding of the centre, which counts on a detector far from the origin.  A
    // whole cell of slack doubled the cells looked at.)
    const float h = fmaf(q.rr + s + 1.2e-7f * (fabsf(p.qh[k]) + fabsf(ax.first)), ax.inv_step,
                         fmaf(1e-4f, (float)ax.n, 0.01f));
    const float lo = ceilf(c - h), hi = floorf(c + h);
    const bool fin = ok && (lo == lo) && (hi == hi) && fabsf(c) < 1e8f && h < 1e8f;
    q.lo[k] = fin ? max(0, (int)lo) : 1;
    q.hi[k] = fin ? min(ax.n - 1, (int)hi) : 0;
  }
}

// Kind of a cell: 0 empty, 1 total, 2 quadrature; fills the quadrature
// start (offset from the atom centre) and step per axis.
template <int K>
__device__ __forceinline__ int psf_cell_kind(const PsfPair<K> &q, const float *dc,
                                             float s, float *base, float *step) {
  float n2 = 0.f;
#pragma unroll
  for (int k = 0; k < K; ++k) n2 = fmaf(dc[k], dc[k], n2);
  const float n = sqrtf(n2);
  if (n + q.rr < s) return 1;
  if (n - q.rr > s) return 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float c = -dc[k];  // atom centre relative to the cell centre
    const float lo = fmaxf(c - q.rr, -s), hi = fminf(c + q.rr, s);
    step[k] = 0.1f * (hi - lo);
    base[k] = dc[k] + lo;     // point offsets from the atom centre: base + t step
  }
  return 2;
}

// A row of the 3D quadrature: its 11 points two to a register pair (1..10, then
// 11).  The form m(d) = t + d (u + G11 d) is scaled by -30 log2 e once (with the
// factor in each coefficient, a fused operation a pair less, every coefficient
// is rounded once more).
struct PsfRow {
  F2 d[5];
  float last, g, l2amp;
  F2 g2, amp;
  __device__ __forceinline__ PsfRow(float base, float step, float G11, float l2a) {
#pragma unroll
    for (int i = 0; i < 5; ++i)
      d[i] = f2_fma(f2((float)(2 * i + 1), (float)(2 * i + 2)), f2(step, step), f2(base, base));
    last = fmaf(11.f, step, base);
    g = G11;
    g2 = f2(g, g);
    l2amp = l2a;
    amp = f2(l2a, l2a);
  }
  // weights of points 2i + 1 and 2i + 2, and of point 11
  __device__ __forceinline__ F2 pair(int i, F2 u, F2 t) const {
    const F2 m = f2_fma(d[i], f2_fma(g2, d[i], u), t);
    float x, y;
    f2_get(f2_fma(m, f2(kNegThirtyLog2e, kNegThirtyLog2e), amp), x, y);
    return f2(ex2_approx(x), ex2_approx(y));
  }
  __device__ __forceinline__ float end(float u, float t) const {
    const float m = fmaf(last, fmaf(g, last, u), t);
    return ex2_approx(fmaf(m, kNegThirtyLog2e, l2amp));
  }
};

// Pixel integral of E = n exp(-30 m) (times |I| through l2amp) over the
// quadrature points; returns the sum of point values times the rule's scale.
// 3D: two points of a row at a time (packed FP32; 121 exponentials and about
// 350 other instructions a cell instead of 650).
template <int K>
__device__ __forceinline__ float psf_quadrature(const Pair<K> &p, const float *base,
                                                const float *step) {
  if constexpr (K == 1) {
    float sum = 0.f;
#pragma unroll
    for (int t = 1; t <= 11; ++t) {
      const float d = fmaf((float)t, step[0], base[0]);
      sum += ex2_approx(fmaf(p.G[0] * d * d, kNegThirtyLog2e, p.l2amp));
    }
    return sum * (10.f * step[0] / 11.f);
  } else {
    const PsfRow row(base[1], step[1], p.G[2], p.l2amp);
    F2 sum = f2(0.f, 0.f);
    float sum1 = 0.f;
#pragma unroll 1
    for (int t = 1; t <= 11; ++t) {
      const float d0 = fmaf((float)t, step[0], base[0]);
      const float t0 = p.G[0] * d0 * d0, u = 2.f * p.G[1] * d0;
      const F2 tp = f2(t0, t0), up = f2(u, u);
#pragma unroll
      for (int i = 0; i < 5; ++i) sum = f2_add(sum, row.pair(i, up, tp));
      sum1 += row.end(u, t0);
    }
    float s0, s1;
    f2_get(sum, s0, s1);
    return ((s0 + s1) + sum1) * (100.f * step[0] * step[1] / 121.f);
  }
}

// Reduce-scatter of 32 values over the warp (recursive halving): on return
// v[0] of lane l is the sum over all lanes of their v[l].  At the step with
// offset m each lane keeps the half of its remaining values whose index bit m
// matches its lane bit and receives the partner's copy of that half.
__device__ __forceinline__ void warp_reduce_scatter32(float (&v)[32], int lane) {
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) {
    const bool up = (lane & m) != 0;
#pragma unroll
    for (int k = 0; k < m; ++k) {
      const float keep = up ? v[k + m] : v[k];
      const float give = up ? v[k] : v[k + m];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, give, m);
    }
  }
}

// Sums of FP32 pairs (value and compensation): (s, c) += (t, d).
__device__ __forceinline__ void pair_add(float &s, float &c, float t, float d) {
  float h, e;
  two_sum(s, t, h, e);
  s = h;
  c += d + e;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// A block's NW warps (every thread calls it) sum n FP64 partials (written by other
// blocks before a __threadfence) in a fixed order and write the total to *out.  A
// dependent FP64 add takes about 64 cycles on this GPU, so thread k keeps 4 running
// sums over elements k + NW*32*(4 i + s), chains of n / (128 NW) adds; the threads'
// sums are combined pairwise, across each warp, then across the warps in order.
template <int NW>
__device__ __forceinline__ void sum_partials_block(const double *part, int n, double *out) {
  constexpr int T = NW * 32;
  constexpr int kSums = 4;
  __shared__ double ws[NW];
  const int tid = threadIdx.x;
  double s[kSums];
#pragma unroll
  for (int k = 0; k < kSums; ++k) s[k] = 0.0;
  for (int base = 0; base < n; base += T * kSums) {
#pragma unroll
    for (int k = 0; k < kSums; ++k) {
      const int i = base + T * k + tid;
      if (i < n) s[k] += __ldcg(part + i);
    }
  }
  s[0] += s[1];
  s[2] += s[3];
  const double t = warp_sum_d(s[0] + s[2]);
  if ((tid & 31) == 0) ws[tid >> 5] = t;
  __syncthreads();
  if (tid == 0) {
    double tot = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) tot += ws[w];
    *out = tot;
  }
}

}  // namespace gr
