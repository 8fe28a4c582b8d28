// Rendering atoms on a voxel grid (sm_103a).
//
// Replaces __VolProj (GaussDictCode/bin/NewtonBases2D.py:261-271,
// GaussDictCode/bin/NewtonBases.py:700-711), which evaluates every atom at
// every voxel:  u(y) = sum_j I_j sqrt(30/pi) exp(-30 |r_j (y - x_j)|^2) where
// |r_j (y - x_j)| <= 1, else 0 (NewtonBases.py:42-46).
// One CTA per voxel tile; the CTA scans the atoms in index order, keeps those
// whose support box (the ellipsoid |r (y - x)| <= 1, whose half-extent along
// axis i is the norm of row i of r^{-1}) meets the tile, compacting them into
// shared memory in atom order; each thread owns one voxel and adds the listed
// atoms in that order.  Deterministic, no atomics.  Coordinate vectors must be
// monotone (the tile box is read from the tile's end coordinates).
#include "gr_kernels.cuh"

namespace gr {

constexpr int kVolThreads = 256;

struct VolGrid {
  int n[3];
  const float *y[3];
};

// Voxel-integrated value of one atom (point_spread_functions.py __if2 :425,
// __if3 :459): 11^D-point rule over the voxel of half-width s clipped to the
// box +-rr (rr = 1 / min diag r) around the atom, points at lo + t (hi-lo)/10
// (t = 1..11), no cut-off; total mass inside, zero beyond rr + s.
template <int D>
__device__ __forceinline__ float psf_voxel(float Iv, const float *X, const float (&M)[3][3],
                                           float rr, float total, float s) {
  float n2 = 0.f;
#pragma unroll
  for (int i = 0; i < D; ++i) n2 = fmaf(X[i], X[i], n2);
  const float n = sqrtf(n2);
  if (n + rr < s) return total;
  if (n - rr > s) return 0.f;
  float lo[3], st[3];
#pragma unroll
  for (int i = 0; i < D; ++i) {
    const float l = fmaxf(X[i] - rr, -s), h = fminf(X[i] + rr, s);
    st[i] = 0.1f * (h - l);
    lo[i] = l;
  }
  float sum = 0.f;
  for (int a = 1; a <= 11; ++a) {
    const float Y0 = fmaf((float)a, st[0], lo[0]) - X[0];
    for (int b = 1; b <= 11; ++b) {
      const float Y1 = fmaf((float)b, st[1], lo[1]) - X[1];
      if (D == 2) {
        const float p0 = M[0][0] * Y0 + M[0][1] * Y1, p1 = M[1][1] * Y1;
        sum += ex2_approx((p0 * p0 + p1 * p1) * kNegThirtyLog2e);
      } else {
#pragma unroll
        for (int c = 1; c <= 11; ++c) {
          const float Y2 = fmaf((float)c, st[2], lo[2]) - X[2];
          const float p0 = M[0][0] * Y0 + M[0][1] * Y1 + M[0][2] * Y2;
          const float p1 = M[1][1] * Y1 + M[1][2] * Y2, p2 = M[2][2] * Y2;
          sum += ex2_approx((p0 * p0 + p1 * p1 + p2 * p2) * kNegThirtyLog2e);
        }
      }
    }
  }
  constexpr float kNorm = 3.0901936161855166f;  // sqrt(30 / pi)
  return D == 2 ? Iv * kNorm * sum * (100.f * st[0] * st[1] / 121.f)
                : Iv * kNorm * sum * (1000.f * st[0] * st[1] * st[2] / 1331.f);
}

template <int D, bool PSF>
__global__ void __launch_bounds__(kVolThreads)
    gr_volproj_kernel(Atoms at, VolGrid vg, int t0, int t1, int t2, float s, float *u) {
  static_assert(D == 2 || PSF, "3D point values: gr_volproj3_kernel");
  __shared__ float sI[kVolThreads], sx[3][kVolThreads], sr[6][kVolThreads];
  __shared__ int wcount[kVolThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // tile extents: D == 3: t0 x t1 x t2 voxels; D == 2: t0 x t1
  const int nt1 = (vg.n[1] + t1 - 1) / t1;
  const int nt2 = D == 3 ? (vg.n[2] + t2 - 1) / t2 : 1;
  int b = blockIdx.x;
  const int b2 = b % nt2;
  b /= nt2;
  const int b1 = b % nt1, b0 = b / nt1;
  const int o0 = b0 * t0, o1 = b1 * t1, o2 = b2 * (D == 3 ? t2 : 1);
  // this thread's voxel
  const int l2 = D == 3 ? tid % t2 : 0;
  const int l1 = D == 3 ? (tid / t2) % t1 : tid % t1;
  const int l0 = D == 3 ? tid / (t1 * t2) : tid / t1;
  const int i0 = o0 + l0, i1 = o1 + l1, i2 = o2 + l2;
  const bool inside = i0 < vg.n[0] && i1 < vg.n[1] && (D == 2 || i2 < vg.n[2]);
  float yv[3] = {0.f, 0.f, 0.f};
  if (inside) {
    yv[0] = vg.y[0][i0];
    yv[1] = vg.y[1][i1];
    if (D == 3) yv[2] = vg.y[2][i2];
  }
  // coordinate box of the tile
  float blo[3], bhi[3];
  {
    const int e0 = min(o0 + t0, vg.n[0]) - 1, e1 = min(o1 + t1, vg.n[1]) - 1;
    const float a0 = vg.y[0][o0], c0 = vg.y[0][e0], a1 = vg.y[1][o1], c1 = vg.y[1][e1];
    blo[0] = fminf(a0, c0); bhi[0] = fmaxf(a0, c0);
    blo[1] = fminf(a1, c1); bhi[1] = fmaxf(a1, c1);
    if (D == 3) {
      const int e2 = min(o2 + t2, vg.n[2]) - 1;
      const float a2 = vg.y[2][o2], c2 = vg.y[2][e2];
      blo[2] = fminf(a2, c2); bhi[2] = fmaxf(a2, c2);
    }
  }
  constexpr float kNorm = 3.0901936161855166f;  // sqrt(30 / pi)
  float acc = 0.f;
  for (int base = 0; base < at.n; base += kVolThreads) {
    const int j = base + tid;
    bool hit = false;
    float M[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    float xj[3] = {0.f, 0.f, 0.f};
    if (j < at.n) {
      float Mk[D][D];
      load_r<D - 1>(at, j, Mk);
#pragma unroll
      for (int a = 0; a < D; ++a)
#pragma unroll
        for (int c = 0; c < D; ++c) M[a][c] = Mk[a][c];
#pragma unroll
      for (int i = 0; i < D; ++i) xj[i] = at.x[(size_t)D * j + i];
      // rows of r^{-1} for the upper-triangular r (back substitution)
      float inv[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
      bool ok = true;
#pragma unroll
      for (int i = 0; i < D; ++i) ok = ok && M[i][i] != 0.f;
      if (ok) {
#pragma unroll
        for (int c = D - 1; c >= 0; --c) {
          inv[c][c] = 1.f / M[c][c];
#pragma unroll
          for (int rr = c - 1; rr >= 0; --rr) {
            float s = 0.f;
#pragma unroll
            for (int k = rr + 1; k <= c; ++k) s += M[rr][k] * inv[k][c];
            inv[rr][c] = -s / M[rr][rr];
          }
        }
        hit = true;
        float rr = M[0][0];
#pragma unroll
        for (int i = 1; i < D; ++i) rr = fminf(rr, M[i][i]);
        rr = 1.f / rr;
#pragma unroll
        for (int i = 0; i < D; ++i) {
          float e = 0.f;
#pragma unroll
          for (int k = 0; k < D; ++k) e += inv[i][k] * inv[i][k];
          e = PSF ? (rr + s) * 1.0001f : sqrtf(e) * 1.0001f;
          hit = hit && (xj[i] + e >= blo[i]) && (xj[i] - e <= bhi[i]);
        }
      }
    }
    // ordered compaction of the hits of this chunk
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wcount[warp] = __popc(bal);
    __syncthreads();
    int off = 0, total = 0;
    for (int w = 0; w < kVolThreads / 32; ++w) {
      if (w < warp) off += wcount[w];
      total += wcount[w];
    }
    if (hit) {
      const int pos = off + __popc(bal & ((1u << lane) - 1u));
      sI[pos] = at.I[j] * kNorm;
#pragma unroll
      for (int i = 0; i < 3; ++i) sx[i][pos] = xj[i];
      sr[0][pos] = M[0][0];
      sr[1][pos] = M[1][1];
      sr[2][pos] = M[0][1];
      if (D == 3) {
        sr[2][pos] = M[2][2];
        sr[3][pos] = M[0][1];
        sr[4][pos] = M[1][2];
        sr[5][pos] = M[0][2];
      }
    }
    __syncthreads();
    if (inside) {
      for (int k = 0; k < total; ++k) {
        if constexpr (!PSF) {
          const float Y0 = yv[0] - sx[0][k], Y1 = yv[1] - sx[1][k];
          const float a = sr[0][k] * Y0 + sr[2][k] * Y1, c = sr[1][k] * Y1;
          const float nn = a * a + c * c;
          if (nn <= 1.f) acc += sI[k] * ex2_approx(nn * kNegThirtyLog2e);
        }
        if (PSF) {
          float Mk[3][3] = {{sr[0][k], D == 2 ? sr[2][k] : sr[3][k], D == 2 ? 0.f : sr[5][k]},
                            {0.f, sr[1][k], D == 2 ? 0.f : sr[4][k]},
                            {0.f, 0.f, D == 2 ? 0.f : sr[2][k]}};
          float X[3] = {sx[0][k] - yv[0], sx[1][k] - yv[1], D == 3 ? sx[2][k] - yv[2] : 0.f};
          float mn = Mk[0][0];
#pragma unroll
          for (int i = 1; i < D; ++i) mn = fminf(mn, Mk[i][i]);
          const float rr = 1.f / mn;
          constexpr float kNormV = 3.0901936161855166f;
          const float Iv = sI[k] / kNormV;
          const float det = D == 2 ? Mk[0][0] * Mk[1][1] : Mk[0][0] * Mk[1][1] * Mk[2][2];
          const float total = D == 2 ? Iv / det * 0.32360019f : Iv / det * 0.10471976f;
          acc += psf_voxel<D>(Iv, X, Mk, rr, total, s);
        }
      }
    }
    __syncthreads();
  }
  if (inside) {
    const size_t gi = D == 3 ? (((size_t)i0 * vg.n[1] + i1) * vg.n[2] + i2)
                             : ((size_t)i0 * vg.n[1] + i1);
    u[gi] = acc;
  }
}

// ---- 3D, point values -------------------------------------------------------
// A block of 256 threads owns V0 x 16 x 16 voxels (W0 = 1; V0 = 8 on large grids) or
// 4 x 8 x 8 (W0 = 4, V0 = 1), a warp V0 x 4 x 8 of them: a lane a column of V0 voxels
// along axis 0, its sums in registers.  The block finds the atoms that meet its
// voxels, kAtoms at a time (a thread each, so an atom is set up once per 2048 voxels),
// and stages them in index order; each warp ballots them against its own voxels, 32 at
// a time, and adds those left; with a voxel a lane it takes all 32 where kVolMost of
// them are left (a loop of known ends hides the latency of the staged values).
// Voxels sum their atoms in index order, as above.
// What bounds it: the scan of all atoms by every block (1000 atoms on 128 x 124
// x 120 voxels: 13.2 us; with 256 voxels a block, one per thread, 65.7 us: eight
// times the scans, and every listed atom evaluated at every voxel of the tile), on
// small grids the latency of a lane's chain of atoms (4000 atoms on 31^3, r = 1.2 and
// 8: 1 x 16 x 16 tiles 289 and 27 us, 4 x 8 x 8 158 and 29).
constexpr int kVolMost = 12;
template <int V0, int W0>
__global__ void __launch_bounds__(kVolThreads)
    gr_volproj3_kernel(Atoms at, VolGrid vg, float *u) {
  constexpr int kAtoms = kVolThreads;
  constexpr int NWarp = kVolThreads / 32;
  constexpr int W1 = W0 == 1 ? 4 : 2, W2 = NWarp / W0 / W1;   // warps along axes 1, 2
  constexpr int T0 = V0 * W0, T1 = 4 * W1, T2 = 8 * W2;       // the tile
  // centre, r (r00 r11 r22 r01 r12 r02), intensity; half-extents of the support
  __shared__ float4 sX[kAtoms], sR[kAtoms], sQ[kAtoms];
  __shared__ float2 sE[kAtoms];
  __shared__ float sE0[W0 > 1 ? kAtoms : 1];
  __shared__ int wcount[NWarp];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt1 = (vg.n[1] + T1 - 1) / T1, nt2 = (vg.n[2] + T2 - 1) / T2;
  int b = blockIdx.x;
  const int b2 = b % nt2;
  b /= nt2;
  const int b1 = b % nt1, b0 = b / nt1;
  const int o0 = b0 * T0, o1 = b1 * T1, o2 = b2 * T2;
  // the warp's voxels: 4 x 8 columns of V0
  const int w0 = o0 + V0 * (warp / (W1 * W2));
  const int w1 = o1 + 4 * (warp / W2 % W1), w2 = o2 + 8 * (warp % W2);
  const int i1 = w1 + (lane >> 3), i2 = w2 + (lane & 7);
  const bool inside = i1 < vg.n[1] && i2 < vg.n[2];
  const int n0 = min(V0, vg.n[0] - w0);
  float y0[V0], acc[V0];
#pragma unroll
  for (int k = 0; k < V0; ++k) {
    y0[k] = vg.y[0][min(w0 + k, vg.n[0] - 1)];
    acc[k] = 0.f;
  }
  const float y1 = vg.y[1][min(i1, vg.n[1] - 1)], y2 = vg.y[2][min(i2, vg.n[2] - 1)];
  // coordinate boxes (coordinates are monotone) of the tile and of the warp
  auto box = [&](int axis, int first, int n, float &lo, float &hi) {
    const int a = min(first, vg.n[axis] - 1), c = min(first + n, vg.n[axis]) - 1;
    const float p = vg.y[axis][a], q = vg.y[axis][max(c, a)];
    lo = fminf(p, q);
    hi = fmaxf(p, q);
  };
  float blo[3], bhi[3], wlo[3], whi[3];
  box(0, o0, T0, blo[0], bhi[0]);
  box(1, o1, T1, blo[1], bhi[1]);
  box(2, o2, T2, blo[2], bhi[2]);
  box(0, w0, V0, wlo[0], whi[0]);
  box(1, w1, 4, wlo[1], whi[1]);
  box(2, w2, 8, wlo[2], whi[2]);
  constexpr float kNorm = 3.0901936161855166f;  // sqrt(30 / pi)
  for (int base = 0; base < at.n; base += kAtoms) {
    const int j = base + tid;
    bool hit = false;
    float M[3][3] = {}, x[3] = {0.f, 0.f, 0.f}, e[3] = {0.f, 0.f, 0.f};
    if (j < at.n) {
      load_r<2>(at, j, M);
#pragma unroll
      for (int i = 0; i < 3; ++i) x[i] = at.x[(size_t)3 * j + i];
      if (M[0][0] != 0.f && M[1][1] != 0.f && M[2][2] != 0.f) {
        // half-extents: norms of the rows of r^{-1} (back substitution)
        const float i0 = 1.f / M[0][0], i1r = 1.f / M[1][1], i2r = 1.f / M[2][2];
        const float a12 = -M[1][2] * i2r * i1r, a01 = -M[0][1] * i1r * i0;
        const float a02 = -(M[0][1] * a12 + M[0][2] * i2r) * i0;
        e[2] = fabsf(i2r) * 1.0001f;
        e[1] = sqrtf(i1r * i1r + a12 * a12) * 1.0001f;
        e[0] = sqrtf(i0 * i0 + a01 * a01 + a02 * a02) * 1.0001f;
        hit = true;
#pragma unroll
        for (int i = 0; i < 3; ++i)
          hit = hit && (x[i] + e[i] >= blo[i]) && (x[i] - e[i] <= bhi[i]);
      }
    }
    // ordered compaction of the hits of this chunk
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) wcount[warp] = __popc(bal);
    __syncthreads();
    int off = 0, total = 0;
#pragma unroll
    for (int w = 0; w < NWarp; ++w) {
      if (w < warp) off += wcount[w];
      total += wcount[w];
    }
    if (hit) {
      const int pos = off + __popc(bal & ((1u << lane) - 1u));
      sX[pos] = make_float4(x[0], x[1], x[2], at.I[j] * kNorm);
      sR[pos] = make_float4(M[0][0], M[0][1], M[0][2], 0.f);
      sQ[pos] = make_float4(M[1][1], M[1][2], M[2][2], 0.f);
      sE[pos] = make_float2(e[1], e[2]);
      if constexpr (W0 > 1) sE0[pos] = e[0];
    }
    __syncthreads();
    for (int k0 = 0; k0 < total; k0 += 32) {
      const int k = k0 + lane;
      bool mine = false;
      if (k < total) {
        const float4 X = sX[k];
        const float2 E = sE[k];
        mine = X.y + E.x >= wlo[1] && X.y - E.x <= whi[1] && X.z + E.y >= wlo[2] &&
               X.z - E.y <= whi[2];
        // (with one warp along axis 0 the tile's test there was its own)
        if constexpr (W0 > 1)
          mine = mine && X.x + sE0[k] >= wlo[0] && X.x - sE0[k] <= whi[0];
      }
      unsigned m = __ballot_sync(0xffffffffu, mine);
      auto add = [&](int q) {
        const float4 X = sX[q], R = sR[q], Q = sQ[q];
        const float Y1 = y1 - X.y, Y2 = y2 - X.z;
        const float t = fmaf(R.y, Y1, R.z * Y2);
        const float c = fmaf(Q.x, Y1, Q.y * Y2), d = Q.z * Y2;
        const float cd = fmaf(c, c, d * d);
#pragma unroll
        for (int k2 = 0; k2 < V0; ++k2) {
          const float a = fmaf(R.x, y0[k2] - X.x, t);
          const float nn = fmaf(a, a, cd);
          if (nn <= 1.f) acc[k2] = fmaf(X.w, ex2_approx(nn * kNegThirtyLog2e), acc[k2]);
        }
      };
      if (V0 == 1 && __popc(m) >= kVolMost) {
        const int end = min(k0 + 32, total);
#pragma unroll 8
        for (int q = k0; q < end; ++q) add(q);
        continue;
      }
      while (m) {
        add(k0 + __ffs(m) - 1);
        m &= m - 1;
      }
    }
    __syncthreads();
  }
  if (inside)
#pragma unroll
    for (int k = 0; k < V0; ++k)
      if (k < n0) u[((size_t)(w0 + k) * vg.n[1] + i1) * vg.n[2] + i2] = acc[k];
}

// 3D point values: the most voxels a lane (of 8, 4, 2 along axis 0) that still
// gives two blocks an SM: a block scans all atoms, so few blocks of many voxels
// leave the SMs idle (16 blocks for 32^3 voxels).  Smaller grids: a voxel a lane in
// compact tiles, which fewer atoms meet (48^3, 4000 atoms, r = 2.4: 111 us in tiles of
// 2 x 16 x 16, 95 in 4 x 8 x 8; 64^3: 119 and 137).
constexpr int kVolBlocks = 304;
int launch_volproj(const Atoms &at, int dim, const int *n, const float *const *y,
                   float *u, int psf, float s, cudaStream_t stream) {
  VolGrid vg;
  for (int k = 0; k < 3; ++k) {
    vg.n[k] = k < dim ? n[k] : 1;
    vg.y[k] = k < dim ? y[k] : nullptr;
  }
  if (dim == 2) {
    const int t0 = 16, t1 = 16;
    const int blocks = ((vg.n[0] + t0 - 1) / t0) * ((vg.n[1] + t1 - 1) / t1);
    if (psf) gr_volproj_kernel<2, true><<<blocks, kVolThreads, 0, stream>>>(at, vg, t0, t1, 1, s, u);
    else gr_volproj_kernel<2, false><<<blocks, kVolThreads, 0, stream>>>(at, vg, t0, t1, 1, s, u);
  } else {
    if (!psf) {
      auto nb = [&](int t0, int t1, int t2) {
        return ((vg.n[0] + t0 - 1) / t0) * ((vg.n[1] + t1 - 1) / t1) * ((vg.n[2] + t2 - 1) / t2);
      };
      const int b8 = nb(8, 16, 16), b4 = nb(4, 16, 16), b2 = nb(2, 16, 16), b1 = nb(4, 8, 8);
      if (b8 >= kVolBlocks) gr_volproj3_kernel<8, 1><<<b8, kVolThreads, 0, stream>>>(at, vg, u);
      else if (b4 >= kVolBlocks) gr_volproj3_kernel<4, 1><<<b4, kVolThreads, 0, stream>>>(at, vg, u);
      else if (b2 >= kVolBlocks) gr_volproj3_kernel<2, 1><<<b2, kVolThreads, 0, stream>>>(at, vg, u);
      else gr_volproj3_kernel<1, 4><<<b1, kVolThreads, 0, stream>>>(at, vg, u);
      note_launches(1);
      return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
    }
    const int t0 = 4, t1 = 8, t2 = 8;
    const int blocks = ((vg.n[0] + t0 - 1) / t0) * ((vg.n[1] + t1 - 1) / t1) *
                       ((vg.n[2] + t2 - 1) / t2);
    gr_volproj_kernel<3, true><<<blocks, kVolThreads, 0, stream>>>(at, vg, t0, t1, t2, s, u);
  }
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

int preload_volume() {
  return preload_fn(gr_volproj_kernel<2, false>) + preload_fn(gr_volproj3_kernel<8, 1>) +
         preload_fn(gr_volproj3_kernel<4, 1>) + preload_fn(gr_volproj3_kernel<2, 1>) +
         preload_fn(gr_volproj3_kernel<1, 4>) +
         preload_fn(gr_volproj_kernel<2, true>) + preload_fn(gr_volproj_kernel<3, true>);
}

}  // namespace gr
