// Forward projection of Gaussian atoms (sm_103a).
//
// Replaces the reference's dense per-cell loops __RadProj
// (GaussDictCode/bin/NewtonBases2D.py:286-296) and __RadProj_3D/_2p5D
// (GaussDictCode/bin/NewtonBases.py:731-756), which evaluate every atom at
// every detector cell.  Here:
//   1. binning (gr_bin_kernel, gr_bin3d_kernel): per (atom, angle) pair,
//      compute the support box of m <= 1, write the pair's projection data and
//      set the atom's bit in the bitmap of every detector tile the box touches
//      (bits only, so the bitmap does not depend on the order in which pairs
//      run).
//   2. gr_project3d_kernel (3D / 2.5D detectors) and gr_project1d_kernel
//      (2D sinograms): a block per (angle, tile) item, the cells' sums in
//      registers.  Every cell meets the tile's atoms in increasing index order
//      and adds them with a compensated add and no float atomics, so results
//      are bitwise reproducible.  The epilogue writes the sinogram and, fused,
//      the residual or KL weight fields and per-tile loss partials.
//   3. gr_loss_finalize_kernel: fixed-order FP64 sum of the loss partials.
#include "gr_kernels.cuh"

namespace gr {

// 2D binning: the body of a 128-thread block, atoms bx * 128 .., angle a (the
// launch's block (bx, a); a multi-problem launch maps its blocks to (problem,
// bx, a)).  pairs (nullable): the pair's projection data as the projection
// stages it, two float4 per (angle, atom) at [a n + j], written here once
// instead of being recomputed by every tile the atom touches.
__device__ __forceinline__ void bin_body(const Atoms &at, const Geom &g, const TileCfg &tc,
                                         uint32_t *bitmap, int W, float4 *pairs, int bx, int a) {
  const int j = bx * 128 + (int)threadIdx.x;
  const uint32_t bit = 1u << (j & 31);
  const size_t base = (size_t)a * tc.ntiles;
  const int wj = j >> 5;
  // a warp holds 32 consecutive atoms: one bitmap word per tile.  Their
  // bits are merged per tile across the warp (one atomicOr per tile the
  // warp touches, not one per atom and tile: the 32 atoms of a word would
  // otherwise all hit the same address)
  int t_lo = 1 << 30, t_hi = -1;
  if (j < at.n) {
    Frame<1> f;
    load_frame<1>(g.frames, a, f);
    Pair<1> p;
    pair_setup<1>(at, j, f, g, p);
    if (pairs) {
      // (the sign of I rides on G's, which is >= 0)
      pairs[(size_t)a * at.n + j] =
          make_float4(p.qh[0], p.ql[0], copysignf(p.G[0], p.sgn), p.l2amp);
    }
    if (p.lo[0] <= p.hi[0]) {
      t_lo = p.lo[0] / tc.t0;
      t_hi = p.hi[0] / tc.t0;
    }
  }
  const int w_lo = __reduce_min_sync(0xffffffffu, t_lo);
  const int w_hi = __reduce_max_sync(0xffffffffu, t_hi);
  for (int t = w_lo; t <= w_hi; ++t) {
    const unsigned bits = __reduce_or_sync(0xffffffffu, (t >= t_lo && t <= t_hi) ? bit : 0u);
    if ((threadIdx.x & 31) == 0 && bits) atomicOr(bitmap + (base + t) * W + wj, bits);
  }
}

__global__ void __launch_bounds__(128) gr_bin_kernel(Atoms at, Geom g, TileCfg tc,
                                                     uint32_t *bitmap, int W, float4 *pairs) {
  bin_body(at, g, tc, bitmap, W, pairs, blockIdx.x, blockIdx.y);
}

// Per-cell KL term f log(f/g) - f + g = g h(u), u = f/g, h(u) = u log u - u + 1,
// evaluated without cancellation: a series in e = u - 1 near u = 1.
__device__ __forceinline__ float kl_term(float f, float g) {
  if (!(f > 0.f)) return g;
  const float e = (f - g) / g;
  float h;
  if (fabsf(e) < 0.125f) {
    // h = sum_{k>=2} (-1)^k e^k / (k (k-1))
    float e2 = e * e;
    h = e2 * (0.5f + e * (-1.f / 6.f + e * (1.f / 12.f + e * (-1.f / 20.f +
             e * (1.f / 30.f + e * (-1.f / 42.f + e * (1.f / 56.f)))))));
  } else {
    const float u = f / g;
    h = u * logf(u) - u + 1.f;
  }
  return g * h;
}

// 3D detectors: a block of NW warps per (angle, tile) item, tile 4 NW x 32
// cells.  Each cell's sum lives in the registers of one lane; the atoms come to
// the cells:
//   * the tile's atoms (its bitmap, increasing index) are taken in passes of
//     32 NW; a thread stages one atom's record (Proj3Rec: written once per
//     (atom, angle) by the binning launch) in shared memory and marks the
//     4 x 2 subtiles its ellipse meets; a 32 x 32 bit transpose per warp turns
//     the atoms' subtile bits into the subtiles' atom masks;
//   * a warp owns 16 x 8 cells, 16 subtiles, one per pair of lanes, 2 x 2
//     cells a lane; each pair of lanes walks its own subtile's mask, so a warp
//     step is 16 (subtile, atom) visits.
// A cell therefore adds its atoms in index order with an exact two-sum and a
// running compensation, whatever the tiling: results are bitwise reproducible
// and the same under every tile height.
// What bounds it: instruction issue (77 % of the slots on 8192 atoms x 2000
// orientations; DRAM under 10 %).  Per (atom, angle) pair of 22 in-support
// cells it issues 60 warp instructions: the visits 28, the masks' walk 15, the
// staging the rest.  One warp walking an atom's whole box over sums in shared
// memory, the layout before this one, issued 141: index arithmetic and the
// read-modify-write of the sums for every 32 box cells, two lanes in three
// active.  Why 2 x 2 cells a lane and 4 x 2 subtiles: of the shapes from
// 2 x 2 to 8 x 4 cells they gave the fewest warp steps times instructions for
// footprints of 20 to 140 cells; packed FP32 pairs do both rows at once.
// 8192 atoms x 20000 x 128^2 cells: binning + projection 23.6 -> 15.1 ms; 1000
// atoms x 1001 x 95^2: 185 -> 128 us; 2936 atoms x 148 x 493^2: 309 -> 260 us
// (there about half is the 73408 items' own work, some 600 warp instructions each;
// forwards of few atoms over many items are all that: 20 atoms x 600 x 200^2 105 us,
// 82 with a warp an item).  64 registers, 8 blocks an SM; 48 registers: 5 to 10 % slower.
struct Proj3Rec {
  float4 a;   // (-qh0, -ql0, -qh1, -ql1): the centre's negative, as a float pair
  float4 b;   // (G00, 2 G01, G11, log2 amplitude)
};

// The pair's record.  The sign of I rides on G00's (>= 0 where a record is
// written).
__device__ __forceinline__ Proj3Rec proj3_record(const Pair<2> &p) {
  Proj3Rec o;
  o.a = make_float4(-p.qh[0], -p.ql[0], -p.qh[1], -p.ql[1]);
  o.b = make_float4(copysignf(p.G[0], p.sgn), 2.f * p.G[1], p.G[2], p.l2amp);
  return o;
}

__device__ __forceinline__ float rcp_approx(float v) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
  return y;
}

// The subtiles of the tile (rows r0.., columns c0..) that the record's support
// ellipse meets: bit 16 (b % 2) + c of word b / 2 for rows r0 + 4 b .. + 3,
// columns c0 + 2 c, + 1.  Over a band of 4 rows the ellipse's column range is
// reached at the row nearest to its rightmost (leftmost) point; it is widened
// by 0.02 cells (approximate square roots, FP32 rounding near the ellipse's
// tips): the cells' own test decides.
template <int NB>
__device__ __forceinline__ void proj3_subtiles(const Proj3Rec &q, const Geom &g, int r0, int c0,
                                               uint32_t (&cols)[NB / 2]) {
  const float g00 = fabsf(q.b.x), g01 = 0.5f * q.b.y, g11 = q.b.z;
  const float det = fmaf(g00, g11, -g01 * g01);
  const float h0 = rcp_approx(g.ax[0].inv_step), i1 = g.ax[1].inv_step, i11 = rcp_approx(g11);
  const float q0 = (-q.a.x - g.ax[0].first) * g.ax[0].inv_step - (float)r0;   // centre in
  const float q1 = (-q.a.z - g.ax[1].first) * i1 - (float)c0;                 // tile cells
  const float S = -g01 * i11 * h0 * i1;                   // columns q1 + S d +- hw(d),
  const float k = i1 * sqrt_approx(i11);                  // hw(d) = k sqrt(1 - a2 d^2)
  const float a2 = det * i11 * h0 * h0;
  const float dmax = rcp_approx(sqrt_approx(a2));         // rows within dmax
  const float dx = S * dmax * rcp_approx(sqrt_approx(fmaf(S, S, k * k * a2)));  // of the rightmost
  const bool plain = fabsf(dx) < 1e8f && dmax < 1e8f;     // else every subtile
  const float top = q0 - dmax - 0.02f, bot = q0 + dmax + 0.02f;
#pragma unroll
  for (int w = 0; w < NB / 2; ++w) cols[w] = 0u;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const float ra = fmaxf(top, (float)(4 * b)), rb = fminf(bot, (float)(4 * b + 3));
    const float da = ra - q0, db = rb - q0;
    const float dr = fminf(fmaxf(dx, da), db), dl = fminf(fmaxf(-dx, da), db);
    const float hr = k * sqrt_approx(fmaxf(fmaf(-a2 * dr, dr, 1.f), 0.f));
    const float hl = k * sqrt_approx(fmaxf(fmaf(-a2 * dl, dl, 1.f), 0.f));
    const float xr = fminf(fmaf(S, dr, q1) + fmaf(hr, 1.0001f, 0.02f), 31.f);
    const float xl = fmaxf(fmaf(S, dl, q1) - fmaf(hl, 1.0001f, 0.02f), 0.f);
    const int xa = (int)ceilf(xl), xb = (int)floorf(xr);
    uint32_t m = xa <= xb && ra <= rb ? (2u << (xb >> 1)) - (1u << (xa >> 1)) : 0u;
    if (!plain) m = 0xffffu;
    cols[b / 2] |= m << (16 * (b % 2));
  }
}

// Bit transpose over the warp: bit i of lane l becomes bit l of lane i.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1) {
    const uint32_t lo = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu
                        : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    const bool up = (lane & j) != 0;
    const uint32_t rot = __funnelshift_l(y, y, up ? 32 - j : j);
    const uint32_t keep = up ? ~lo : lo;
    x = (x & keep) | (rot & ~keep);
  }
  return x;
}

// One visit: the record's values at a lane's 2 x 2 cells, added to their sums.
// row, col: the cells' coordinates; s, c: sums and compensations of the two
// cells of each column.
__device__ __forceinline__ void proj3_visit(const Proj3Rec &q, const float (&row)[2],
                                            const float (&col)[2], F2 (&s)[2], F2 (&c)[2]) {
  const float g00 = fabsf(q.b.x);
  float t[2], u[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float d0 = (row[r] + q.a.x) + q.a.y;
    t[r] = g00 * d0 * d0;
    u[r] = q.b.y * d0;
  }
  const float sg = copysignf(1.f, q.b.x);
  const F2 S = f2(sg, sg), tp = f2(t[0], t[1]);
  const F2 K2 = f2(kNegThirtyLog2e, kNegThirtyLog2e), amp = f2(q.b.w, q.b.w);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float d1 = (col[k] + q.a.z) + q.a.w;
    const F2 m = f2_fma(f2(d1, d1), f2(fmaf(q.b.z, d1, u[0]), fmaf(q.b.z, d1, u[1])), tp);
    float m0, m1, e0, e1;
    f2_get(m, m0, m1);
    f2_get(f2_fma(m, K2, amp), e0, e1);
    e0 = ex2_approx(e0);
    e1 = ex2_approx(e1);
    const F2 v = f2(m0 <= 1.f ? e0 : 0.f, m1 <= 1.f ? e1 : 0.f);
    // two-sum of s and S v, both cells at once
    const F2 tt = f2_fma(v, S, s[k]);
    const F2 nb = f2_sub(s[k], tt);
    const F2 w = f2_sub(s[k], f2_add(tt, nb));
    c[k] = f2_add(c[k], f2_add(w, f2_fma(v, S, nb)));
    s[k] = tt;
  }
}

// With loss_out, the last block to finish sums the items' loss partials in
// item order (no separate finalize launch).
// LIST: only the n_list[0] items of item_list are taken (those some atom
// meets; the loss partials of the others are already in place).
// rec (nullable): the (angle, atom) records; without it a thread sets its
// pairs up itself.
template <int NW, bool LIST>
__global__ void __launch_bounds__(NW * 32, 32 / NW)
    gr_project3d_kernel(Atoms at, Geom g, TileCfg tc, const uint32_t *bitmap, int W,
                        const Proj3Rec *__restrict__ rec, ProjOut out, int *next_item,
                        double *loss_out, const int *item_list, const int *n_list) {
  constexpr int T = NW * 32;            // threads
  constexpr int kWords = 2 * NW;        // 32-atom words per pass
  constexpr int kSub = 16 * NW;         // subtiles of the tile
  constexpr int kList = 1024;           // atoms listed at a time
  constexpr int kPitch = 36;
  // slot 33 k + 1 + l: the record of bit l of word k; slot 33 k adds nothing
  // (where a mask runs dry)
  __shared__ float4 sA[33 * kWords], sB[33 * kWords];
  __shared__ uint32_t sMask[kWords][kSub];
  __shared__ int list[kList];
  __shared__ int s_count[NW];
  __shared__ float sV[4 * NW][kPitch];
  __shared__ int s_item, s_last;
  __shared__ float2 s_loss[T];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_items = g.n_angles * tc.ntiles;
  const int D0 = g.ax[0].n, D1 = g.ax[1].n;
  // the lane's subtile and cells
  const int grp = lane >> 1;
  // (a warp's columns differ from block to block: a warp beyond the detector's last
  // column has no walk, and should not be the same scheduler's in every block)
  const int wcol = (warp + (int)blockIdx.x) & 3;
  const int band = 4 * (warp >> 2) + (grp >> 2), cpair = 4 * wcol + (grp & 3);
  const int row_in = 4 * band + 2 * (lane & 1), col_in = 2 * cpair;
  const int n_take = LIST ? *n_list : n_items;
  if (tid < kWords) {
    sA[33 * tid] = make_float4(0.f, 0.f, 0.f, 0.f);
    sB[33 * tid] = make_float4(0.f, 0.f, 0.f, __int_as_float(0xff800000));
  }

  // persistent blocks: the first item is the block's own, the others come from
  // a counter (asked for an item ahead), so heavy tiles do not hold the others
  // idle; what an item computes does not depend on which block takes it
  int take = blockIdx.x, done = -1;
  // the loss of the item done before: a column's cells as an FP32 pair, the columns in
  // FP64, by the first warp while it waits for the next item's data (s_loss is written
  // again behind that item's first barrier)
  auto close_loss = [&]() {
    if (!out.loss_part || done < 0 || warp != 0) return;
    float ls = s_loss[lane].x, lc = s_loss[lane].y;
#pragma unroll
    for (int w = 1; w < NW; ++w) pair_add(ls, lc, s_loss[32 * w + lane].x, s_loss[32 * w + lane].y);
    const double d = warp_sum_d((double)ls + (double)lc);
    if (lane == 0) out.loss_part[done] = d;
  };
  while (take < n_take) {
    int ahead = 0;
    if (tid == 0) ahead = (int)gridDim.x + atomicAdd(next_item, 1);
    const int item = LIST ? item_list[take] : take;
    const int a = tile_div(item, tc.ntiles, tc.inv_ntiles), t = item - a * tc.ntiles;
    const int tr = tile_div(t, tc.nt1, tc.inv_nt1), tcix = t - tr * tc.nt1;
    const int r0 = tr * (4 * NW), c0 = tcix * 32;
    // the tile's atoms: warp w counts the words [w per, (w + 1) per)
    const uint32_t *words = bitmap + (size_t)item * W;
    int per = (W + NW - 1) / NW;
    int wlo = min(W, warp * per), whi = min(W, wlo + per);
    uint32_t wd0 = wlo + lane < whi ? __ldg(words + wlo + lane) : 0u;
    int mine = __popc(wd0);
    for (int wb = wlo + 32 + lane; wb < whi; wb += 32) mine += __popc(__ldg(words + wb));
    // the epilogue's cells of this thread: rows 4 warp .. + 3, column lane;
    // their data is read before the atoms so that the epilogue does not wait
    const bool want_data = out.epilogue == kEpiL2 || out.epilogue == kEpiKL;
    const int er = r0 + 4 * warp, ec = c0 + lane;
    const int nr = ec < D1 ? min(4, D0 - er) : 0;   // its cells inside the detector
    const size_t gi0 = ((size_t)a * D0 + er) * D1 + ec;
    float dv[4] = {0.f, 0.f, 0.f, 0.f};
    if (want_data) {
      const float *src = out.data + gi0;
#pragma unroll
      for (int r = 0; r < 4; ++r, src += D1)
        if (r < nr) dv[r] = __ldg(src);
    }
    close_loss();
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) s_count[warp] = mine;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) total += s_count[w];

    if (total > 0) {
      float row[2], col[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        row[k] = r0 + row_in + k < D0 ? __ldg(g.ax[0].coords + r0 + row_in + k) : 0.f;
        col[k] = c0 + col_in + k < D1 ? __ldg(g.ax[1].coords + c0 + col_in + k) : 0.f;
      }
      F2 acc[2], cmp[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) acc[k] = cmp[k] = f2(0.f, 0.f);
      // all words at once where the list holds their atoms, else 32 words at
      // a time
      const int step = total <= kList ? W : 32;
      for (int wbase = 0; wbase < W; wbase += step) {
        int n_listed = total;
        if (step < W) {
          __syncthreads();              // s_count is read
          const int wi = wbase + lane;
          per = 32;
          wlo = warp == 0 ? wbase : W;  // the first warp lists them
          whi = warp == 0 ? min(W, wbase + 32) : W;
          wd0 = wi < W ? __ldg(words + wi) : 0u;
          n_listed = __reduce_add_sync(0xffffffffu, __popc(wd0));
          if (warp != 0) wd0 = 0u;
          if (lane == 0) s_count[warp] = warp == 0 ? n_listed : 0;
          __syncthreads();
          if (n_listed == 0) continue;
        }
        int at_pos = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w)
          if (w < warp) at_pos += s_count[w];
        for (int wb = wlo; wb < whi; wb += 32) {
          uint32_t wd = wb == wlo ? wd0 : (wb + lane < whi ? __ldg(words + wb + lane) : 0u);
          const int cnt = __popc(wd);
          int incl = cnt;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
          }
          int pos = at_pos + incl - cnt;
          while (wd) {
            list[pos++] = ((wb + lane) << 5) + (__ffs(wd) - 1);
            wd &= wd - 1;
          }
          at_pos += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();
        for (int first = 0; first < n_listed; first += 32 * kWords) {
          const int nwords = min(kWords, (n_listed - first + 31) >> 5);
          // bit l of a word is the (31 - l)-th of its atoms: a mask's highest
          // bit is its first atom
#pragma unroll
          for (int k0 = 0; k0 < kWords; k0 += NW) {
            const int k = k0 + warp;
            if (k >= nwords) break;     // (the warp leaves together)
            const int e = first + 32 * k + 31 - lane;
            uint32_t cols[NW / 2];
#pragma unroll
            for (int u = 0; u < NW / 2; ++u) cols[u] = 0u;
            if (e < n_listed) {
              const int j = list[e];
              Proj3Rec q;
              if (rec) {
                const Proj3Rec *p = rec + (size_t)a * at.n + j;
                q.a = __ldg(&p->a);
                q.b = __ldg(&p->b);
              } else {
                Frame<2> f;
                load_frame<2>(g.frames, a, f);
                Pair<2> p;
                pair_setup<2>(at, j, f, g, p);
                q = proj3_record(p);
              }
              sA[33 * k + 1 + lane] = q.a;
              sB[33 * k + 1 + lane] = q.b;
              proj3_subtiles<NW>(q, g, r0, c0, cols);
            }
#pragma unroll
            for (int u = 0; u < NW / 2; ++u)
              sMask[k][32 * u + lane] = warp_transpose32(cols[u], lane);
          }
          __syncthreads();
          // walk the subtile's masks; a step takes the next atom of the word,
          // or the first one of the next word (nothing if that one is empty)
          const char *pa = reinterpret_cast<const char *>(sA);
          const char *pb = reinterpret_cast<const char *>(sB);
          const uint32_t *pm = &sMask[0][16 * band + cpair];
          const bool off = c0 + 8 * wcol >= D1;
          uint32_t m = off ? 0u : *pm;
          int left = off ? 0 : nwords - 1;
          int base = 16;
          while (m != 0u || left > 0) {
            if (m == 0u) {
              pm += kSub;
              m = *pm;
              base += 33 * 16;
              --left;
            }
            const int i = 31 - __clz(m);              // -1: the empty slot
            m &= ~(1u << (i & 31));
            const int o = base + 16 * i;
            Proj3Rec q;
            q.a = *reinterpret_cast<const float4 *>(pa + o);
            q.b = *reinterpret_cast<const float4 *>(pb + o);
            proj3_visit(q, row, col, acc, cmp);
          }
          __syncthreads();  // the pass's staged records are done with
        }
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        float s0, s1, e0, e1;
        f2_get(acc[k], s0, s1);
        f2_get(cmp[k], e0, e1);
        sV[row_in][col_in + k] = __fadd_rn(s0, e0);
        sV[row_in + 1][col_in + k] = __fadd_rn(s1, e1);
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] = sV[4 * warp + r][lane];
    }

    // write the cells, fused fit fields and loss partial (rounding spelled
    // out, so that both forms of the kernel give the same bits)
    float lsum = 0.f, lcmp = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r >= nr) break;
      const size_t gi = gi0 + (size_t)(r * D1);
      if (out.R) out.R[gi] = v[r];
      float l = 0.f;
      if (out.epilogue == kEpiL2) {
        const float res = v[r] - dv[r];
        if (out.alpha) out.alpha[gi] = res;
        l = __fmul_rn(__fmul_rn(0.5f, res), res);
      } else if (out.epilogue == kEpiKL) {
        const float fo = dv[r];
        const float gg = v[r] + out.bg;
        const float ig = 1.f / gg;
        if (out.alpha) out.alpha[gi] = fmaf(-fo, ig, 1.f);
        if (out.beta) out.beta[gi] = __fmul_rn(__fmul_rn(fo, ig), ig);
        l = kl_term(fo, gg);
      }
      const float tt = lsum + l;
      lcmp += (fabsf(lsum) >= fabsf(l)) ? ((lsum - tt) + l) : ((l - tt) + lsum);
      lsum = tt;
    }
    if (out.loss_part) s_loss[tid] = make_float2(lsum, lcmp);
    if (tid == 0) s_item = ahead;
    __syncthreads();  // sV and s_count are reused
    take = s_item;
    done = item;
  }
  close_loss();

  if (loss_out && out.loss_part) {
    // the last block to finish sums the items' partials in item order (a flag of
    // its own: a slower warp may still have the last s_item to read)
    if (tid == 0) {
      __threadfence();
      s_last = atomicAdd(next_item + 1, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      sum_partials_block<NW>(out.loss_part, n_items, loss_out);
    }
  }
}

// Binning of a 3D forward: a block takes 256 atoms (8 bitmap words) of one
// angle, writes their records (rec, nullable) and gathers the tiles' words in
// shared memory, a range of kBinTiles tiles at a time, so that every word of
// the bitmap is written once: no clear, and no global atomics (whose latency
// and contention bounded the launch before).  Instruction issue bounds it (91 % of
// the slots, 500 a warp of pairs): four divisions by the tile's sides were a
// fifth of them (8192 atoms x 20000: 3.05 ms, 2.46 with shifts).  In a range a
// thread goes through its tiles there only (all of them in every range: 2.3 ms
// for one atom across 2048^2 cells, 1024 cells wide 600 atoms x 60: 272 us; 10 and
// 89 us so).  Where atoms and angles give few blocks, the ranges are dealt to
// blocks of their own (kBinFewBlocks, two an SM: one narrow atom x 2048^2 31 ->
// 3.6 us, 5000 x 1024^2 16.5 -> 5.6 us; from there on a block takes all ranges, so
// that a pair is set up once).
// counters (nullable): zeroed, for the projection that follows.
// Each block takes the ranges z, z + gridDim.z, ... of its atoms and angle.
constexpr int kBinTiles = 512;
constexpr int kBinOwnTiles = 32;
constexpr int kBinFewBlocks = 304;
__global__ void __launch_bounds__(256)
    gr_bin3d_kernel(Atoms at, Geom g, TileCfg tc, uint32_t *bitmap, int W, Proj3Rec *rec,
                    int *counters, uint32_t *flag, int *list, int *n_list) {
  __shared__ uint32_t sw[kBinTiles][8];
  const int tid = threadIdx.x, a = blockIdx.y, w0 = 8 * blockIdx.x;
  const int j = 32 * w0 + tid;
  if (counters && blockIdx.x == 0 && a == 0 && blockIdx.z == 0 && tid < 4) counters[tid] = 0;
  int r_lo = 1, r_hi = 0, c_lo = 1, c_hi = 0;
  if (j < at.n) {
    Frame<2> f;
    load_frame<2>(g.frames, a, f);
    Pair<2> p;
    pair_setup<2>(at, j, f, g, p);
    if (p.lo[0] <= p.hi[0] && p.lo[1] <= p.hi[1]) {
      const int sh = 31 - __clz(tc.t0);  // (16 or 32 rows a tile, 32 columns)
      r_lo = p.lo[0] >> sh;
      r_hi = p.hi[0] >> sh;
      c_lo = p.lo[1] / kTileDim1;
      c_hi = p.hi[1] / kTileDim1;
      if (rec && blockIdx.z == 0) rec[(size_t)a * at.n + j] = proj3_record(p);
    }
  }
  const uint32_t bit = 1u << (j & 31);
  const int nw = min(8, W - w0);
  const int first = kBinTiles * blockIdx.z, stride = kBinTiles * gridDim.z;
  for (int t0 = first; t0 < tc.ntiles; t0 += stride) {
    const int nt = min(kBinTiles, tc.ntiles - t0);
    if (t0 > first) __syncthreads();
    for (int e = tid; e < nt * 8; e += 256) (&sw[0][0])[e] = 0u;
    // the thread's tiles among these: rows of tiles r_a .. r_b, the first and
    // last of which may lie in the range only in part
    int r_a = r_lo, r_b = r_hi;
    if (nt < tc.ntiles) {
      r_a = max(r_a, tile_div(t0, tc.nt1, tc.inv_nt1));
      r_b = min(r_b, tile_div(t0 + nt - 1, tc.nt1, tc.inv_nt1));
    }
    const int width = c_hi - c_lo + 1, own = max(r_b - r_a + 1, 0) * width;
    __syncthreads();
    auto set = [&](int r, int c, uint32_t b) {
      const int t = r * tc.nt1 + c - t0;
      if (t >= 0 && t < nt) atomicOr(&sw[t][tid >> 5], b);
    };
    // a lane sets its own atom's tiles; where a few wide supports would keep the
    // others waiting (an atom's tiles shared out cost some four times as much a
    // tile), the lanes set theirs together
    uint32_t wide = __ballot_sync(0xffffffffu, own > kBinOwnTiles);
    if (wide && __reduce_add_sync(0xffffffffu, own) >= 8 * __reduce_max_sync(0xffffffffu, own))
      wide = 0u;
    if (!(wide >> (tid & 31) & 1u))
      for (int r = r_a; r <= r_b; ++r)
        for (int c = c_lo; c <= c_hi; ++c) set(r, c, bit);
    while (wide) {
      const int src = __ffs(wide) - 1;
      wide &= wide - 1;
      const int n = __shfl_sync(0xffffffffu, own, src), w = __shfl_sync(0xffffffffu, width, src);
      const int ra = __shfl_sync(0xffffffffu, r_a, src), ca = __shfl_sync(0xffffffffu, c_lo, src);
      for (int e = tid & 31; e < n; e += 32) set(ra + e / w, ca + e % w, 1u << src);
    }
    __syncthreads();
    const size_t base = (size_t)a * tc.ntiles + t0;
    for (int e0 = 0; e0 < nt * 8; e0 += 256) {
      const int e = e0 + tid;
      const uint32_t wd = e < nt * 8 ? (&sw[0][0])[e] : 0u;
      const int t = e >> 3, w = e & 7;
      if (e < nt * 8 && w < nw) bitmap[(base + t) * W + w0 + w] = wd;
      if (flag) {
        // an item is listed by the first block that meets it
        const uint32_t any = __ballot_sync(0xffffffffu, wd != 0u) >> (tid & 24);
        if (w == 0 && (any & 0xffu) && atomicExch(flag + base + t, 1u) == 0u)
          list[atomicAdd(n_list, 1)] = (int)(base + t);
      }
    }
  }
}

// 2D sinograms: atom footprints are a few cells wide, so a block owns a tile
// of 32 CPL consecutive cells of one angle, CPL cells per lane of every warp
// (lane l: cells l, l + 32, ...).  CPL = 2 (Tuning key 3, form 2) halves the
// tiles an atom of a wide footprint touches, and with them the listing,
// staging and binning per evaluated cell; narrow footprints leave more lanes
// idle in it.  The
// tile's atoms come from its bitmap in index order, in passes: a pass lists
// as many whole bitmap words as fit in NW*32 entries (block-wide prefix sum
// of the words' bit counts), every thread sets up the pair data of one listed
// atom in shared memory, and warp w adds the atoms of the w-th of NW
// contiguous slices of the pass's list to its lane's cell, in list order, in
// registers (compensated).  The warps' partial sums are combined in warp
// order: results depend only on the atoms listed, bitwise reproducible.
// LM: a pass lists up to LM * NW * 32 atoms (each thread stages LM of them),
// so tiles crossed by many atoms take fewer passes and barriers (2150 atoms x
// 153 angles: 87.9 us with one atom per thread, 82.6 with two, 79.5 with
// four; 512 atoms: 20.6, 20.7, 21.1 us).
// What bounds it: issue (81 % of the slots), some 17 instructions a cell and
// atom: one 16-byte record, the form, the exponential and the compensated sum,
// without a branch (with the support box in a second record and tests of it and
// of the form: 75 us where this takes 51.1; with the form's test alone as a
// branch 57.7; 64 cells a tile 68.8).
// The body of one block of the 2D projection: (angle, tile) item of n_items
// (the launch's block; a multi-problem launch maps its blocks to (problem,
// item)).
template <bool KAHAN, int NW, int CPL = 1, int LM = 1>
__device__ __forceinline__ void project1d_body(const Atoms &at, const Geom &g, const TileCfg &tc,
                                               const uint32_t *bitmap, int W, const ProjOut &out,
                                               double *loss_out, int *done,
                                               const float4 *__restrict__ pairs, int item,
                                               int n_items) {
  constexpr int T = NW * 32;
  constexpr int LT = LM * T;
  __shared__ float4 prm[LT];
  __shared__ int list[LT];
  __shared__ int wsum[NW];
  __shared__ float parts[NW][2][32 * CPL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = tile_div(item, tc.ntiles, tc.inv_ntiles), t = item - a * tc.ntiles;
  const int D0 = g.ax[0].n;
  int cell[CPL];
  float pc[CPL], acc[CPL], cmp[CPL];
#pragma unroll
  for (int k = 0; k < CPL; ++k) {
    cell[k] = t * tc.t0 + lane + 32 * k;
    pc[k] = cell[k] < D0 ? g.ax[0].coords[cell[k]] : 0.f;
    acc[k] = 0.f;
    cmp[k] = 0.f;
  }
  const float4 *apairs = pairs + (size_t)a * at.n;

  const uint32_t *words = bitmap + (size_t)item * W;
  for (int wb = 0; wb < W;) {
    // thread k holds word wb + k; inclusive prefix of the bit counts
    const int wi = wb + (int)threadIdx.x;
    uint32_t wd = wi < W ? words[wi] : 0u;
    const int cnt = __popc(wd);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int any = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      any += wsum[w];
      if (w < warp) incl += wsum[w];
    }
    if (any == 0) {     // (a tile without atoms: nothing to list)
      wb += T;
      if (wb < W) __syncthreads();
      continue;
    }
    // the words that fit form a prefix (incl never decreases); one word
    // always fits (a word holds at most 32 <= LT atoms)
    const bool take = incl <= LT;
    const int pos = incl - cnt;
    if (take)
      for (int p = pos; wd; ++p) {
        list[p] = (wi << 5) + (__ffs(wd) - 1);
        wd &= wd - 1;
      }
    const int ntake = __syncthreads_count(take && wi < W);
    // entries listed: the inclusive count of the last word taken
    int total = 0;
    if (ntake > 0 && (int)threadIdx.x == ntake - 1) wsum[0] = incl;
    __syncthreads();
    total = wsum[0];
    wb += ntake > 0 ? ntake : W;   // ntake = 0 only past the last word
    // pair data of the listed atoms (set up once per pair by the binning
    // launch), up to LM per thread
    for (int e = threadIdx.x; e < total; e += T) prm[e] = __ldg(apairs + list[e]);
    __syncthreads();
    // warp w: slice [w total / NW, (w + 1) total / NW) in list order
    const int s_lo = (warp * total) / NW, s_hi = ((warp + 1) * total) / NW;
#pragma unroll 4
    for (int s2 = s_lo; s2 < s_hi; ++s2) {
      const float4 q = prm[s2];
#pragma unroll
      for (int k = 0; k < CPL; ++k) {
        const float d = (pc[k] - q.x) - q.y;
        const float m = fabsf(q.z) * d * d;
        // (a cell that the atom misses adds zero, which leaves both sums as they
        // are)
        const float E = ex2_approx(fmaf(m, kNegThirtyLog2e, q.w));
        const float v = m <= 1.f ? copysignf(E, q.z) : 0.f;
        if (KAHAN) {
          const float tt = acc[k] + v;
          cmp[k] += (fabsf(acc[k]) >= fabsf(v)) ? ((acc[k] - tt) + v) : ((v - tt) + acc[k]);
          acc[k] = tt;
        } else {
          acc[k] += v;
        }
      }
    }
    __syncthreads();  // list, prm and wsum are reused by the next pass
  }
#pragma unroll
  for (int k = 0; k < CPL; ++k) {
    parts[warp][0][lane + 32 * k] = acc[k];
    parts[warp][1][lane + 32 * k] = cmp[k];
  }
  __syncthreads();
  __shared__ int s_last;
  if (warp == 0) {
    // combine the warps' partial sums in warp order (compensated)
    float l = 0.f;
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
      float s0 = 0.f, c0 = 0.f;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float v = parts[w][h][lane + 32 * k];
          const float tt = s0 + v;
          c0 += (fabsf(s0) >= fabsf(v)) ? ((s0 - tt) + v) : ((v - tt) + s0);
          s0 = tt;
        }
      }
      if (cell[k] < D0) {
        const float v = s0 + c0;
        const size_t gi = (size_t)a * D0 + cell[k];
        float lk = 0.f;
        if (out.R) out.R[gi] = v;
        if (out.epilogue == kEpiL2) {
          const float res = v - out.data[gi];
          if (out.alpha) out.alpha[gi] = res;
          lk = 0.5f * res * res;
        } else if (out.epilogue == kEpiKL) {
          const float fo = out.data[gi];
          const float gg = v + out.bg;
          const float ig = 1.f / gg;
          if (out.alpha) out.alpha[gi] = 1.f - fo * ig;
          if (out.beta) out.beta[gi] = fo * ig * ig;
          lk = kl_term(fo, gg);
        }
        l += lk;
      }
    }
    if (out.loss_part) {
      const double d = warp_sum_d((double)l);
      if (lane == 0) out.loss_part[item] = d;
      if (loss_out && lane == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1) == n_items - 1;
      }
    }
  }  // warp 0
  if (!out.loss_part || !loss_out) return;
  __syncthreads();
  if (!s_last) return;
  // the last block to finish sums the per-tile partials, all its threads
  __threadfence();
  sum_partials_block<NW>(out.loss_part, n_items, loss_out);
}

// The item (angle a, tile t: a ntiles + t) of block b, in launches of a block per
// item: the tiles at the detector's middle first, of every angle, those at its
// ends last.  Atoms sit about the middle, so the blocks that start last are the
// short ones (in angle order, the SMs idled for a third of the launch on 2150
// atoms x 153 angles x 15 tiles: 51.1 us, 41.1 us; pixel-integrated, 128
// x 401 x 8 tiles: 64.8 and 62.5 us).
template <int K>
__device__ __forceinline__ int centre_out(int b, int n_angles, const TileCfg &tc) {
  auto at = [](int k, int n) { return (k & 1) ? n / 2 - (k + 1) / 2 : n / 2 + k / 2; };
  const int rank = tile_div(b, n_angles, tc.inv_angles), a = b - rank * n_angles;
  if constexpr (K == 1) return a * tc.ntiles + at(rank, tc.ntiles);
  const int k0 = tile_div(rank, tc.nt1, tc.inv_nt1), k1 = rank - k0 * tc.nt1;
  return a * tc.ntiles + at(k0, tc.nt0) * tc.nt1 + at(k1, tc.nt1);
}

template <bool KAHAN, int NW, int CPL = 1, int LM = 1>
__global__ void __launch_bounds__(NW * 32)
    gr_project1d_kernel(Atoms at, Geom g, TileCfg tc, const uint32_t *bitmap,
                        int W, ProjOut out, double *loss_out, int *done,
                        const float4 *__restrict__ pairs) {
  project1d_body<KAHAN, NW, CPL, LM>(at, g, tc, bitmap, W, out, loss_out, done, pairs,
                                     centre_out<1>(blockIdx.x, g.n_angles, tc), gridDim.x);
}

// ---- pixel-integrated operator: binning and projection -------------------
template <int K>
__global__ void __launch_bounds__(128) gr_psf_bin_kernel(Atoms at, Geom g, TileCfg tc,
                                                         uint32_t *bitmap, int W, float s) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int a = blockIdx.y;
  if (j >= at.n) return;
  Frame<K> f;
  load_frame<K>(g.frames, a, f);
  Pair<K> p;
  const bool ok = pair_setup<K>(at, j, f, g, p);
  PsfPair<K> q;
  psf_setup<K>(at, j, g, p, ok, s, q);
  if (q.lo[0] > q.hi[0]) return;
  const uint32_t bit = 1u << (j & 31);
  const size_t base = (size_t)a * tc.ntiles;
  const int wj = j >> 5;
  if constexpr (K == 1) {
    for (int t = q.lo[0] / tc.t0; t <= q.hi[0] / tc.t0; ++t)
      atomicOr(bitmap + (base + t) * W + wj, bit);
  } else {
    if (q.lo[1] > q.hi[1]) return;
    for (int tr = q.lo[0] / tc.t0; tr <= q.hi[0] / tc.t0; ++tr)
      for (int tcix = q.lo[1] / tc.t1; tcix <= q.hi[1] / tc.t1; ++tcix)
        atomicOr(bitmap + (base + (size_t)tr * tc.nt1 + tcix) * W + wj, bit);
  }
}

// A block per (angle, tile): its atoms, in index order, go round its NW
// warps.  A warp's lanes look over an atom's cell box clipped to the tile and
// queue the cells it reaches; 32 queued cells at a time, of as many atoms as
// that takes, get their value by the quadrature rule (121 exponentials, what
// bounds it) and go into the warp's own compensated sums in shared memory,
// those of one cell in atom order; a cell then adds the warps' sums in warp order
// (deterministic).  128 atoms x 401 x 64^2: 138 us with a warp per tile of 32 x
// 32 cells, 109 us with four, 15 of 32 lanes at work; with the queue 69 us (issue, 68 %
// of the slots).
struct PsfStage {
  float4 a, b;   // qh0 ql0 qh1 ql1; G00 G01 G11 log2 amplitude
  float4 c;      // sign of I, rr, total mass
  int4 box;      // first and last cell along each axis, clipped to the tile
};
constexpr int kPsfTileWarps = 4;
// 2D: many tiles of few atoms take a warp each (latency: 32 tiles an SM in flight, not 8;
// 1 and 4 warps: 4 atoms x 1500 x 435 cells, 21000 tiles, 31 and 55 us; 64 x 800 x 300, 8000
// tiles, 67 and 75; 256 there 214 and 191, x 1500 x 435 193 and 208; 16 x 400 x 300, 4000
// tiles, 33 and 29).
static int psf_tile_warps(int K, size_t items, int n_atoms) {
  return K == 1 && items >= 6144 && items >= 64 * (size_t)n_atoms ? 1 : kPsfTileWarps;
}
constexpr int kPsfList = 256;  // atoms listed at a time (8 bitmap words)
// 2D: an atom that meets at least this many of a tile's 32 cells takes a lane a cell
// (us, queued and so: 32 atoms x 647 x 811, r = 0.9: 170, 93; 256 x 400 x 300, r = 3: 109,
// 82; 16 there, a third of the atoms so wide: 30.6, 30.4).
constexpr int kPsfWide1 = 20;
static_assert(kTileDim0 <= 32 && kTileDim1 <= 32, "a queued cell's row and column: 5 bits each");

// words a warp's staging and sums take (rows x cols cells)
__host__ __device__ constexpr int psf_warp_words(int cells) { return 2 * cells + 32 * 16; }

template <int K, int NW>
__global__ void __launch_bounds__(NW * 32, 32 / NW)
    gr_psf_project_kernel(Atoms at, Geom g, TileCfg tc, const uint32_t *bitmap, int W,
                          float s, ProjOut out, double *loss_out, int *done) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int list[kPsfList];
  __shared__ float pc0[kTileDim0], pc1[kTileDim1];
  __shared__ float2 s_loss[NW * 32];
  __shared__ uint32_t s_queue[NW][64];
  __shared__ int s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t *queue = s_queue[warp];
  const int item = centre_out<K>(blockIdx.x, g.n_angles, tc), n_items = g.n_angles * tc.ntiles;
  const int cells = tc.t0 * tc.t1;
  float *acc = smem + (size_t)warp * psf_warp_words(cells);
  float *cmp = acc + cells;
  PsfStage *stage = reinterpret_cast<PsfStage *>(cmp + cells);  // (cells: a multiple of 4)
  const int a = tile_div(item, tc.ntiles, tc.inv_ntiles), t = item - a * tc.ntiles;
  const int tr = tile_div(t, tc.nt1, tc.inv_nt1), tcix = t - tr * tc.nt1;
  const int r0 = tr * tc.t0, c0 = tcix * tc.t1;
  const int D0 = g.ax[0].n, D1 = (K == 1) ? 1 : g.ax[1].n;
  for (int e = lane; e < 2 * cells; e += 32) acc[e] = 0.f;
  if (tid < tc.t0) pc0[tid] = (r0 + tid < D0) ? g.ax[0].coords[r0 + tid] : 0.f;
  if constexpr (K == 2)
    if (tid < tc.t1) pc1[tid] = (c0 + tid < D1) ? g.ax[1].coords[c0 + tid] : 0.f;
  const uint32_t *words = bitmap + (size_t)item * W;
  for (int wb = 0; wb < W; wb += 8) {
    // list 8 words' atoms (the first warp), then deal them out
    __syncthreads();
    int total = 0;
    {
      uint32_t wd = lane < 8 && wb + lane < W ? words[wb + lane] : 0u;
      const int cnt = __popc(wd);
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      total = __shfl_sync(0xffffffffu, incl, 31);
      if (warp == 0) {
        int pos = incl - cnt;
        while (wd) {
          list[pos++] = ((wb + lane) << 5) + (__ffs(wd) - 1);
          wd &= wd - 1;
        }
      }
    }
    __syncthreads();
    const int mine = (total - warp + NW - 1) / NW;   // entries warp, warp + 4, ..
    for (int bs = 0; bs < mine; bs += 32) {
      const int nb = min(32, mine - bs);
      if (lane < nb) {
        const int j = list[warp + NW * (bs + lane)];
        Frame<K> f;
        load_frame<K>(g.frames, a, f);
        Pair<K> p;
        const bool ok = pair_setup<K>(at, j, f, g, p);
        PsfPair<K> q;
        psf_setup<K>(at, j, g, p, ok, s, q);
        PsfStage st;
        st.a = make_float4(p.qh[0], p.ql[0], K == 2 ? p.qh[K - 1] : 0.f, K == 2 ? p.ql[K - 1] : 0.f);
        st.b = make_float4(p.G[0], p.G[1], p.G[2], p.l2amp);
        st.c = make_float4(p.sgn, q.rr, q.total, 0.f);
        st.box = make_int4(max(q.lo[0], r0), min(q.hi[0], r0 + tc.t0 - 1),
                           K == 2 ? max(q.lo[K - 1], c0) : 0,
                           K == 2 ? min(q.hi[K - 1], c0 + tc.t1 - 1) : 0);
        stage[lane] = st;
      }
      __syncwarp();
      // the values of the first n queued cells, into the sums
      auto add_cells = [&](int n) {
        const bool on = lane < n;
        const uint32_t it = queue[on ? lane : 0];
        const int slot = it & 31, lr = (it >> 5) & 31, lc = it >> 10;
        const float4 qa = stage[slot].a, qb = stage[slot].b, qc = stage[slot].c;
        Pair<K> p;
        p.G[0] = qb.x;
        p.G[1] = qb.y;
        p.G[2] = qb.z;
        p.l2amp = qb.w;
        PsfPair<K> q;
        q.rr = qc.y;
        float dc[K], base[K], step[K];
        dc[0] = (pc0[lr] - qa.x) - qa.y;
        if constexpr (K == 2) dc[1] = (pc1[lc] - qa.z) - qa.w;
        const int kind = psf_cell_kind<K>(q, dc, s, base, step);
        float v = qc.z;
        if (kind == 2) v = qc.x * psf_quadrature<K>(p, base, step);
        const int ci = lr * tc.t1 + lc;
        const unsigned same = __match_any_sync(0xffffffffu, on ? ci : -1 - lane);
        const int rank = __popc(same & ((1u << lane) - 1u));
        const int ranks = __reduce_max_sync(0xffffffffu, rank);
        for (int k = 0; k <= ranks; ++k) {
          if (on && rank == k) {
            const float s0 = acc[ci];
            const float tt = s0 + v;
            cmp[ci] += (fabsf(s0) >= fabsf(v)) ? ((s0 - tt) + v) : ((v - tt) + s0);
            acc[ci] = tt;
          }
          __syncwarp();
        }
      };
      // 2D: an atom's value at the lane's cell of the tile
      auto direct = [&](int s2, const int4 &box) {
        const int lr = lane;
        if (lr < box.x - r0 || lr > box.y - r0) return;
        const float4 qa = stage[s2].a, qb = stage[s2].b, qc = stage[s2].c;
        Pair<K> p;
        p.G[0] = qb.x;
        p.l2amp = qb.w;
        PsfPair<K> q;
        q.rr = qc.y;
        float dc[K], base[K], step[K];
        dc[0] = (pc0[lr] - qa.x) - qa.y;
        const int kind = psf_cell_kind<K>(q, dc, s, base, step);
        if (kind == 0) return;
        float v = qc.z;
        if (kind == 2) v = qc.x * psf_quadrature<K>(p, base, step);
        const float s0 = acc[lr], tt = s0 + v;
        cmp[lr] += (fabsf(s0) >= fabsf(v)) ? ((s0 - tt) + v) : ((v - tt) + s0);
        acc[lr] = tt;
      };
      int queued = 0;
      for (int s2 = 0; s2 < nb; ++s2) {
        const int4 box = stage[s2].box;
        if (box.x > box.y || box.z > box.w) continue;
        const float4 qa = stage[s2].a;
        PsfPair<K> q;
        q.rr = stage[s2].c.y;
        const int bw = box.w - box.z + 1;
        const int ncell = (box.y - box.x + 1) * bw;
        if constexpr (K == 1) {
          if (ncell >= kPsfWide1) {
            // most of a 2D tile: its cells at once, a lane each, no queue
            direct(s2, box);
            __syncwarp();  // (a queued cell's sum may be another lane's next)
            continue;
          }
        }
        const float inv_bw = 1.f / (float)bw;
        for (int e0 = 0; e0 < ncell; e0 += 32) {
          const int e = e0 + lane;
          const int rr_ = (int)(((float)e + 0.5f) * inv_bw);
          const int lr = box.x - r0 + rr_;
          const int lc = (K == 2) ? (box.z - c0 + (e - rr_ * bw)) : 0;
          bool hit = false;
          if (e < ncell) {
            float dc[K], base[K], step[K];
            dc[0] = (pc0[lr] - qa.x) - qa.y;
            if constexpr (K == 2) dc[1] = (pc1[lc] - qa.z) - qa.w;
            hit = psf_cell_kind<K>(q, dc, s, base, step) != 0;
          }
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          if (hit)
            queue[queued + __popc(m & ((1u << lane) - 1u))] =
                (uint32_t)s2 | (uint32_t)lr << 5 | (uint32_t)lc << 10;
          queued += __popc(m);
          __syncwarp();
          if (queued >= 32) {
            add_cells(32);
            queued -= 32;
            const uint32_t left = queue[32 + lane];
            __syncwarp();
            if (lane < queued) queue[lane] = left;
            __syncwarp();
          }
        }
      }
      if (queued) add_cells(queued);
      __syncwarp();  // the staged atoms are done with
    }
  }
  __syncthreads();
  float lsum = 0.f, lcmp = 0.f;
  for (int e = tid; e < cells; e += NW * 32) {
    const int lr = e / tc.t1, lc = e - lr * tc.t1;
    const int row = r0 + lr, col = c0 + lc;
    if (row >= D0 || col >= D1) continue;
    // the warps' sums in warp order
    float sv = 0.f, cv = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float *aw = smem + (size_t)w * psf_warp_words(cells);
      pair_add(sv, cv, aw[e], aw[cells + e]);
    }
    const float v = sv + cv;
    const size_t gi = ((size_t)a * D0 + row) * D1 + col;
    if (out.R) out.R[gi] = v;
    float l = 0.f;
    if (out.epilogue == kEpiL2) {
      const float res = v - out.data[gi];
      if (out.alpha) out.alpha[gi] = res;
      l = 0.5f * res * res;
    } else if (out.epilogue == kEpiKL) {
      const float fo = out.data[gi];
      const float gg = v + out.bg;
      const float ig = 1.f / gg;
      if (out.alpha) out.alpha[gi] = 1.f - fo * ig;
      if (out.beta) out.beta[gi] = fo * ig * ig;
      l = kl_term(fo, gg);
    }
    const float tt = lsum + l;
    lcmp += (fabsf(lsum) >= fabsf(l)) ? ((lsum - tt) + l) : ((l - tt) + lsum);
    lsum = tt;
  }
  if (!out.loss_part) return;
  s_loss[tid] = make_float2(lsum, lcmp);
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int w = 1; w < NW; ++w)
      pair_add(lsum, lcmp, s_loss[32 * w + lane].x, s_loss[32 * w + lane].y);
    const double d = warp_sum_d((double)lsum + (double)lcmp);
    if (lane == 0) {
      out.loss_part[item] = d;
      if (loss_out) {
        __threadfence();
        s_last = atomicAdd(done, 1) == n_items - 1;
      }
    }
  }
  if (!loss_out) return;
  __syncthreads();
  if (!s_last) return;
  // the last block to finish sums the items' partials in item order
  __threadfence();
  sum_partials_block<NW>(out.loss_part, n_items, loss_out);
}

// Fixed-order FP64 sum of n loss partials over many blocks (one block's FP64
// pipe, at 16 cycles per warp instruction, would take ~0.3 ms for the 640k
// partials of 20000 images): block b sums the contiguous segment
// [b seg, (b + 1) seg), each thread a strided part of it, then a fixed tree;
// the last block to finish reduces the block sums with a fixed tree.
// bsum: gridDim.x doubles (<= kLossMaxBlocks); done: a counter zeroed before
// the launch.
constexpr int kLossThreads = 256;
constexpr int kLossMaxBlocks = 256;
__global__ void __launch_bounds__(kLossThreads)
    gr_loss_finalize_kernel(const double *part, int n, double *out, double *bsum, int *done) {
  __shared__ double sh[kLossThreads];
  __shared__ int s_last;
  const int seg = (n + (int)gridDim.x - 1) / (int)gridDim.x;
  const int lo = blockIdx.x * seg, hi = min(n, lo + seg);
  double s = 0.0;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) s += part[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    bsum[blockIdx.x] = sh[0];
    __threadfence();
    s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  sh[threadIdx.x] = (int)threadIdx.x < (int)gridDim.x ? __ldcg(bsum + threadIdx.x) : 0.0;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = sh[0];
}

static dim3 bin3d_grid(int W, int n_angles, int ntiles) {
  const long long blocks = (long long)((W + 7) / 8) * n_angles;
  const int ranges = (ntiles + kBinTiles - 1) / kBinTiles;
  const long long z = blocks < kBinFewBlocks ? (kBinFewBlocks + blocks - 1) / blocks : 1;
  return dim3((W + 7) / 8, n_angles, (unsigned)(z < ranges ? z : ranges));
}

// Tiling of the point-sampled 3D projection (Tuning::proj_form, key 3):
// 1: 16-row tiles (more resident warps), 2: 32-row tiles (fewer atoms cut
// by tile edges).
static int proj_rows(int form) { return form == 2 ? kTileDim0 : 16; }

// Loss partials of up to this many items are summed by the projection's last
// block (sum_partials_block), more by gr_loss_finalize_kernel (7 us and a launch).
// With a block per item each block has a fence and an atomic to end with, and a
// block's short life pays for them; the persistent 3D blocks do it once.  Fused
// and separate, whole forward (us): 2D, 4 atoms x 510 cells: 3280 items 17.9 and
// 20.6, 6400: 24.7 and 24.0, 16384: 43.0 and 34.8; pixel-integrated 3D: 2550:
// 25.8 and 28.9, 5100: 37.4 and 37.4, 10200: 63.3 and 59.8; 3D, 20 atoms x 70^2:
// 7695: 31.7 and 33.4, 10350: 39.3 and 39.2, 13500: 47.6 and 45.9 (a launch less
// is 2 us less on the host, too).
constexpr size_t kFusedLossItems = 5120, kFusedLossItems3D = 12288;

template <int NW>
static void launch_project3d(size_t items, const Atoms &at, const Geom &g, const TileCfg &tc,
                             const uint32_t *bitmap, int W, const Proj3Rec *rec, const ProjOut &o,
                             int *next_item, double *loss_out, const int *item_list,
                             cudaStream_t stream) {
  // persistent grid: the resident blocks of every SM, at most one per item
  static int resident[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (resident[dev] == 0) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gr_project3d_kernel<NW, true>,
                                                  NW * 32, 0);
    resident[dev] = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  }
  const int grid = (int)(items < (size_t)resident[dev] ? items : (size_t)resident[dev]);
  if (item_list)
    gr_project3d_kernel<NW, true><<<grid, NW * 32, 0, stream>>>(
        at, g, tc, bitmap, W, rec, o, next_item, loss_out, item_list, next_item + 2);
  else
    gr_project3d_kernel<NW, false><<<grid, NW * 32, 0, stream>>>(
        at, g, tc, bitmap, W, rec, o, next_item, loss_out, nullptr, nullptr);
}

// rows: the tile's rows (3D) or cells (2D)
TileCfg make_tiles(int K, int D0, int D1, int rows, int n_angles) {
  TileCfg tc;
  if (K == 1) {
    tc.t0 = rows;
    tc.t1 = 1;
    tc.nt0 = (D0 + tc.t0 - 1) / tc.t0;
    tc.nt1 = 1;
  } else {
    tc.t0 = rows;
    tc.t1 = kTileDim1;
    tc.nt0 = (D0 + tc.t0 - 1) / tc.t0;
    tc.nt1 = (D1 + tc.t1 - 1) / tc.t1;
  }
  tc.ntiles = tc.nt0 * tc.nt1;
  auto inv = [](int d) { return d > 1 ? (uint32_t)((1ull << 32) / (unsigned)d) : 0xffffffffu; };
  tc.inv_ntiles = inv(tc.ntiles);
  tc.inv_nt1 = inv(tc.nt1);
  tc.inv_angles = inv(n_angles);
  return tc;
}

size_t project_skip_items(const Geom &g, int psf, const Tuning &t) {
  if (g.K != 2 || psf) return 0;
  const TileCfg tc = make_tiles(2, g.ax[0].n, g.ax[1].n, proj_rows(t.proj_form));
  return (size_t)g.n_angles * tc.ntiles;
}

// Workspace of a projection without the 3D pair records: the least a launch
// takes.
size_t project_min_bytes(int K, int n_atoms, int n_angles, int D0, int D1, const Tuning &t) {
  // sized for the smaller of the point-sampled and pixel-integrated tilings
  const int rows = K == 1 ? kTile1D
                          : (proj_rows(t.proj_form) < kTileDim0 ? proj_rows(t.proj_form)
                                                                : kTileDim0);
  TileCfg tc = make_tiles(K, D0, D1, rows);
  const size_t W = (size_t)(n_atoms + 31) / 32;
  const size_t items = (size_t)n_angles * tc.ntiles;
  // item counter of the persistent 3D kernel, finished-block counter, count
  // of listed items
  size_t bytes = align_up(4 * sizeof(int));
  // 3D: a flag per item (cleared with the counters) before the bitmap, and
  // the list of items some atom meets (a forward that skips the others)
  bytes += align_up(items * W * sizeof(uint32_t) + (K == 2 ? items * sizeof(uint32_t) : 0));
  bytes += align_up(items * sizeof(double));
  bytes += align_up(kLossMaxBlocks * sizeof(double));  // block sums of the loss finalize
  if (K == 1)  // per-(angle, atom) pair records of the 2D projection
    bytes += align_up((size_t)n_angles * (size_t)n_atoms * sizeof(float4));
  else
    bytes += align_up(items * sizeof(int));
  return bytes;
}

// 3D pair records: setting a pair up again in each of the 1.3 to 2.5 tiles it
// touches took 40 % of the projection (8.4 of 20.9 ms on 8192 atoms x 20000
// orientations), so the binning writes each pair's 32-byte record once.  Problems
// whose records pass kRecBytes run in ranges of angles, each binned and projected in
// turn.  A range must fill the GPU many times over: 8192 atoms x 2000 x 128^2 in
// ranges of 512, 4096, 16384 and 64000 items 7.9, 3.1, 2.25 and 2.01 ms, without
// records 2.18; 20000 x 60 x 64^2 in 15 ranges of 32 items 2.45 ms, without 0.26.  So
// ranges of fewer than kRangeItems are not taken: then no records.
constexpr size_t kRecBytes = (size_t)512 << 20;
constexpr size_t kRangeItems = 32768;

// Angles whose records `bytes` hold and that are taken at a time (0: no records).
static size_t record_range(size_t bytes, int n_atoms, int n_angles, int ntiles) {
  const size_t row = (size_t)n_atoms * sizeof(Proj3Rec), range = row > 0 ? bytes / row : 0;
  if (range >= (size_t)n_angles) return n_angles;
  return range * ntiles >= kRangeItems ? range : 0;
}

size_t project_workspace_bytes(int K, int n_atoms, int n_angles, int D0, int D1,
                               const Tuning &t) {
  size_t bytes = project_min_bytes(K, n_atoms, n_angles, D0, D1, t);
  if (K == 2) {
    const int ntiles = make_tiles(2, D0, D1, proj_rows(t.proj_form)).ntiles;
    bytes += align_up(record_range(kRecBytes, n_atoms, n_angles, ntiles) * n_atoms *
                      sizeof(Proj3Rec));
  }
  return bytes;
}

int launch_project(const Atoms &at, const Geom &g, const ProjOut &o_in,
                   double *loss_out, void *ws, size_t ws_bytes,
                   cudaStream_t stream, const Tuning &t) {
  const int K = g.K;
  const int D0 = g.ax[0].n, D1 = K == 1 ? 1 : g.ax[1].n;
  const int form = t.proj_form;
  // 2D: 64-cell tiles (two cells per lane) for form 2, 128 (four) for form
  // 3, else 32
  const bool wide2d = K == 1 && !o_in.psf && form == 2;
  const bool wide4 = K == 1 && !o_in.psf && form == 3;
  TileCfg tc = make_tiles(K, D0, D1,
                          K == 1 ? (wide4 ? 4 * kTile1D : wide2d ? 2 * kTile1D : kTile1D)
                                 : proj_rows(form),
                          g.n_angles);
  const int W = (at.n + 31) / 32;
  const size_t items = (size_t)g.n_angles * tc.ntiles;
  const size_t need = project_min_bytes(K, at.n, g.n_angles, D0, D1, t);
  // items no atom meets: point-sampled 3D only, fields only
  const int emode = o_in.empty_mode;
  if (emode != kEmptyNone &&
      (K != 2 || o_in.psf || o_in.R || !o_in.empty_loss || emode < 0 || emode > kEmptySkip))
    return kErrArg;
  const bool record = emode == kEmptyRecord;
  if (ws_bytes < need || (ws == nullptr && need > 0)) return kErrWorkspace;
  // (the binning grid's y extent; a forward without atoms has no such limit)
  if (W > 0 && !record && g.n_angles > 65535) return kErrLaunch;
  const bool skip = emode == kEmptySkip;
  const bool point3 = K == 2 && !o_in.psf;
  char *wp = static_cast<char *>(ws);
  int *next_item = reinterpret_cast<int *>(wp);
  wp += align_up(4 * sizeof(int));
  uint32_t *flag = reinterpret_cast<uint32_t *>(wp);  // 3D: one per item
  uint32_t *bitmap = flag + (K == 2 ? items : 0);
  wp += align_up(items * W * sizeof(uint32_t) + (K == 2 ? items * sizeof(uint32_t) : 0));
  double *loss_part = reinterpret_cast<double *>(wp);
  wp += align_up(items * sizeof(double)) + align_up(kLossMaxBlocks * sizeof(double));
  float4 *pairs = K == 1 ? reinterpret_cast<float4 *>(wp) : nullptr;
  int *item_list = K == 2 ? reinterpret_cast<int *>(wp) : nullptr;
  // the 3D binning writes every word of the bitmap and clears the counters;
  // the others want the counters and the bitmap cleared, a skipping forward
  // the counters and the item flags
  size_t clear = align_up(4 * sizeof(int));
  if (!point3) clear += (K == 2 ? items * sizeof(uint32_t) : 0) + items * W * sizeof(uint32_t);
  else if (skip) clear += items * sizeof(uint32_t);
  else if (W > 0 && !record) clear = 0;
  if (clear && cudaMemsetAsync(ws, 0, clear, stream) != cudaSuccess) return kErrLaunch;
  ProjOut o = o_in;
  o.loss_part = loss_out ? loss_part : nullptr;
  // skipping: the items no atom meets take their recorded loss partials
  // (copied first, the listed items' partials overwrite theirs)
  if (skip && o.loss_part &&
      cudaMemcpyAsync(o.loss_part, o_in.empty_loss, items * sizeof(double),
                      cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
    return kErrLaunch;
  if (record) {
    // every item as if no atom met it: its loss partial goes to empty_loss,
    // under the tiling of a forward of these atoms, so it equals bitwise what
    // that forward computes for an empty item
    o.alpha = o.beta = nullptr;
    o.loss_part = o_in.empty_loss;
    loss_out = nullptr;
  }
  // half-width of the (square) cells of the pixel-integrated operator
  const float psf_s = 0.5f / g.ax[0].inv_step;
  if (W > 0 && !point3) {
    dim3 bgrid((at.n + 127) / 128, g.n_angles);
    if (o.psf) {
      if (K == 1) gr_psf_bin_kernel<1><<<bgrid, 128, 0, stream>>>(at, g, tc, bitmap, W, psf_s);
      else gr_psf_bin_kernel<2><<<bgrid, 128, 0, stream>>>(at, g, tc, bitmap, W, psf_s);
    } else {
      gr_bin_kernel<<<bgrid, 128, 0, stream>>>(at, g, tc, bitmap, W, pairs);
    }
    note_launches(1);
  }
  // below the 48 KB that needs no opt-in, so no function attribute is set (safe
  // under capture)
  static_assert(kPsfTileWarps * psf_warp_words(kTileDim0 * kTileDim1) * sizeof(float) <= 42 * 1024,
                "smem");
  bool fused_loss = false;
  if (point3) {
    // records: as many angles at a time as the workspace holds; a skipping
    // forward (one list of items) takes all angles at once or none
    const size_t base = align_up(need);
    Proj3Rec *rec = reinterpret_cast<Proj3Rec *>(static_cast<char *>(ws) + base);
    size_t range = ws_bytes > base ? record_range(ws_bytes - base, at.n, g.n_angles, tc.ntiles) : 0;
    if (range == 0 || record || (skip && range < (size_t)g.n_angles)) {
      rec = nullptr;
      range = g.n_angles;
    }
    const size_t cells = (size_t)D0 * D1;
    fused_loss = loss_out != nullptr && items <= kFusedLossItems3D && range == (size_t)g.n_angles;
    double *lo = fused_loss ? loss_out : nullptr;
    for (size_t a0 = 0; a0 < (size_t)g.n_angles; a0 += range) {
      Geom gr = g;
      gr.n_angles = (int)(g.n_angles - a0 < range ? g.n_angles - a0 : range);
      gr.frames = g.frames + a0 * kFrameStride3D;
      const size_t i0 = a0 * tc.ntiles, ni = (size_t)gr.n_angles * tc.ntiles;
      ProjOut oc = o;
      if (oc.R) oc.R += a0 * cells;
      if (oc.data) oc.data += a0 * cells;
      if (oc.alpha) oc.alpha += a0 * cells;
      if (oc.beta) oc.beta += a0 * cells;
      if (oc.loss_part) oc.loss_part += i0;
      uint32_t *bm = bitmap + i0 * W;
      if (W > 0 && !record) {
        gr_bin3d_kernel<<<bin3d_grid(W, gr.n_angles, tc.ntiles), 256, 0, stream>>>(
            at, gr, tc, bm, W, rec, skip ? nullptr : next_item,
            skip ? flag : nullptr, item_list, next_item + 2);
        note_launches(1);
      }
      const int Wk = record ? 0 : W;  // recording: no atom in any item
      // skipping: only the listed items (none without atoms)
      const int *il = skip ? item_list : nullptr;
      timer_mark(1, 0, stream);
      if (form == 2)
        launch_project3d<8>(ni, at, gr, tc, bm, Wk, rec, oc, next_item, lo, il, stream);
      else
        launch_project3d<4>(ni, at, gr, tc, bm, Wk, rec, oc, next_item, lo, il, stream);
      timer_mark(1, 1, stream);
      note_launches(1);
    }
  } else {
    timer_mark(1, 0, stream);
    if (o.psf) {
      fused_loss = loss_out != nullptr && items <= kFusedLossItems;
      double *lo = fused_loss ? loss_out : nullptr;
      const int nw = psf_tile_warps(K, items, at.n);
      const size_t smem = (size_t)nw * psf_warp_words(tc.t0 * tc.t1) * sizeof(float);
      auto go = [&](auto kernel) {
        kernel<<<(unsigned)items, nw * 32, smem, stream>>>(at, g, tc, bitmap, W, psf_s, o, lo,
                                                           next_item + 1);
      };
      if (K == 2) go(gr_psf_project_kernel<2, kPsfTileWarps>);
      else if (nw == 1) go(gr_psf_project_kernel<1, 1>);
      else go(gr_psf_project_kernel<1, kPsfTileWarps>);
    } else {
      // one block per (angle, tile) item; for up to kFusedLossItems tiles the
      // last block also sums the loss partials (no separate finalize launch)
      fused_loss = loss_out != nullptr && items <= kFusedLossItems;
      double *lo = fused_loss ? loss_out : nullptr;
      if (wide4 && W >= 8)
        gr_project1d_kernel<true, 8, 4, 2><<<(unsigned)items, 8 * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
      else if (wide4)
        gr_project1d_kernel<true, kProjWarps, 4><<<(unsigned)items, kProjWarps * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
      else if (wide2d && W >= 8)
        gr_project1d_kernel<true, 8, 2, 2><<<(unsigned)items, 8 * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
      else if (wide2d)
        gr_project1d_kernel<true, kProjWarps, 2><<<(unsigned)items, kProjWarps * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
      else if (W >= 32)  // 1024 atoms up: four list entries per thread
        gr_project1d_kernel<true, 8, 1, 4><<<(unsigned)items, 8 * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
      else if (W >= 8)  // 8 warps share a tile's atoms from 8 bitmap words (256 atoms) up
        gr_project1d_kernel<true, 8, 1, 2><<<(unsigned)items, 8 * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
      else
        gr_project1d_kernel<true, kProjWarps><<<(unsigned)items, kProjWarps * 32, 0, stream>>>(
            at, g, tc, bitmap, W, o, lo, next_item + 1, pairs);
    }
    timer_mark(1, 1, stream);
    note_launches(1);
  }
  if (loss_out && !fused_loss) {
    // about 8 partials per thread, at most kLossMaxBlocks blocks; the
    // finished-block counter (next_item + 1) is unused when the loss is not
    // fused into the projection
    size_t lb = (items + kLossThreads * 8 - 1) / (kLossThreads * 8);
    lb = lb < 1 ? 1 : (lb > kLossMaxBlocks ? kLossMaxBlocks : lb);
    double *bsum = loss_part + align_up(items * sizeof(double)) / sizeof(double);
    gr_loss_finalize_kernel<<<(unsigned)lb, kLossThreads, 0, stream>>>(loss_part, (int)items,
                                                                        loss_out, bsum,
                                                                        next_item + 1);
    note_launches(1);
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

// ---- multi-problem launches (2D) -------------------------------------------
// Blocks of problems whose fit has stopped return at once (the whole block).
__global__ void __launch_bounds__(128)
    gr_batch_bin_kernel(const BatchProb *__restrict__ probs, const int *__restrict__ off, int n,
                        const int *__restrict__ active, int use_trial) {
  const int p = batch_find(off, n, blockIdx.x);
  if (!active[p]) return;
  const BatchProb &B = probs[p];
  const int lb = blockIdx.x - off[p];
  const int bxn = (B.cur.n + 127) / 128;
  bin_body(use_trial ? B.trial : B.cur, B.g, B.tc, B.bitmap, B.W, B.pairs, lb % bxn,
              lb / bxn);
}

__global__ void __launch_bounds__(kProjWarps * 32)
    gr_batch_project_kernel(const BatchProb *__restrict__ probs, const int *__restrict__ off,
                            int n, const int *__restrict__ active, int use_trial) {
  const int p = batch_find(off, n, blockIdx.x);
  if (!active[p]) return;
  const BatchProb &B = probs[p];
  project1d_body<true, kProjWarps>(use_trial ? B.trial : B.cur, B.g, B.tc, B.bitmap, B.W, B.out,
                                   use_trial ? B.loss_trial : B.loss_cur, B.done, B.pairs,
                                   blockIdx.x - off[p], B.items);
}

int launch_batch_bin(const BatchLaunch &b, int use_trial, cudaStream_t stream) {
  if (b.grid_bin <= 0) return kOk;
  gr_batch_bin_kernel<<<b.grid_bin, 128, 0, stream>>>(b.probs, b.off_bin, b.n, b.active,
                                                      use_trial);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

int launch_batch_project(const BatchLaunch &b, int use_trial, cudaStream_t stream) {
  if (b.grid_proj <= 0) return kOk;
  gr_batch_project_kernel<<<b.grid_proj, kProjWarps * 32, 0, stream>>>(
      b.probs, b.off_proj, b.n, b.active, use_trial);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

int preload_project() {
  return preload_fn(gr_bin_kernel) + preload_fn(gr_bin3d_kernel) +
         preload_fn(gr_psf_bin_kernel<1>) + preload_fn(gr_psf_bin_kernel<2>) +
         preload_fn(gr_project3d_kernel<4, false>) + preload_fn(gr_project3d_kernel<4, true>) +
         preload_fn(gr_project3d_kernel<8, false>) + preload_fn(gr_project3d_kernel<8, true>) +
         preload_fn(gr_project1d_kernel<true, 8, 1, 4>) +
         preload_fn(gr_project1d_kernel<true, 8, 1, 2>) +
         preload_fn(gr_project1d_kernel<true, kProjWarps>) +
         preload_fn(gr_project1d_kernel<true, 8, 2, 2>) +
         preload_fn(gr_project1d_kernel<true, kProjWarps, 2>) +
         preload_fn(gr_project1d_kernel<true, 8, 4, 2>) +
         preload_fn(gr_project1d_kernel<true, kProjWarps, 4>) +
         preload_fn(gr_psf_project_kernel<1, 1>) + preload_fn(gr_psf_project_kernel<1, kPsfTileWarps>) +
         preload_fn(gr_psf_project_kernel<2, kPsfTileWarps>) +
         preload_fn(gr_loss_finalize_kernel) + preload_fn(gr_batch_bin_kernel) +
         preload_fn(gr_batch_project_kernel);
}

}  // namespace gr
