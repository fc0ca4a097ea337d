// Per-step shooting and adjoint sweeps of the 3D Gaussian deformation kernel on 128-row
// tiles: the kernels of every large registration and of uneven batches.
//
// K(q_i, q_j) = 2^-|x_i - x_j|^2 in the scaled coordinates (kernels.cuh).  With both
// points taken relative to the centre c of the row tile, x' = x - c,
//   -|x_i - x_j|^2 = 2 x_i'.x_j' - |x_j'|^2 - |x_i'|^2:
// 3 FMAs per pair instead of 6 operations, |x_j'|^2 is formed once per staged column and
// 2^-|x_i'|^2 is a factor of the row.  The rounding of the expanded form is
// 2^-24 (2 |x_i'| |x_j'| + |x_j'|^2), of the same size as that of the stored FP32
// coordinates as long as |x_i'| is about 1; a tile whose points lie further apart
// (kCompactR2) is evaluated from coordinate differences instead.
//
// Distance test (shooting; the adjoint's: cull.h).  A 32-column block B is skipped for a row tile I when its whole
// contribution is bounded by
//   2^-gap(I, B)^2 S_B  <=  2^-26 / nblk * 2^-diag(I)^2 S_I,
// S the sum of the momenta's absolute values over a block's (the tile's) points, gap the
// distance of the bounding boxes, diag the tile's diagonal, nblk the pair's blocks.  The
// right side is at most 2^-26 / nblk of sum_j K_ij |a_j| of every row of the tile (its
// own tile's points alone give 2^-diag^2 S_I), so all skipped blocks together change a
// row's sum by less than 2^-26 of its sum of absolute values: a quarter of the half-ulp
// that every FP32 term carries.  Zero, tiny or unevenly distributed momenta move the
// cut-off outwards by themselves.  A block with a non-finite point or momentum has a box
// of all of space and S_B = inf: it is never skipped.
#pragma once

#include "cull.h"
#include "griddesc.cuh"
#include "kernels.cuh"
#include "layout.h"
#include "ops.cuh"
#include "persist.cuh"
#include "sweep.cuh"

namespace lddmm {

constexpr int kGaussRows = 128;         // rows per work item (two 64-row tiles)
constexpr float kCompactR2 = 3.0f;      // squared half diagonal of a compact row tile

// Block statistics of one time step (32-point blocks of the concatenated points).
struct GaussStats {
  const float4 *box;  // per block: (lo, -), (hi, -) of the scaled positions
  const float4 *wa;   // per block: (sum |a|, -, -, -) of alpha_t
  const float4 *wu;   // adjoint, per block: (sum |u|, -, -, -)
  // (pairs with a grid have them only in the steps that it cannot hold: grid_conv_yz_kernel)
  float4 *box_n;      // shooting: boxes of the next step's positions (written)
  float4 *wu_n;       // adjoint: weights of the next backward step's u (written; or null)
  // contexts with a grid (grid.cuh): the next positions' box keys [pair][6], max |u| of the
  // next backward step [pair] (or null)
  unsigned *key_n, *umax_n;
};

// Bounding box of a row tile, its centre and diagonal (each warp of a CTA holds all the
// tile's rows, four per lane, and computes the same).
struct GaussTile {
  float lo[3], hi[3], c[3];
  float diag2;       // squared diagonal of the box
  bool compact;
};

__device__ __forceinline__ GaussTile gauss_tile(const float4 (&q)[4], const bool (&live)[4]) {
  GaussTile t;
  bool fin = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    t.lo[d] = INFINITY;
    t.hi[d] = -INFINITY;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float x = d == 0 ? q[r].x : d == 1 ? q[r].y : q[r].z;
      fin &= !live[r] || isfinite(x);
      if (live[r]) {
        t.lo[d] = fminf(t.lo[d], x);
        t.hi[d] = fmaxf(t.hi[d], x);
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      t.lo[d] = fminf(t.lo[d], __shfl_xor_sync(0xffffffffu, t.lo[d], off));
      t.hi[d] = fmaxf(t.hi[d], __shfl_xor_sync(0xffffffffu, t.hi[d], off));
    }
  }
  fin = __all_sync(0xffffffffu, fin);
  t.diag2 = 0.0f;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (!fin) {
      t.lo[d] = -INFINITY;
      t.hi[d] = INFINITY;
    }
    const float e = t.hi[d] - t.lo[d];
    t.diag2 = fmaf(e, e, t.diag2);
    t.c[d] = 0.5f * (t.lo[d] + t.hi[d]);
  }
  t.compact = t.diag2 <= 4.0f * kCompactR2;  // false for an infinite box
  if (!t.compact) t.c[0] = t.c[1] = t.c[2] = 0.0f;
  return t;
}

__device__ __forceinline__ float gauss_gap2(const GaussTile &t, const float4 &lo,
                                            const float4 &hi) {
  const float gx = fmaxf(0.0f, fmaxf(lo.x - t.hi[0], t.lo[0] - hi.x));
  const float gy = fmaxf(0.0f, fmaxf(lo.y - t.hi[1], t.lo[1] - hi.y));
  const float gz = fmaxf(0.0f, fmaxf(lo.z - t.hi[2], t.lo[2] - hi.z));
  return fmaf(gz, gz, fmaf(gy, gy, gx * gx));
}

// ------------------------------------------------------------------- statistics

// Box of one 32-point block, one point per lane (live: not padding), and its part in the
// pair's box (keys).  blk < 0: not a block of the storage order, keys only.
__device__ __forceinline__ void gauss_block_box(float4 *box, int blk, bool live, float x,
                                                float y, float z, unsigned *keys) {
  const bool fin = isfinite(x) && isfinite(y) && isfinite(z);
  const float v[3] = {x, y, z};
  float lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = live ? (fin ? v[d] : -INFINITY) : INFINITY;
    hi[d] = live ? (fin ? v[d] : INFINITY) : -INFINITY;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], off));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], off));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    if (blk >= 0) {
      box[2 * blk] = make_float4(lo[0], lo[1], lo[2], 0.0f);
      box[2 * blk + 1] = make_float4(hi[0], hi[1], hi[2], 0.0f);
    }
    if (keys)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        atomicMin(&keys[d], float_key(lo[d]));
        atomicMin(&keys[3 + d], float_key(-hi[d]));
      }
  }
}

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
__device__ __forceinline__ float abs_sum(const float4 &a) {
  return fabsf(a.x) + fabsf(a.y) + fabsf(a.z);
}
__device__ __forceinline__ float abs_max(const float4 &a) {
  return fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z)));
}
// A NaN or infinity anywhere in the block gives S = inf (fmaxf drops NaNs, sums keep them).
__device__ __forceinline__ float or_inf(float s) { return s < INFINITY ? s : INFINITY; }

// Weights of alpha at every time step (or of u): one warp per (step, block), nblk blocks
// per step; mx (or null): max |a| per (step, pair).
__global__ void gauss_alpha_kernel(const float4 *as, long long nblk_tot, int nblk, float4 *wa,
                                   const int *pt_pair, unsigned *mx, int P) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long b = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
       b < nblk_tot; b += nw) {
    const float4 a = __ldcg(&as[b * 32 + lane]);
    const float s = or_inf(warp_sum_f(abs_sum(a))), m = warp_max_f(abs_max(a));
    if (lane == 0) {
      wa[b] = make_float4(s, 0.0f, 0.0f, 0.0f);
      const int t = (int)(b / nblk), p = pt_pair[(b - (long long)t * nblk) * 32];
      if (mx && p >= 0) atomicMax(&mx[t * P + p], __float_as_uint(s < INFINITY ? m : s));
    }
  }
}

// Boxes of the initial positions: one warp per block.
__global__ void gauss_box_kernel(const float4 *qs, const int *pt_pair, int nblk, float4 *box,
                                 unsigned *keys) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= nblk) return;
  const float4 q = __ldcg(&qs[(size_t)b * 32 + lane]);
  const int p = pt_pair[(size_t)b * 32 + lane], p0 = __shfl_sync(0xffffffffu, p, 0);
  gauss_block_box(box, b, p >= 0, q.x, q.y, q.z, keys && p0 >= 0 ? keys + 6 * p0 : nullptr);
}

// Statistics of the rows a warp has just finalised (one per lane, whose new values the
// lane itself wrote): the boxes of the next positions, the weights of the next u; of
// storage block blk (-1: rows of another order, only the pair's keys and maxima).  g: the
// row's point, any valid one when not live.
template <int D, int ORDER>
__device__ __forceinline__ void gauss_next_stats(const ShootOp<D, ORDER> &op,
                                                 const GaussStats &gs, int p, int blk, int g,
                                                 bool live) {
  const float4 q = op.qs_n[g];
  gauss_block_box(gs.box_n, blk, live, q.x, q.y, q.z, gs.key_n ? gs.key_n + 6 * p : nullptr);
}
template <int D, int ORDER>
__device__ __forceinline__ void gauss_next_stats(const AdjointOp<D, ORDER> &op,
                                                 const GaussStats &gs, int p, int blk, int g,
                                                 bool live) {
  if (!op.us_n) return;
  const float4 u = live ? op.us_n[g] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float s = or_inf(warp_sum_f(abs_sum(u))), m = warp_max_f(abs_max(u));
  if ((threadIdx.x & 31) == 0) {
    if (blk >= 0) gs.wu_n[blk] = make_float4(s, 0.0f, 0.0f, 0.0f);
    if (gs.umax_n) atomicMax(&gs.umax_n[p], __float_as_uint(s < INFINITY ? m : s));
  }
}

template <int D, char CT, char DT>
__device__ __forceinline__ void gauss_next_stats(const VarifoldOp<D, CT, DT> &,
                                                 const GaussStats &, int, int, int, bool) {}

// ------------------------------------------------------------------- split items
//
// The columns of an item are dealt to S independent CTAs (not a cluster: clusters are
// placed only where S slots of one GPC are free at once, which left SMs idle).  Every
// CTA leaves its FP64 row sums in a slot; the one that completes the item's arrival count
// adds them in rank order and finalises the rows, so results do not depend on the order
// of arrival.

struct SplitPlan {
  int S;               // CTAs per item
  int items;           // work items: items * S units, walked by the grid
  bool one;            // all of one pair
  double *part;        // [item * S + rank][row of the item][NA]
  unsigned int *cnt;   // per item: arrivals (left at zero)
};

// v: the warp's sums of rows 32 r + lane of the item (R * 32 rows; R = 4: the upper half
// only when `two`).
template <class Op, int W, int R>
__device__ __forceinline__ void finish_split(const Op &op, int p, int tile, int item, int rank,
                                             const SplitPlan &sp, bool two,
                                             const GaussStats &gs,
                                             const double (&v)[R][Op::NA]) {
  constexpr int NA = Op::NA, ROWS = R * 32;
  static_assert(ROWS <= W * 32, "one thread per row");
  __shared__ double s_red[W][32][NA];
  __shared__ double s_scr[W];
  __shared__ int s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double t[NA];
#pragma unroll
  for (int r = 0; r < R; ++r) {  // 32 rows at a time: warp r keeps the sums of its rows
    if (r) __syncthreads();
#pragma unroll
    for (int a = 0; a < NA; ++a) s_red[warp][lane][a] = v[r][a];
    __syncthreads();
    if (warp == r) {
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) x += s_red[w][lane][a];
        t[a] = x;
      }
    }
  }
  const bool mine = tid < ROWS && (tid < kTile || two);
  if (sp.S > 1) {
    double *slot = sp.part + (size_t)item * sp.S * ROWS * NA;
    if (mine)
#pragma unroll
      for (int a = 0; a < NA; ++a) __stcg(&slot[((size_t)rank * NA + a) * ROWS + tid], t[a]);
    __syncthreads();
    if (tid == 0) {
      // release: this CTA's part is visible with the count; acquire: the last arriver
      // sees every other part
      s_last = atom_add_acq_rel_gpu(&sp.cnt[item], 1u) == (unsigned int)sp.S - 1u;
      if (s_last) sp.cnt[item] = 0u;
    }
    __syncthreads();
    if (!s_last) return;
    if (mine) {
#pragma unroll
      for (int a = 0; a < NA; ++a) t[a] = 0.0;
#pragma unroll 4
      for (int k = 0; k < sp.S; ++k)
#pragma unroll
        for (int a = 0; a < NA; ++a) t[a] += __ldcg(&slot[((size_t)k * NA + a) * ROWS + tid]);
    }
  }
  double e = 0.0;
  const int row = tile * kTile + tid;
  if (mine) e = op.finalize(p, row, t);
  if (mine) {  // whole warps: the statistics of this warp's block for the next step
    const PairDesc &P = op.pd[p];
    gauss_next_stats(op, gs, p, (P.pt_off + row) / kSub, P.pt_off + row, row < P.N);
  }
  if (Op::kTileSum) {
    for (int h = 0; h < (two ? 2 : 1); ++h) {
      const double tot = block_sum(tid / kTile == h ? e : 0.0, s_scr);
      if (tid == 0) op.write_tile(p, tile + h, tot);
    }
  }
}

// -------------------------------------------------------------------- shooting
//
// Bound: one ex2 per pair on the MUFU pipe (16 per SM and clock; 4 lanes per sub-core, so
// 8 issue slots per warp instruction); the 6 packed FP32x2 instructions of two pairs take
// 12 of the 16 clocks.  A lane holds 4 rows, two columns go into one packed instruction
// (the row's value twice, in registers), so that columns are staged once and not
// duplicated: 7 shared-memory loads of 16 bytes serve 16 pairs of a lane.

template <int W>
__global__ void __launch_bounds__(W * 32, 4)
    gauss_shoot_kernel(const ShootOp<3, -1> op, const GaussStats gs,
                       const int2 *__restrict__ items, const SplitPlan sp, const GridArgs ga) {
  constexpr int NA = 3;
  __shared__ __align__(16) float s_j[W][7][kSub];
  pdl_wait();
  pdl_trigger();
  int skip = -1;  // pair found to have nothing to do here
  for (int unit = blockIdx.x; unit < sp.items * sp.S; unit += gridDim.x) {
    const int S = sp.S;
    const int item = unit / S;
    const int rank = unit - item * S;
    const int2 it = items[item];
    const int p = it.x, tile = it.y;
    if (p == skip) continue;
    GridDesc gd;
    if (!op.active(p) || grid_active(ga, p, false, gd)) {
      if (sp.one) return;
      skip = p;
      continue;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const PairDesc &P = op.pd[p];
    const int pt = P.pt_off, npad = P.Npad;
    const int row0 = tile * kTile;
    const bool two = row0 + kTile < npad;  // uniform over the cluster
    const int blk0 = pt / kSub, nblk = npad / kSub;
    float4 q[4];
    bool live[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = (r < 2 || two) ? row0 + 32 * r + lane : row0 + lane;
      live[r] = row < P.N;
      q[r] = __ldcg(&op.qs_t[pt + row]);
    }
    const GaussTile T = gauss_tile(q, live);
    float S_I = 0.0f;
    for (int b = 0; b < (two ? 4 : 2); ++b) S_I += __ldcg(&gs.wa[blk0 + row0 / kSub + b].x);
    const float thr = T.diag2 - lg2_finite(S_I) + kCullBits + lg2f_approx((float)nblk);
    float2 q2[4][3];  // compact: (2 x', 2 x'); else (x, x)
    double b2[4];     // |x'|^2
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float x = q[r].x - T.c[0], y = q[r].y - T.c[1], z = q[r].z - T.c[2];
      b2[r] = (double)x * x + (double)y * y + (double)z * z;
      const float f = T.compact ? 2.0f : 1.0f;
      q2[r][0] = make_float2(f * x, f * x);
      q2[r][1] = make_float2(f * y, f * y);
      q2[r][2] = make_float2(f * z, f * z);
    }
    float hi[4][NA], lo[4][NA];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int a = 0; a < NA; ++a) hi[r][a] = lo[r][a] = 0.0f;

    const int nw = S * W, gw = rank * W + warp;
    int base = gw - 32 * nw;
    unsigned mask = 0u;
    auto next = [&]() {  // warp-uniform: the next block to evaluate, or nblk
      while (mask == 0u) {
        base += 32 * nw;
        if (base >= nblk) return nblk;
        const int sb = base + lane * nw;
        bool keep = sb < nblk;
        if (keep) {
          const float4 l = __ldcg(&gs.box[2 * (blk0 + sb)]);
          const float4 h = __ldcg(&gs.box[2 * (blk0 + sb) + 1]);
          const float w = __ldcg(&gs.wa[blk0 + sb].x);
          keep = !(gauss_gap2(T, l, h) >= lg2f_approx(w) + thr);
        }
        mask = __ballot_sync(0xffffffffu, keep);
      }
      const int k = __ffs(mask) - 1;
      mask &= mask - 1u;
      return base + k * nw;
    };
    float4 nq, na;
    auto fetch = [&](int s) {
      nq = __ldcg(&op.qs_t[pt + s * kSub + lane]);
      na = __ldcg(&op.as_t[pt + s * kSub + lane]);
    };
    float(*sj)[kSub] = s_j[warp];
    int s = next();
    if (s < nblk) fetch(s);
    while (s < nblk) {
      __syncwarp();
      {
        float x = nq.x - T.c[0], y = nq.y - T.c[1], z = nq.z - T.c[2];
        const float r2 = fmaf(z, z, fmaf(y, y, x * x));
        // a point at infinity: K = 2^-inf in the expanded exponent too, not inf - inf
        if (T.compact && r2 == INFINITY) x = y = z = 0.0f;
        sj[0][lane] = x;
        sj[1][lane] = y;
        sj[2][lane] = z;
        sj[3][lane] = -r2;
        sj[4][lane] = na.x;
        sj[5][lane] = na.y;
        sj[6][lane] = na.z;
      }
      __syncwarp();
      s = next();
      if (s < nblk) fetch(s);
      float2 acc[4][NA];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int a = 0; a < NA; ++a) acc[r][a] = make_float2(0.0f, 0.0f);
      if (T.compact) {
#pragma unroll 2
        for (int jj = 0; jj < kSub; jj += 4) {
          float4 v[7];
#pragma unroll
          for (int k = 0; k < 7; ++k) v[k] = *reinterpret_cast<const float4 *>(&sj[k][jj]);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float2 w[7];
#pragma unroll
            for (int k = 0; k < 7; ++k)
              w[k] = h ? make_float2(v[k].z, v[k].w) : make_float2(v[k].x, v[k].y);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              float2 e = __ffma2_rn(q2[r][0], w[0], w[3]);
              e = __ffma2_rn(q2[r][1], w[1], e);
              e = __ffma2_rn(q2[r][2], w[2], e);
              const float2 K = make_float2(ex2f(e.x), ex2f(e.y));
#pragma unroll
              for (int a = 0; a < NA; ++a) acc[r][a] = __ffma2_rn(K, w[4 + a], acc[r][a]);
            }
          }
        }
      } else {
#pragma unroll 2
        for (int jj = 0; jj < kSub; jj += 2) {
          float2 w[7];
#pragma unroll
          for (int k = 0; k < 7; ++k) w[k] = *reinterpret_cast<const float2 *>(&sj[k][jj]);
          const float2 m1 = make_float2(-1.0f, -1.0f);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float2 dx = __ffma2_rn(w[0], m1, q2[r][0]), dy = __ffma2_rn(w[1], m1, q2[r][1]),
                         dz = __ffma2_rn(w[2], m1, q2[r][2]);
            float2 r2 = __fmul2_rn(dx, dx);
            r2 = __ffma2_rn(dy, dy, r2);
            r2 = __ffma2_rn(dz, dz, r2);
            const float2 K = make_float2(ex2f(-r2.x), ex2f(-r2.y));
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[r][a] = __ffma2_rn(K, w[4 + a], acc[r][a]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int a = 0; a < NA; ++a) two_sum_acc(hi[r][a], lo[r][a], acc[r][a].x + acc[r][a].y);
    }
    double v[4][NA];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const double f = T.compact ? exp2(-b2[r]) : 1.0;
#pragma unroll
      for (int a = 0; a < NA; ++a) v[r][a] = f * ((double)hi[r][a] + (double)lo[r][a]);
    }
    __syncthreads();  // the previous unit's reduction is done with the shared arrays
    finish_split<ShootOp<3, -1>, W, 4>(op, p, tile, item, rank, sp, two, gs, v);
  }
}

// --------------------------------------------------------------------- adjoint
//
// u = a - p, r = a, so with m = u - r = -p the pair weight is
//   l_i.r_j + l_j.r_i = m_i.r_j + r_i.u_j
// and the column operands are x', u and r alone.  With s_ij = K_ij (m_i.r_j + r_i.u_j),
//   sum_j K u_j,   sum_j s_ij (x_i - x_j) = x_i' sum_j s_ij - sum_j s_ij x_j':
// 17 packed instructions per two pairs.

template <int W>
__global__ void __launch_bounds__(W * 32)
    gauss_adjoint_kernel(const AdjointOp<3, -1> op, const GaussStats gs,
                         const int2 *__restrict__ items, const SplitPlan sp, const GridArgs ga) {
  using Op = AdjointOp<3, -1>;
  constexpr int R = 4;    // rows per lane
  constexpr int NS = 7;   // sums per row: K u (3), s x' (3), s
  constexpr int NJ = 10;  // staged values per column: x', -|x'|^2, u, r
  __shared__ __align__(16) float s_j[W][NJ][kSub];
  pdl_wait();
  pdl_trigger();
  int skip = -1;  // as in the shooting sweep
  for (int unit = blockIdx.x; unit < sp.items * sp.S; unit += gridDim.x) {
    const int S = sp.S;
    const int item = unit / S;
    const int rank = unit - item * S;
    const int2 it = items[item];
    const int p = it.x, tile = it.y;
    if (p == skip) continue;
    GridDesc gd;
    if (!op.active(p) || grid_active(ga, p, true, gd)) {
      if (sp.one) return;
      skip = p;
      continue;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const PairDesc &P = op.pd[p];
    const int pt = P.pt_off, npad = P.Npad;
    const int row0 = tile * kTile;
    const bool two = row0 + kTile < npad;
    const int nbt = two ? 4 : 2;
    const int blk0 = pt / kSub, nblk = npad / kSub;
    float4 q[R];
    bool live[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = (r < 2 || two) ? row0 + 32 * r + lane : row0 + lane;
      live[r] = row < P.N;
      q[r] = __ldcg(&op.qs_t[pt + row]);
    }
    const GaussTile T = gauss_tile(q, live);
    float U_I = 0.0f, R_I = 0.0f;
    for (int b = 0; b < nbt; ++b) {
      U_I += __ldcg(&gs.wu[blk0 + row0 / kSub + b].x);
      R_I += __ldcg(&gs.wa[blk0 + row0 / kSub + b].x);
    }
    const AdjointCut cut = adjoint_cut(T.diag2, nblk, U_I, R_I);
    float2 q2[R][3], mi[R][3], ri[R][3];
    const float qf = T.compact ? 2.0f : 1.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = pt + ((r < 2 || two) ? row0 + 32 * r + lane : row0 + lane);
      const float4 u = __ldcg(&op.us_t[row]), a = __ldcg(&op.as_t[row]);
      const float x[3] = {qf * (q[r].x - T.c[0]), qf * (q[r].y - T.c[1]), qf * (q[r].z - T.c[2])};
      const float m[3] = {u.x - a.x, u.y - a.y, u.z - a.z}, rr[3] = {a.x, a.y, a.z};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        q2[r][d] = make_float2(x[d], x[d]);
        mi[r][d] = make_float2(m[d], m[d]);
        ri[r][d] = make_float2(rr[d], rr[d]);
      }
    }
    float hi[R][NS], lo[R][NS];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int a = 0; a < NS; ++a) hi[r][a] = lo[r][a] = 0.0f;
    const int nw = S * W, gw = rank * W + warp;
    int base = gw - 32 * nw;
    unsigned mask = 0u;
    auto next = [&]() {
      while (mask == 0u) {
        base += 32 * nw;
        if (base >= nblk) return nblk;
        const int sb = base + lane * nw;
        bool keep = sb < nblk;
        if (keep) {
          const int b = blk0 + sb;
          const float4 l = __ldcg(&gs.box[2 * b]), h = __ldcg(&gs.box[2 * b + 1]);
          keep = !adjoint_skips(cut, gauss_gap2(T, l, h), __ldcg(&gs.wu[b].x),
                                __ldcg(&gs.wa[b].x));
        }
        mask = __ballot_sync(0xffffffffu, keep);
      }
      const int k = __ffs(mask) - 1;
      mask &= mask - 1u;
      return base + k * nw;
    };
    float4 nq, nu, na;
    auto fetch = [&](int s) {
      nq = __ldcg(&op.qs_t[pt + s * kSub + lane]);
      nu = __ldcg(&op.us_t[pt + s * kSub + lane]);
      na = __ldcg(&op.as_t[pt + s * kSub + lane]);
    };
    float(*sj)[kSub] = s_j[warp];
    int s = next();
    if (s < nblk) fetch(s);
    while (s < nblk) {
      __syncwarp();
      {
        const float x = nq.x - T.c[0], y = nq.y - T.c[1], z = nq.z - T.c[2];
        const float v[NJ] = {x,    y,    z,    -fmaf(z, z, fmaf(y, y, x * x)), nu.x, nu.y,
                             nu.z, na.x, na.y, na.z};
#pragma unroll
        for (int k = 0; k < NJ; ++k) sj[k][lane] = v[k];
      }
      __syncwarp();
      s = next();
      if (s < nblk) fetch(s);
      float2 acc[R][NS];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int a = 0; a < NS; ++a) acc[r][a] = make_float2(0.0f, 0.0f);
      auto rest = [&](int r, const float2 (&w)[NJ], const float2 &K, const float2 (&x)[3]) {
        float2 lr = __fmul2_rn(mi[r][0], w[7]);
#pragma unroll
        for (int d = 1; d < 3; ++d) lr = __ffma2_rn(mi[r][d], w[7 + d], lr);
#pragma unroll
        for (int d = 0; d < 3; ++d) lr = __ffma2_rn(ri[r][d], w[4 + d], lr);
        lr = __fmul2_rn(lr, K);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          acc[r][d] = __ffma2_rn(K, w[4 + d], acc[r][d]);
          acc[r][3 + d] = __ffma2_rn(lr, x[d], acc[r][3 + d]);
        }
        acc[r][6] = __fadd2_rn(acc[r][6], lr);
      };
      if (T.compact) {
#pragma unroll 2
        for (int jj = 0; jj < kSub; jj += 4) {
          float4 v[NJ];
#pragma unroll
          for (int k = 0; k < NJ; ++k) v[k] = *reinterpret_cast<const float4 *>(&sj[k][jj]);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float2 w[NJ];
#pragma unroll
            for (int k = 0; k < NJ; ++k)
              w[k] = h ? make_float2(v[k].z, v[k].w) : make_float2(v[k].x, v[k].y);
            const float2 x[3] = {w[0], w[1], w[2]};
#pragma unroll
            for (int r = 0; r < R; ++r) {
              float2 e = __ffma2_rn(q2[r][0], w[0], w[3]);
              e = __ffma2_rn(q2[r][1], w[1], e);
              e = __ffma2_rn(q2[r][2], w[2], e);
              rest(r, w, make_float2(ex2f(e.x), ex2f(e.y)), x);
            }
          }
        }
      } else {
#pragma unroll 2
        for (int jj = 0; jj < kSub; jj += 2) {
          float2 w[NJ];
#pragma unroll
          for (int k = 0; k < NJ; ++k) w[k] = *reinterpret_cast<const float2 *>(&sj[k][jj]);
          const float2 m1 = make_float2(-1.0f, -1.0f);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            float2 x[3];  // x_j - x_i: the s x' sums are then the negated result
#pragma unroll
            for (int d = 0; d < 3; ++d) x[d] = __ffma2_rn(q2[r][d], m1, w[d]);
            float2 r2 = __fmul2_rn(x[0], x[0]);
            r2 = __ffma2_rn(x[1], x[1], r2);
            r2 = __ffma2_rn(x[2], x[2], r2);
            rest(r, w, make_float2(ex2f(-r2.x), ex2f(-r2.y)), x);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int a = 0; a < NS; ++a) two_sum_acc(hi[r][a], lo[r][a], acc[r][a].x + acc[r][a].y);
    }
    double v[R][6];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double f = 1.0, x[3] = {0.0, 0.0, 0.0};
      if (T.compact) {
#pragma unroll
        for (int d = 0; d < 3; ++d) x[d] = 0.5 * (double)q2[r][d].x;
        f = exp2(-(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]));
      }
      const double ss = (double)hi[r][6] + (double)lo[r][6];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        v[r][d] = f * ((double)hi[r][d] + (double)lo[r][d]);
        v[r][3 + d] = f * (x[d] * ss - ((double)hi[r][3 + d] + (double)lo[r][3 + d]));
      }
    }
    __syncthreads();
    finish_split<Op, W, R>(op, p, tile, item, rank, sp, two, gs, v);
  }
}

}  // namespace lddmm
