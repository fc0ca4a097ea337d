// Varifold sweep of 3D surfaces with the Gaussian centre kernel and the Binet direction
// kernel (every configured surface pair), in the manner of the Gaussian pair sweeps
// (gauss.cuh): centres relative to the row tile's centre, columns packed in pairs,
// distance test, items split over independent CTAs.
//
// With x' a scaled centre minus the tile's centre, k = 2^-|x_i - x_j|^2 =
// 2^(2 x_i'.x_j' - |x_j'|^2 - 1) 2^(1 - |x_i'|^2), and the sums of VarifoldOp (ops.cuh) are
//   S = sum k w ang^2,  A = sum k w ang n_j,
//   C = sum k w ang^2 (x_i - x_j) = x_i' (S_DD + S_DT) - sum k w ang^2 x_j':
// 16 packed instructions per two pairs instead of 25, 8 staged values per column instead
// of 10 doubled ones.  x' is formed from the double-single centres, (hi - c) + lo, and is
// rounded at 2^-24 of the tile's size, not of the coordinates': neighbour distances keep
// the accuracy that the small differences of the deformed and target sums need (a tile of
// 64 neighbouring elements is some 8 neighbour distances wide at any mesh size).  The
// rounding of the expanded exponent grows with the square of the tile's size, so tiles
// wider than kVfdCompactR2 are evaluated from differences of x' (19 instructions), those
// wider than kVfdNearR2 (elements in no spatial order) from the double-single differences
// (25).
//
// Systematic errors.  The value V = DD - 2 DT + TT keeps a common relative error of DD and
// DT whole, since TT is formed in FP64, and near convergence V is small against TT.  ex2.approx
// is low by 5.0e-8 on average over [-1, 0) and high by 3.3e-8 over [0, 1) (measured on 2^20
// arguments, the same in every unit interval; exact at 0).  The compact tiles' arguments are
// therefore kept negative by a factor 2^-1 that the row undoes, and the FP64 sums are raised by
// the error that is left, the mean of ex2's over the kernel's pairs on a surface: 4.6e-8 there,
// 3.7e-8 for arguments -r^2 (the error is smaller near r = 0).  The centre scale is not rounded
// to FP32: its 2.5e-8 widened the kernel and had hidden part of this.  |V - V64| / TT of 20,000
// landmarks, centre width 0.2: 1.4e-8 with neither (0.9e-8 with double-single differences
// throughout), 0.12e-8 now.
//
// A block is skipped when 2^-gap^2 times its area is at most 2^-32 / nblk of 2^-diag^2
// times the tile's own area (all skipped blocks: 2^-32 of what the tile's own elements
// contribute without their direction factors).
#pragma once

#include "gauss.cuh"
#include "ops.cuh"

namespace lddmm {

constexpr float kVfdCompactR2 = 1.0f;  // squared half diagonal of a compact row tile
constexpr float kVfdNearR2 = 16.0f;    // of one evaluated from centred differences
constexpr float kVfdCullBits = 32.0f;
constexpr double kEx2Low = 4.6e-8;     // ex2's mean error, compact tiles (see above)
constexpr double kEx2LowR2 = 3.7e-8;   // the others

template <int W>
__global__ void __launch_bounds__(W * 32, 4)
    vfd_split_kernel(const VarifoldOp<3, 'G', 'B'> op, const int2 *__restrict__ items,
                     const SplitPlan sp) {
  using Op = VarifoldOp<3, 'G', 'B'>;
  constexpr int R = 2, NS = 8;  // S_DD, S_DT, A, sum tb x'
  constexpr int NJ = 11;        // x', -|x'|^2 - 1, n, w; wide tiles: centre hi, lo
  __shared__ __align__(16) float s_j[W][NJ][kSub];
  const int S = sp.S;
  const int item = blockIdx.x / S;
  const int rank = blockIdx.x - item * S;
  const int2 it = items[item];
  pdl_wait();
  pdl_trigger();
  const int p = it.x, tile = it.y;
  if (!op.active(p)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const PairDesc &P = op.pd[p];
  const int ndb = P.Edpad / 32, nblk = ndb + P.Etpad / 32;
  const float4 *db = op.dbb + 2 * (P.el_off / 32), *tb = op.tbb + 2 * (P.tg_off / 32);
  float lo3[3], hi3[3], c[3], diag2 = 0.0f, area;
  {
    const float4 l0 = __ldcg(&db[4 * tile]), h0 = __ldcg(&db[4 * tile + 1]),
                 l1 = __ldcg(&db[4 * tile + 2]), h1 = __ldcg(&db[4 * tile + 3]);
    lo3[0] = fminf(l0.x, l1.x); lo3[1] = fminf(l0.y, l1.y); lo3[2] = fminf(l0.z, l1.z);
    hi3[0] = fmaxf(h0.x, h1.x); hi3[1] = fmaxf(h0.y, h1.y); hi3[2] = fmaxf(h0.z, h1.z);
    area = l0.w + l1.w;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float e = hi3[d] - lo3[d];
    diag2 = fmaf(e, e, diag2);
    c[d] = 0.5f * (lo3[d] + hi3[d]);
  }
  const bool compact = diag2 <= 4.0f * kVfdCompactR2;  // false for an infinite box
  const bool near = diag2 <= 4.0f * kVfdNearR2;
  const float thr = diag2 - lg2_finite(area) + kVfdCullBits + lg2f_approx((float)nblk);
  // 2 x' (compact), -x' (near) or -hi and -lo; n
  float2 q2[R][3], ql[R][3], ni[R][3];
  double xi[R][3];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = P.el_off + tile * kTile + 32 * r + lane;
    const float4 h = __ldcg(&op.ec[row]), l = __ldcg(&op.el[row]), n = __ldcg(&op.en[row]);
    const float hh[3] = {h.x, h.y, h.z}, ll[3] = {l.x, l.y, l.z}, nn[3] = {n.x, n.y, n.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float x = (hh[d] - c[d]) + ll[d];
      xi[r][d] = x;
      const float q = compact ? 2.0f * x : near ? -x : -hh[d];
      q2[r][d] = make_float2(q, q);
      ql[r][d] = make_float2(-ll[d], -ll[d]);
      ni[r][d] = make_float2(nn[d], nn[d]);
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
  auto next = [&]() {  // warp-uniform: the next block to evaluate, or nblk
    while (mask == 0u) {
      base += 32 * nw;
      if (base >= nblk) return nblk;
      const int sb = base + lane * nw;
      bool keep = false;
      if (sb < nblk) {
        const float4 *b = sb < ndb ? db + 2 * sb : tb + 2 * (sb - ndb);
        const float4 l = __ldcg(&b[0]), h = __ldcg(&b[1]);
        const float gx = fmaxf(0.0f, fmaxf(l.x - hi3[0], lo3[0] - h.x));
        const float gy = fmaxf(0.0f, fmaxf(l.y - hi3[1], lo3[1] - h.y));
        const float gz = fmaxf(0.0f, fmaxf(l.z - hi3[2], lo3[2] - h.z));
        keep = !(fmaf(gz, gz, fmaf(gy, gy, gx * gx)) >= lg2f_approx(l.w) + thr);
      }
      mask = __ballot_sync(0xffffffffu, keep);
    }
    const int k = __ffs(mask) - 1;
    mask &= mask - 1u;
    return base + k * nw;
  };
  float4 nc, nl, nn;
  auto fetch = [&](int s) {
    const bool d = s < ndb;
    const int j = d ? P.el_off + s * kSub + lane : P.tg_off + (s - ndb) * kSub + lane;
    nc = __ldcg(&(d ? op.ec : op.tc)[j]);
    nn = __ldcg(&(d ? op.en : op.tn)[j]);
    nl = __ldcg(&(d ? op.el : op.tl)[j]);
  };
  float(*sj)[kSub] = s_j[warp];
  int s = next();
  if (s < nblk) fetch(s);
  while (s < nblk) {
    const bool dset = s < ndb;
    __syncwarp();
    {
      const float x = (nc.x - c[0]) + nl.x, y = (nc.y - c[1]) + nl.y, z = (nc.z - c[2]) + nl.z;
      sj[3][lane] = -1.0f - fmaf(z, z, fmaf(y, y, x * x));
      sj[4][lane] = nn.x;
      sj[5][lane] = nn.y;
      sj[6][lane] = nn.z;
      sj[7][lane] = nc.w;
      if (near) {
        sj[0][lane] = x;
        sj[1][lane] = y;
        sj[2][lane] = z;
      } else {
        sj[0][lane] = nc.x;
        sj[1][lane] = nc.y;
        sj[2][lane] = nc.z;
        sj[8][lane] = nl.x;
        sj[9][lane] = nl.y;
        sj[10][lane] = nl.z;
      }
    }
    __syncwarp();
    s = next();
    if (s < nblk) fetch(s);
    float2 acc[R][7];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int a = 0; a < 7; ++a) acc[r][a] = make_float2(0.0f, 0.0f);
    // one pair of columns against row r: exponent e, x the operand of the C sums
    auto pair = [&](int r, const float2 &e, const float2 *n, const float2 &wt, const float2 *x) {
      float2 ang = __fmul2_rn(ni[r][0], n[0]);
      ang = __ffma2_rn(ni[r][1], n[1], ang);
      ang = __ffma2_rn(ni[r][2], n[2], ang);
      const float2 t1 = __fmul2_rn(__fmul2_rn(make_float2(ex2f(e.x), ex2f(e.y)), wt), ang);
      const float2 tb2 = __fmul2_rn(t1, ang);
      acc[r][0] = __fadd2_rn(acc[r][0], tb2);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        acc[r][1 + d] = __ffma2_rn(t1, n[d], acc[r][1 + d]);
        acc[r][4 + d] = __ffma2_rn(tb2, x[d], acc[r][4 + d]);
      }
    };
    // four columns at a time, two per packed instruction
    auto four = [&](int jj, auto &&one) {
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = *reinterpret_cast<const float4 *>(&sj[k][jj]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          w[k] = h ? make_float2(v[k].z, v[k].w) : make_float2(v[k].x, v[k].y);
#pragma unroll
        for (int r = 0; r < R; ++r) one(r, w);
      }
    };
    if (compact) {
#pragma unroll 2
      for (int jj = 0; jj < kSub; jj += 4)
        four(jj, [&](int r, const float2 *w) {
          float2 e = __ffma2_rn(q2[r][0], w[0], w[3]);
          e = __ffma2_rn(q2[r][1], w[1], e);
          e = __ffma2_rn(q2[r][2], w[2], e);
          pair(r, e, w + 4, w[7], w);
        });
    } else if (near) {
#pragma unroll 2
      for (int jj = 0; jj < kSub; jj += 4)
        four(jj, [&](int r, const float2 *w) {
          float2 x[3];  // x_j' - x_i': the C sums are then the negated result
#pragma unroll
          for (int d = 0; d < 3; ++d) x[d] = __fadd2_rn(q2[r][d], w[d]);
          float2 e = __fmul2_rn(x[0], x[0]);
          e = __ffma2_rn(x[1], x[1], e);
          e = __ffma2_rn(x[2], x[2], e);
          pair(r, make_float2(-e.x, -e.y), w + 4, w[7], x);
        });
    } else {
#pragma unroll 2
      for (int jj = 0; jj < kSub; jj += 2) {
        float2 w[NJ];
#pragma unroll
        for (int k = 0; k < NJ; ++k) w[k] = *reinterpret_cast<const float2 *>(&sj[k][jj]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float2 x[3];  // x_j - x_i, from the negated hi and lo of the row
#pragma unroll
          for (int d = 0; d < 3; ++d)
            x[d] = __fadd2_rn(__fadd2_rn(q2[r][d], w[d]), __fadd2_rn(ql[r][d], w[8 + d]));
          float2 e = __fmul2_rn(x[0], x[0]);
          e = __ffma2_rn(x[1], x[1], e);
          e = __ffma2_rn(x[2], x[2], e);
          pair(r, make_float2(-e.x, -e.y), w + 4, w[7], x);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float v = acc[r][0].x + acc[r][0].y;
      if (dset) two_sum_acc(hi[r][0], lo[r][0], v);
      else two_sum_acc(hi[r][1], lo[r][1], v);
#pragma unroll
      for (int a = 1; a < 7; ++a)
        two_sum_acc(hi[r][1 + a], lo[r][1 + a], acc[r][a].x + acc[r][a].y);
    }
  }
  double v[R][NS];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double f = compact ? exp2(1.0 - (xi[r][0] * xi[r][0] + xi[r][1] * xi[r][1] +
                                           xi[r][2] * xi[r][2])) : 1.0;
    const double low = compact ? kEx2Low : kEx2LowR2;
#pragma unroll
    for (int a = 0; a < NS; ++a) v[r][a] = (1.0 + low) * f * ((double)hi[r][a] + (double)lo[r][a]);
    const double t = compact ? v[r][0] + v[r][1] : 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) v[r][5 + d] = xi[r][d] * t - v[r][5 + d];
  }
  if (!compact) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int d = 0; d < 3; ++d)  // xi may be infinite or meaningless here
        v[r][5 + d] = -(1.0 + kEx2LowR2) * ((double)hi[r][5 + d] + (double)lo[r][5 + d]);
  }
  finish_split<Op, W, R>(op, p, tile, item, rank, sp, false, GaussStats{}, v);
}

}  // namespace lddmm
