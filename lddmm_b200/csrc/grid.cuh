// Gaussian kernel sums through a uniform grid: the 3D shooting and adjoint steps of pairs
// with many landmarks, in O(N) instead of O(N^2) operations.
//
// K(x, y) = 2^-|x - y|^2 (scaled coordinates) is a product over the axes and smooth: on a
// grid of spacing h = 1/4,
//   2^-(x - y)^2 = sum_mn psi(x - m h) T(m - n) psi(y - n h)   per axis,
// psi a Kaiser-Bessel window over 10 nodes and T the matching grid kernel (grid.h), to
// 3.6e-11 of K(0) = 1, and its derivative to 5e-9 (the FP32 pair sums round every term
// at 6e-8).  The error falls with the distance, slower than K: 1e-7 of K itself at 3.3, 1e-6
// at 4.2, 1e-5 at 5.2 scaled units.  A kernel sum is then
//   spread    S(n) = sum_j psi(y_j - n h) a_j       (10^3 nodes per point)
//   convolve  F = T * S, one axis after the other
//   interpolate  v_i = sum_n psi(x_i - n h) F(n), and the gradient with psi'.
// All of it is FP64.  At 163,842 landmarks this is 1e10 operations per step where the
// pairs are 2.7e10 exponentials.
//
// One evaluation step of the adjoint needs U = sum_j K u_j and R = sum_j K r_j (r = a):
//   sum_j K u_j = U(x_i),
//   sum_j K (m_i.r_j + r_i.u_j) (x_i - x_j) = -grad(m_i.R + r_i.U)(x_i) / (2 ln 2),
// m = u - r = -p (gauss.cuh).
//
// The grid of a step covers the points' bounding box at that step: nodes at multiples of
// h, first node and extent per axis from the box.  Spreading adds with 64-bit integer
// atomics, in units that hold N max|a| in 61 bits (resolution N max|a| 2^-61): integer
// addition is associative, so the sums do not depend on the order of arrival and results
// are reproducible bit for bit.  A pair whose box outgrows its grid or whose operands are
// not finite is evaluated by the pair sums (gauss.cuh) in that step; both sides read the
// same descriptor, and the first convolution's CTAs, which have nothing else to do then,
// write the statistics of the pair's blocks that the pair sums' distance test reads.
#pragma once

#include "gauss.cuh"
#include "griddesc.cuh"
#include "layout.h"
#include "ops.cuh"

namespace lddmm {

constexpr int kGridMaxDim = 112;  // nodes per axis: a plane of doubles fits shared memory
constexpr int kGridKZ = 16;       // z nodes handled at once in registers
constexpr int kGridThreads = 128;
constexpr int kSpreadPts = 32;    // points of a spread tile
constexpr int kConvThreads = 256;
constexpr int kInterpWarps = 4;

// Window values (and derivatives) on one axis of point pt (of npts) at scaled coordinate
// x: val[node * npts + pt], and the window's first node relative to the grid, kept inside
// its n nodes.
template <bool DERIV>
__device__ __forceinline__ void grid_windows(const GridTables *T, double x, int pt, int npts,
                                             int first, int n, double *val, double *dval,
                                             int *o) {
  const double y = x * (1.0 / kGridH);
  const double fl = floor(y);
  const double z = 2.0 * (y - fl) - 1.0;
  o[pt] = min(max((int)fl - (kWin / 2 - 1) - first, 0), n - kWin);
#pragma unroll 5
  for (int k = 0; k < kWin; ++k) {
    double s = __ldg(&T->win[k][kWinDeg]);
#pragma unroll
    for (int i = kWinDeg - 1; i >= 0; --i) s = fma(s, z, __ldg(&T->win[k][i]));
    val[k * npts + pt] = s;
    if (DERIV) {
      double e = __ldg(&T->dwin[k][kWinDeg - 1]);
#pragma unroll
      for (int i = kWinDeg - 2; i >= 0; --i) e = fma(e, z, __ldg(&T->dwin[k][i]));
      dval[k * npts + pt] = e;
    }
  }
}

// Clears the box keys and maxima that this evaluation's sweeps fill (boxes of steps
// 1 .. T, maxima of alpha and u of every step).
__global__ void grid_reset_kernel(unsigned *keys, int nkeys, unsigned *mx, int nmx) {
  pdl_wait();
  pdl_trigger();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nkeys + nmx; i += gridDim.x * blockDim.x)
    if (i < nkeys) keys[i] = 0xffffffffu;
    else mx[i - nkeys] = 0u;
}

// FP64 tensor-core product of 8 x 4 and 4 x 8: a = A[lane / 4][lane % 4], b = B[lane % 4]
// [lane / 4], d = D[lane / 4][2 (lane % 4) + 0, 1].
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// ------------------------------------------------------------------------ spread
//
// A CTA takes a tile of 32 points that are close in space (k-d order of the initial
// positions).  For a plane m of x nodes and 8 rows n of y nodes,
//   S_c(n, k) = sum_p [psi_m psi_n a_c](p) psi_k(p)
// is an (8 x points) x (points x 16 z nodes) product for each of the 3 momenta
// components, on the FP64 tensor cores: the left operand is formed in registers, the
// right one holds the points' z windows.  A node receives one atomic per tile.  (128 points per
// tile take fewer atomics but scan four times the points for each of their nodes: shooting
// steps of 40,962 / 163,842 / 655,362 landmarks 234 / 428 / 1186 us, with 32 points 162 / 334 /
// 1120.)

struct GridSpreadSmem {
  double w[2][kWin][kSpreadPts];       // x and y windows
  double z[kWin][kSpreadPts];
  double zw[kSpreadPts][kGridKZ + 4];   // z windows over the current nodes, zero outside
  float a[6][kSpreadPts];
  int o[3][kSpreadPts];
  int lo[3], hi[3];
};

__global__ void __launch_bounds__(kGridThreads)
    grid_spread_kernel(const GridArgs A, const float4 *s0, const float4 *s1,
                       const double *__restrict__ q64, int adj) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GridSpreadSmem &sm = *reinterpret_cast<GridSpreadSmem *>(smem_raw);
  const int2 it = A.blocks[blockIdx.x];
  pdl_wait();
  pdl_trigger();
  const int p = it.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!A.act[p]) return;
  GridDesc g;
  if (!grid_active(A, p, adj != 0, g)) return;
  const PairDesc &P = A.pd[p];
  const int row0 = it.y * 32;
  const int npt = min(kSpreadPts, P.N - row0);
  if (npt <= 0) return;
  if (tid < 3) {
    sm.lo[tid] = 1 << 20;
    sm.hi[tid] = -1;
  }
  const int *ord = A.ord + P.pt_off + row0;
  for (int i = tid; i < kSpreadPts; i += kGridThreads) {
    const int g0 = i < npt ? P.pt_off + ord[i] : 0;
    float4 a = make_float4(0, 0, 0, 0), b = a;
    if (i < npt) {
      a = __ldcg(&s0[g0]);
      if (s1) b = __ldcg(&s1[g0]);
    }
    sm.a[0][i] = a.x; sm.a[1][i] = a.y; sm.a[2][i] = a.z;
    sm.a[3][i] = b.x; sm.a[4][i] = b.y; sm.a[5][i] = b.z;
  }
  __syncthreads();
  for (int i = tid; i < 3 * kSpreadPts; i += kGridThreads) {
    const int axis = i / kSpreadPts, pt = i - axis * kSpreadPts;
    const int src = min(pt, npt - 1);  // padding repeats the last point, with a = 0
    const double x = __ldcg(&q64[(size_t)(P.pt_off + ord[src]) * 3 + axis]) * P.kscale64;
    grid_windows<false>(A.tab, x, pt, kSpreadPts, g.f[axis], g.n[axis],
                        axis == 2 ? &sm.z[0][0] : &sm.w[axis][0][0], nullptr, sm.o[axis]);
    const int o = sm.o[axis][pt];
    atomicMin(&sm.lo[axis], o);
    atomicMax(&sm.hi[axis], o + kWin);
  }
  __syncthreads();
  unsigned long long *raw = A.raw + A.off[A.slot[p]] * 6;
  const int hx = sm.hi[0], hy = sm.hi[1], hz = sm.hi[2];
  const int kr = lane & 3, kq = lane >> 2;
  const int npt4 = (npt + 3) & ~3;
  const double sca = scalbn(1.0, grid_scale_exp(P.N, __ldcg(&A.amax[p])));
  const double scu = s1 ? scalbn(1.0, grid_scale_exp(P.N, __ldcg(&A.umax[p]))) : 0.0;
  for (int z0 = sm.lo[2]; z0 < hz; z0 += kGridKZ) {
    for (int i = tid; i < kSpreadPts * kGridKZ; i += kGridThreads) {
      const int pt = i / kGridKZ, k = i - pt * kGridKZ;
      const int q = z0 + k - sm.o[2][pt];
      sm.zw[pt][k] = (q >= 0 && q < kWin) ? sm.z[q][pt] : 0.0;
    }
    __syncthreads();
    const int nchunk = (hy - sm.lo[1] + 7) / 8;
    for (int u = warp; u < (hx - sm.lo[0]) * nchunk; u += kGridThreads / 32) {
      const int m = sm.lo[0] + u / nchunk, n0 = sm.lo[1] + (u % nchunk) * 8, n = n0 + kq;
      for (int c0 = 0; c0 < (s1 ? 6 : 3); c0 += 3) {
        double d[3][4] = {};
        for (int pt = kr; pt < npt4; pt += 4) {
          const unsigned i = m - sm.o[0][pt], j = n - sm.o[1][pt];
          if (!__any_sync(0xffffffffu, i < kWin && j < kWin)) continue;
          const double w = i < kWin && j < kWin ? sm.w[0][i][pt] * sm.w[1][j][pt] : 0.0;
          const double b0 = sm.zw[pt][kq], b1 = sm.zw[pt][8 + kq];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double x = w * sm.a[c0 + c][pt];
            dmma(d[c][0], d[c][1], x, b0);
            dmma(d[c][2], d[c][3], x, b1);
          }
        }
        const double sc = c0 ? scu : sca;
        if (n < hy) {
          unsigned long long *dst =
              raw + c0 * g.nodes + ((size_t)m * g.n[1] + n) * g.n[2] + z0;
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int z = (k >> 1) * 8 + kr * 2 + (k & 1);
              const long long v = __double2ll_rn(d[c][k] * sc);
              if (z0 + z < hz && v) atomicAdd(dst + (size_t)c * g.nodes + z, (unsigned long long)v);
            }
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------- convolve
//
// out(i) = sum_r T(|i - r|) in(r) along an axis of n entries (stride st) for each of m
// columns (stride ct); in shared memory.  A thread forms 4 consecutive outputs of 4
// columns with a sliding window of T; neighbouring threads take neighbouring columns, so
// an odd ct (or 1) is free of bank conflicts.

__device__ __forceinline__ void conv_axis(const double *in, int n, int st, int m, int ct,
                                          const double *T, double *out, int ost, int oct) {
  // T: 2 * kGridMaxDim + 1 values, centre at kGridMaxDim
  const int ti = (n + 3) / 4, tj = (m + 3) / 4;
  for (int u = threadIdx.x; u < ti * tj; u += kConvThreads) {
    const int i0 = (u / tj) * 4, j0 = u % tj;
    double acc[4][4] = {};
    const double *col[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) col[b] = in + min(j0 + b * tj, m - 1) * ct;
    const int r0 = max(0, i0 - kGridTaps), r1 = min(n, i0 + 4 + kGridTaps);
    const double *Tc = T + kGridMaxDim;
    double t0 = Tc[i0 - r0], t1 = Tc[i0 + 1 - r0], t2 = Tc[i0 + 2 - r0], t3 = Tc[i0 + 3 - r0];
#pragma unroll 4
    for (int r = r0; r < r1; ++r) {
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const double v = col[b][r * st];
        acc[0][b] = fma(t0, v, acc[0][b]);
        acc[1][b] = fma(t1, v, acc[1][b]);
        acc[2][b] = fma(t2, v, acc[2][b]);
        acc[3][b] = fma(t3, v, acc[3][b]);
      }
      t3 = t2;
      t2 = t1;
      t1 = t0;
      t0 = Tc[i0 - r - 1];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (i0 + a < n && j0 + b * tj < m) out[(i0 + a) * ost + (j0 + b * tj) * oct] = acc[a][b];
  }
}

__device__ __forceinline__ void load_ker(const GridTables *tab, double *T) {
  for (int i = threadIdx.x; i < 2 * kGridMaxDim + 1; i += kConvThreads) {
    const int d = abs(i - kGridMaxDim);
    T[i] = d <= kGridTaps ? __ldg(&tab->ker[d]) : 0.0;
  }
}

// Statistics of one block in the points' own order, one point per lane (u or null).
__device__ __forceinline__ void block_stats(int pt, bool live, const float4 *qs, const float4 *us,
                                            float4 *box, float4 *wu) {
  const float4 x = __ldcg(&qs[pt]);
  gauss_block_box(box, pt / kSub, live, x.x, x.y, x.z, nullptr);
  if (!us) return;
  const float s = or_inf(warp_sum_f(abs_sum(__ldcg(&us[pt]))));
  if ((threadIdx.x & 31) == 0) wu[pt / kSub] = make_float4(s, 0.0f, 0.0f, 0.0f);
}

// The plane x = blockIdx.x of component blockIdx.y of grid blockIdx.z: integers to
// doubles (the integers are cleared for the next step), z axis, y axis.  Pairs that the step does not fit: the
// statistics of their blocks (in the spread kernel this branch cost a step of 40,962 landmarks
// that does not take it 0.8 to 2.5 %).
__global__ void __launch_bounds__(kConvThreads) grid_conv_yz_kernel(
    const GridArgs A, int adj, const float4 *qs, const float4 *us, float4 *box, float4 *wu) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *T = reinterpret_cast<double *>(smem_raw);
  pdl_wait();
  pdl_trigger();
  const int p = A.pairs[blockIdx.z], c = blockIdx.y;
  if (!A.act[p]) return;
  GridDesc g;
  if (!grid_active(A, p, adj != 0, g)) {
    const int lane = threadIdx.x & 31, nw = gridDim.x * gridDim.y * (kConvThreads / 32);
    const PairDesc &P = A.pd[p];
    for (int b = (blockIdx.y * gridDim.x + blockIdx.x) * (kConvThreads / 32) + threadIdx.x / 32;
         b < P.Npad / kSub; b += nw)
      block_stats(P.pt_off + b * kSub + lane, b * kSub + lane < P.N, qs, adj ? us : nullptr, box,
                  wu);
    return;
  }
  if ((int)blockIdx.x >= g.n[0]) return;
  const int ny = g.n[1], nz = g.n[2];
  const int zs = nz + 1;  // odd row stride in shared memory
  double *b0 = T + 2 * kGridMaxDim + 2, *b1 = b0 + ny * zs;
  load_ker(A.tab, T);
  const int ex = grid_scale_exp(A.pd[p].N, c >= 3 ? __ldcg(&A.umax[p]) : __ldcg(&A.amax[p]));
  const double sc = scalbn(1.0, -ex);
  const size_t o = A.off[blockIdx.z] * 6 + c * g.nodes + (size_t)blockIdx.x * ny * nz;
  unsigned long long *raw = A.raw + o;
  for (int i0 = threadIdx.x; i0 < ny * nz; i0 += 4 * kConvThreads) {
    long long v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      v[k] = i0 + k * kConvThreads < ny * nz ? (long long)__ldcg(&raw[i0 + k * kConvThreads]) : 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k * kConvThreads;
      if (i < ny * nz) {
        b0[(i / nz) * zs + i % nz] = (double)v[k] * sc;
        raw[i] = 0ull;
      }
    }
  }
  __syncthreads();
  conv_axis(b0, nz, 1, ny, zs, T, b1, 1, zs);
  __syncthreads();
  conv_axis(b1, ny, zs, nz, 1, T, A.fld + o, nz, 1);
}

// The plane y = blockIdx.x of component blockIdx.y: x axis, in place.
__global__ void __launch_bounds__(kConvThreads) grid_conv_x_kernel(const GridArgs A, int adj) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *T = reinterpret_cast<double *>(smem_raw);
  pdl_wait();
  pdl_trigger();
  const int p = A.pairs[blockIdx.z], c = blockIdx.y;
  if (!A.act[p]) return;
  GridDesc g;
  if (!grid_active(A, p, adj != 0, g) || (int)blockIdx.x >= g.n[1]) return;
  const int nx = g.n[0], nz = g.n[2], sx = g.n[1] * nz;
  double *b0 = T + 2 * kGridMaxDim + 2;
  load_ker(A.tab, T);
  double *f = A.fld + A.off[blockIdx.z] * 6 + c * g.nodes + (size_t)blockIdx.x * nz;
  for (int i0 = threadIdx.x; i0 < nx * nz; i0 += 4 * kConvThreads) {
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = min(i0 + k * kConvThreads, nx * nz - 1), x = i / nz;
      v[k] = __ldcg(&f[(size_t)x * sx + (i - x * nz)]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i0 + k * kConvThreads < nx * nz) b0[i0 + k * kConvThreads] = v[k];
  }
  __syncthreads();
  conv_axis(b0, nx, nz, nz, 1, T, f, sx, 1);
}

// ------------------------------------------------------------------- interpolate
//
// CTA = one tile of 32 points; the warps take the x planes of the tile's bounding grid in
// turn.  A warp copies 8 y rows x 16 z nodes of a plane to its shared-memory buffer (all
// its loads in flight at once); the sums over z are (8 points x 16 z nodes) x (16 x 8
// rows) products on the FP64 tensor cores, the points' z windows in registers.  Each sum
// is then weighted with the point's x and y windows.  Node values read through broadcast
// loads into plain FMAs were held by the shared-memory pipe instead (twice the FMA time).

template <bool ADJ>
struct GridInterpSmem {
  double f[kInterpWarps][ADJ ? 6 : 3][8][kGridKZ + 4];
  double w[3][kWin][32];
  double dw[ADJ ? 3 : 1][ADJ ? kWin : 1][32];
  float cf[ADJ ? 6 : 1][32];   // m and r of the points
  int o[3][32];
  double red[kInterpWarps][ADJ ? 6 : 3][32];
};

template <bool ADJ, class Op>
__global__ void __launch_bounds__(kInterpWarps * 32, ADJ ? 2 : 4)
    grid_interp_kernel(const Op op, const GridArgs A, const double *__restrict__ q64,
                       const GaussStats gs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GridInterpSmem<ADJ> &sm = *reinterpret_cast<GridInterpSmem<ADJ> *>(smem_raw);
  constexpr int NV = ADJ ? 6 : 3, NC = ADJ ? 6 : 3;
  const int2 it = A.blocks[blockIdx.x];
  pdl_wait();
  pdl_trigger();
  const int p = it.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!A.act[p]) return;
  GridDesc g;
  if (!grid_active(A, p, ADJ, g)) return;
  const PairDesc &P = A.pd[p];
  const int row0 = it.y * 32, npt = min(32, P.N - row0);
  // a partial tile's idle lanes repeat its last row (and are not finalised)
  const bool live = lane < npt;
  const int row = npt > 0 ? A.ord[P.pt_off + row0 + min(lane, npt - 1)] : 0;
  const int kr = lane & 3, kq = lane >> 2;
  double out[4][NV];  // points 8 r + lane / 4, this lane's share of the y rows
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int k = 0; k < NV; ++k) out[r][k] = 0.0;
  if (npt > 0) {
    if (tid < 96) {
      const int axis = tid >> 5;
      const double x =
          __ldcg(&q64[(size_t)(P.pt_off + row) * 3 + axis]) * P.kscale64;
      grid_windows<ADJ>(A.tab, x, lane, 32, g.f[axis], g.n[axis], &sm.w[axis][0][0],
                        &sm.dw[ADJ ? axis : 0][0][0], sm.o[axis]);
    } else if constexpr (ADJ) {
      if (tid < 128) {
        const int gr = P.pt_off + row;
        const float4 u = __ldcg(&op.us_t[gr]), a = __ldcg(&op.as_t[gr]);
        sm.cf[0][lane] = u.x - a.x; sm.cf[1][lane] = u.y - a.y; sm.cf[2][lane] = u.z - a.z;
        sm.cf[3][lane] = a.x; sm.cf[4][lane] = a.y; sm.cf[5][lane] = a.z;
      }
    }
    __syncthreads();
    // windows of the tile and of its four groups of eight points
    int lo[3], hi[3], glo[2][4], ghi[2][4];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int o = sm.o[d][lane];
      int l = o, h = o;
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) {
        l = min(l, __shfl_xor_sync(0xffffffffu, l, off));
        h = max(h, __shfl_xor_sync(0xffffffffu, h, off));
      }
      if (d < 2)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          glo[d][r] = __shfl_sync(0xffffffffu, l, 8 * r);
          ghi[d][r] = __shfl_sync(0xffffffffu, h, 8 * r) + kWin;
        }
      lo[d] = __reduce_min_sync(0xffffffffu, o);
      hi[d] = __reduce_max_sync(0xffffffffu, o) + kWin;
    }
    lo[2] &= ~1;  // 16-byte aligned pairs of z nodes
    const double *F = A.fld + A.off[A.slot[p]] * 6;
    const int nchunk = (hi[1] - lo[1] + 7) / 8;
    for (int z0 = lo[2]; z0 < hi[2]; z0 += kGridKZ) {
      double az[4][4], adz[ADJ ? 4 : 1][ADJ ? 4 : 1];
      const int nk2 = min(kGridKZ, g.n[2] - z0) / 2;  // pairs of nodes of the grid from z0 on
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int pt = 8 * r + kq, q = z0 + 4 * s + kr - sm.o[2][pt];
          const bool in = q >= 0 && q < kWin;
          az[r][s] = in ? sm.w[2][q][pt] : 0.0;
          if constexpr (ADJ) adz[r][s] = in ? sm.dw[2][q][pt] : 0.0;
        }
      for (int u = warp; u < (hi[0] - lo[0]) * nchunk; u += kInterpWarps) {
        const int m = lo[0] + u / nchunk, n0 = lo[1] + (u % nchunk) * 8;
        const int nr = min(8, hi[1] - n0);
        __syncwarp();
        {
          constexpr int PER = 8 * (kGridKZ / 2), NL = NC * PER / 32;
          const double *f = F + ((size_t)m * g.n[1] + n0) * g.n[2] + z0;
          double2 v[NL];
#pragma unroll
          for (int k = 0; k < NL; ++k) {
            const int i = k * 32 + lane, c = i / PER, r = (i / 8) & 7, z = i & 7;
            v[k] = make_double2(0.0, 0.0);
            if (r < nr && z < nk2)
              v[k] = __ldcg(reinterpret_cast<const double2 *>(
                  f + (size_t)c * g.nodes + (size_t)r * g.n[2] + 2 * z));
          }
#pragma unroll
          for (int k = 0; k < NL; ++k) {
            const int i = k * 32 + lane, c = i / PER, r = (i / 8) & 7, z = i & 7;
            *reinterpret_cast<double2 *>(&sm.f[warp][c][r][2 * z]) = v[k];
          }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (m < glo[0][r] || m >= ghi[0][r] || n0 + 8 <= glo[1][r] || n0 >= ghi[1][r]) continue;
          const int pt = 8 * r + kq;
          const unsigned qx = m - sm.o[0][pt];
          const double wx = qx < kWin ? sm.w[0][qx][pt] : 0.0;
          double wy[2], sv[NC][2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const unsigned qy = n0 + 2 * kr + e - sm.o[1][pt];
            wy[e] = qy < kWin ? sm.w[1][qy][pt] : 0.0;
          }
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            sv[c][0] = sv[c][1] = 0.0;
#pragma unroll
            for (int s = 0; s < 4; ++s)
              dmma(sv[c][0], sv[c][1], az[r][s], sm.f[warp][c][kq][4 * s + kr]);
          }
          if constexpr (!ADJ) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
              out[r][c] = fma(wx, fma(wy[0], sv[c][0], wy[1] * sv[c][1]), out[r][c]);
          } else {
            const double dx = qx < kWin ? sm.dw[0][qx][pt] : 0.0;
            double ph[2] = {0.0, 0.0}, pd[2] = {0.0, 0.0};
#pragma unroll
            for (int c = 0; c < 6; ++c) {
              const double cf = sm.cf[c][pt];
              double dv[2] = {0.0, 0.0};
#pragma unroll
              for (int s = 0; s < 4; ++s)
                dmma(dv[0], dv[1], adz[r][s], sm.f[warp][c][kq][4 * s + kr]);
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                ph[e] = fma(cf, sv[c][e], ph[e]);
                pd[e] = fma(cf, dv[e], pd[e]);
              }
            }
            double dy[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const unsigned qy = n0 + 2 * kr + e - sm.o[1][pt];
              dy[e] = qy < kWin ? sm.dw[1][qy][pt] : 0.0;
            }
#pragma unroll
            for (int c = 0; c < 3; ++c)
              out[r][c] = fma(wx, fma(wy[0], sv[3 + c][0], wy[1] * sv[3 + c][1]), out[r][c]);
            out[r][3] = fma(dx, fma(wy[0], ph[0], wy[1] * ph[1]), out[r][3]);
            out[r][4] = fma(wx, fma(dy[0], ph[0], dy[1] * ph[1]), out[r][4]);
            out[r][5] = fma(wx, fma(wy[0], pd[0], wy[1] * pd[1]), out[r][5]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double x = out[r][k];
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      if (kr == 0) sm.red[warp][k][8 * r + kq] = x;
    }
  __syncthreads();
  if (warp) return;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = 0.0;
#pragma unroll
    for (int w = 0; w < kInterpWarps; ++w) v[k] += sm.red[w][k][lane];
    if (ADJ && k >= 3) v[k] *= -0.5 / 0.69314718055994530942;
  }
  double e = live ? op.finalize(p, row, v) : 0.0;
  gauss_next_stats(op, gs, p, -1, P.pt_off + row, live);
  if (!ADJ) {
    e = warp_sum(e);
    if (lane < 2) op.write_group(p, 2 * it.y + lane, lane ? 0.0 : e);
  }
}

}  // namespace lddmm
