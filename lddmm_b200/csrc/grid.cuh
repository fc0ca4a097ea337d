// Gaussian kernel sums through a uniform grid: the 3D shooting and adjoint steps of pairs
// with many landmarks, in O(N) instead of O(N^2) operations.
//
// K(x, y) = 2^-|x - y|^2 (scaled coordinates) is a product over the axes and smooth: on a
// grid of spacing h = 1/4,
//   2^-(x - y)^2 = sum_mn psi(x - m h) T(m - n) psi(y - n h)   per axis,
// psi a Kaiser-Bessel window over 10 nodes and T the matching grid kernel (grid.h), to
// 3.4e-11 of K(0) = 1, and its derivative to 2.5e-9 (the FP32 pair sums round every term
// at 6e-8).  A kernel sum is then
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
// same descriptor.
#pragma once

#include "gauss.cuh"
#include "griddesc.cuh"
#include "layout.h"
#include "ops.cuh"

namespace lddmm {

constexpr int kGridMaxDim = 112;  // nodes per axis: a plane of doubles fits shared memory
constexpr int kGridKZ = 16;       // z nodes handled at once in registers
constexpr int kGridThreads = 128;
constexpr int kConvThreads = 256;

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

// ------------------------------------------------------------------------ spread
//
// A CTA takes a tile of 32 or 128 points that are close in space (k-d order of the initial
// positions): thread = a line of
// nodes along z of the tile's bounding grid, which it sums over the points in registers,
// so that a node receives one atomic per tile instead of one per point.  Bound by FP64
// FMA issue (3 per node and point).

template <int TPTS>
struct GridSpreadSmem {
  double w[2][kWin][TPTS];        // x and y windows
  double zw[TPTS][kGridKZ];       // z windows over the current nodes, zero outside
  double z[kWin][TPTS];
  float a[6][TPTS];
  unsigned long long st[kGridThreads][kGridKZ + 1];  // sums of a pass, for atomics along z
  int ln[kGridThreads];           // first node of the pass's lines
  int o[3][TPTS];
  int lo[3], hi[3];
};

template <int TPTS>
__global__ void __launch_bounds__(kGridThreads)
    grid_spread_kernel(const GridArgs A, const float4 *s0, const float4 *s1,
                       const double *__restrict__ q64, int adj) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GridSpreadSmem<TPTS> &sm = *reinterpret_cast<GridSpreadSmem<TPTS> *>(smem_raw);
  const int2 it = A.blocks[blockIdx.x];
  pdl_wait();
  pdl_trigger();
  const int p = it.x, tid = threadIdx.x;
  if (!A.act[p]) return;
  GridDesc g;
  if (!grid_active(A, p, adj != 0, g)) return;
  const PairDesc &P = A.pd[p];
  const int row0 = it.y * 32;
  const int npt = min(TPTS, P.N - row0);
  if (npt <= 0) return;
  const int slot = A.slot[p];
  if (tid < 3) {
    sm.lo[tid] = 1 << 20;
    sm.hi[tid] = -1;
  }
  const int *ord = A.ord + P.pt_off + row0;
  for (int i = tid; i < TPTS; i += kGridThreads) {
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
  for (int i = tid; i < 3 * TPTS; i += kGridThreads) {
    const int axis = i / TPTS, pt = i - axis * TPTS;
    const int src = min(pt, npt - 1);
    const double x = __ldcg(&q64[(size_t)(P.pt_off + ord[src]) * 3 + axis]) * P.kscale64;
    grid_windows<false>(A.tab, x, pt, TPTS, g.f[axis], g.n[axis],
                        axis == 2 ? &sm.z[0][0] : &sm.w[axis][0][0], nullptr, sm.o[axis]);
    const int o = sm.o[axis][pt];
    atomicMin(&sm.lo[axis], o);
    atomicMax(&sm.hi[axis], o + kWin);
  }
  __syncthreads();
  const int lx = sm.lo[0], ly = sm.lo[1], lz = sm.lo[2];
  const int nx = sm.hi[0] - lx, ny = sm.hi[1] - ly, nlines = nx * ny;
  unsigned long long *raw = A.raw + A.off[slot] * 6;
  for (int z0 = lz; z0 < sm.hi[2]; z0 += kGridKZ) {
    for (int i = tid; i < TPTS * kGridKZ; i += kGridThreads) {
      const int pt = i / kGridKZ, k = i - pt * kGridKZ;
      const int q = z0 + k - sm.o[2][pt];
      sm.zw[pt][k] = (q >= 0 && q < kWin && pt < npt) ? sm.z[q][pt] : 0.0;
    }
    __syncthreads();
    for (int c0 = 0; c0 < (s1 ? 6 : 3); c0 += 3) {
      const int ex = grid_scale_exp(P.N, c0 ? __ldcg(&A.umax[p]) : __ldcg(&A.amax[p]));
      const double sc = scalbn(1.0, ex);
      for (int l0 = 0; l0 < nlines; l0 += kGridThreads) {
        const int ln = l0 + tid;
        const int m = lx + ln / ny, n = ly + ln % ny;
        double acc[3][kGridKZ];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int k = 0; k < kGridKZ; ++k) acc[c][k] = 0.0;
        if (ln < nlines) {
#pragma unroll 1
          for (int pt = 0; pt < npt; ++pt) {
            const unsigned i = m - sm.o[0][pt], j = n - sm.o[1][pt];
            if (i >= kWin || j >= kWin) continue;
            const double w = sm.w[0][i][pt] * sm.w[1][j][pt];
            const double w0 = w * sm.a[c0][pt], w1 = w * sm.a[c0 + 1][pt],
                         w2 = w * sm.a[c0 + 2][pt];
#pragma unroll
            for (int k = 0; k < kGridKZ; k += 2) {
              const double2 z = *reinterpret_cast<const double2 *>(&sm.zw[pt][k]);
              acc[0][k] = fma(w0, z.x, acc[0][k]);
              acc[1][k] = fma(w1, z.x, acc[1][k]);
              acc[2][k] = fma(w2, z.x, acc[2][k]);
              acc[0][k + 1] = fma(w0, z.y, acc[0][k + 1]);
              acc[1][k + 1] = fma(w1, z.y, acc[1][k + 1]);
              acc[2][k + 1] = fma(w2, z.y, acc[2][k + 1]);
            }
          }
        }
        // neighbouring threads add neighbouring z nodes
        const int nl = min(kGridThreads, nlines - l0), nk = min(kGridKZ, sm.hi[2] - z0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          __syncthreads();  // the previous pass's or component's atomics have read st and ln
          if (c == 0) sm.ln[tid] = (m * g.n[1] + n) * g.n[2];
#pragma unroll
          for (int k = 0; k < kGridKZ; ++k)
            sm.st[tid][k] = (unsigned long long)__double2ll_rn(acc[c][k] * sc);
          __syncthreads();
          unsigned long long *dst = raw + (c0 + c) * g.nodes + z0;
          for (int i = tid; i < nl * kGridKZ; i += kGridThreads) {
            const int l = i / kGridKZ, k = i - l * kGridKZ;
            const unsigned long long v = sm.st[l][k];
            if (k < nk && v) atomicAdd(dst + sm.ln[l] + k, v);
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

// The plane x = blockIdx.x of component blockIdx.y of grid blockIdx.z: integers to
// doubles (the integers are cleared for the next step), z axis, y axis.
__global__ void __launch_bounds__(kConvThreads) grid_conv_yz_kernel(const GridArgs A, int adj) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *T = reinterpret_cast<double *>(smem_raw);
  pdl_wait();
  pdl_trigger();
  const int p = A.pairs[blockIdx.z], c = blockIdx.y;
  if (!A.act[p]) return;
  GridDesc g;
  if (!grid_active(A, p, adj != 0, g) || (int)blockIdx.x >= g.n[0]) return;
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
// CTA = one tile of 32 points, lane = point; the warps take the x planes of the
// tile's bounding grid in turn.  A warp copies 8 or 16 rows x 16 z nodes of a plane to its
// shared-memory buffer (all its loads in flight at once) and sums them against the lanes'
// windows, the z windows in registers; the node values are read by all lanes at the same
// address.  Then the rows are finalised as after a pair sweep.  Bound by FP64 FMA issue.

template <bool ADJ>
struct InterpShape {  // warps per tile, y rows per copy, CTAs per SM
  static constexpr int kWarps = ADJ ? 4 : 8, kRows = ADJ ? 8 : 16, kCtas = ADJ ? 3 : 2;
};

template <bool ADJ>
struct GridInterpSmem {
  double2 f[InterpShape<ADJ>::kWarps][InterpShape<ADJ>::kRows][ADJ ? 6 : 3][kGridKZ / 2];  // reused for the sums
  double w[3][kWin][32];
  double dw[ADJ ? 3 : 1][ADJ ? kWin : 1][32];
  int o[3][32];
};

template <bool ADJ, class Op>
__global__ void __launch_bounds__(InterpShape<ADJ>::kWarps * 32, InterpShape<ADJ>::kCtas)
    grid_interp_kernel(const Op op, const GridArgs A, const double *__restrict__ q64,
                       const GaussStats gs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GridInterpSmem<ADJ> &sm = *reinterpret_cast<GridInterpSmem<ADJ> *>(smem_raw);
  constexpr int NV = ADJ ? 6 : 3, NC = ADJ ? 6 : 3;
  constexpr int kInterpWarps = InterpShape<ADJ>::kWarps, kInterpRows = InterpShape<ADJ>::kRows;
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
  double out[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) out[k] = 0.0;
  if (npt > 0) {
    if (tid < 96) {
      const int axis = tid >> 5;
      const double x =
          __ldcg(&q64[(size_t)(P.pt_off + row) * 3 + axis]) * P.kscale64;
      grid_windows<ADJ>(A.tab, x, lane, 32, g.f[axis], g.n[axis], &sm.w[axis][0][0],
                        &sm.dw[ADJ ? axis : 0][0][0], sm.o[axis]);
    }
    double cm[3], cr[3];  // adjoint: coefficients of R and U in the row's scalar field
    if constexpr (ADJ) {
      const int gr = P.pt_off + row;
      const float4 u = __ldcg(&op.us_t[gr]), a = __ldcg(&op.as_t[gr]);
      cm[0] = (double)u.x - a.x; cm[1] = (double)u.y - a.y; cm[2] = (double)u.z - a.z;
      cr[0] = a.x; cr[1] = a.y; cr[2] = a.z;
    }
    __syncthreads();
    int o[3], lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      o[d] = sm.o[d][lane];
      lo[d] = __reduce_min_sync(0xffffffffu, o[d]);
      hi[d] = __reduce_max_sync(0xffffffffu, o[d]) + kWin;
    }
    lo[2] &= ~1;  // 16-byte aligned pairs of z nodes
    const double *F = A.fld + A.off[A.slot[p]] * 6;
    for (int z0 = lo[2]; z0 < hi[2]; z0 += kGridKZ) {
      double wz[kGridKZ], dz[ADJ ? kGridKZ : 1];
      const int nk2 = min(kGridKZ, g.n[2] - z0) / 2;  // pairs of nodes of the grid from z0 on
#pragma unroll
      for (int k = 0; k < kGridKZ; ++k) {
        const int q = z0 + k - o[2];
        const bool in = q >= 0 && q < kWin;
        wz[k] = in ? sm.w[2][q][lane] : 0.0;
        if (ADJ) dz[k] = in ? sm.dw[2][q][lane] : 0.0;
      }
      for (int m = lo[0] + warp; m < hi[0]; m += kInterpWarps) {
        const unsigned qx = m - o[0];
        const double wx = qx < kWin ? sm.w[0][qx][lane] : 0.0;
        const double dx = ADJ && qx < kWin ? sm.dw[0][qx][lane] : 0.0;
        for (int n0 = lo[1]; n0 < hi[1]; n0 += kInterpRows) {
          const int nr = min(kInterpRows, hi[1] - n0);
          __syncwarp();
          {
            constexpr int PER = NC * (kGridKZ / 2);  // pairs per row
            const double *f = F + ((size_t)m * g.n[1] + n0) * g.n[2] + z0;
            double2 v[(kInterpRows * PER + 31) / 32];
#pragma unroll
            for (int k = 0; k < (kInterpRows * PER + 31) / 32; ++k) {
              const int i = k * 32 + lane, r = i / PER, q = i - r * PER, c = q / (kGridKZ / 2),
                        z = q - c * (kGridKZ / 2);
              v[k] = make_double2(0.0, 0.0);
              if (r < nr && z < nk2)
                v[k] = __ldcg(reinterpret_cast<const double2 *>(
                    f + (size_t)c * g.nodes + (size_t)r * g.n[2] + 2 * z));
            }
#pragma unroll
            for (int k = 0; k < (kInterpRows * PER + 31) / 32; ++k) {
              const int i = k * 32 + lane;
              if (i < kInterpRows * PER) (&sm.f[warp][0][0][0])[i] = v[k];
            }
          }
          __syncwarp();
          for (int r = 0; r < nr; ++r) {
            const unsigned qy = n0 + r - o[1];
            const bool in = qx < kWin && qy < kWin;
            const double wy = in ? sm.w[1][qy][lane] : 0.0;
            const double w = wx * wy;
            if constexpr (!ADJ) {
              double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
              for (int k = 0; k < kGridKZ / 2; ++k)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                  const double2 v = sm.f[warp][r][c][k];
                  s[c] = fma(wz[2 * k], v.x, s[c]);
                  s[c] = fma(wz[2 * k + 1], v.y, s[c]);
                }
#pragma unroll
              for (int c = 0; c < 3; ++c) out[c] = fma(w, s[c], out[c]);
            } else {
              const double dy = in ? sm.dw[1][qy][lane] : 0.0;
              double s[3] = {0.0, 0.0, 0.0}, ph = 0.0, pd = 0.0;
#pragma unroll
              for (int k = 0; k < kGridKZ / 2; ++k) {
                double e0 = 0.0, e1 = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                  const double2 v = sm.f[warp][r][d][k], y = sm.f[warp][r][3 + d][k];
                  e0 = fma(cr[d], y.x, fma(cm[d], v.x, e0));
                  e1 = fma(cr[d], y.y, fma(cm[d], v.y, e1));
                  s[d] = fma(wz[2 * k], y.x, s[d]);
                  s[d] = fma(wz[2 * k + 1], y.y, s[d]);
                }
                ph = fma(wz[2 * k], e0, ph);
                ph = fma(wz[2 * k + 1], e1, ph);
                pd = fma(dz[2 * k], e0, pd);
                pd = fma(dz[2 * k + 1], e1, pd);
              }
#pragma unroll
              for (int c = 0; c < 3; ++c) out[c] = fma(w, s[c], out[c]);
              out[3] = fma(dx * wy, ph, out[3]);
              out[4] = fma(wx * dy, ph, out[4]);
              out[5] = fma(w, pd, out[5]);
            }
          }
        }
      }
    }
  }
  __syncthreads();
  double(*red)[NV][32] = reinterpret_cast<double(*)[NV][32]>(&sm.f[0][0][0][0]);
#pragma unroll
  for (int k = 0; k < NV; ++k) red[warp][k][lane] = out[k];
  __syncthreads();
  if (warp) return;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = 0.0;
#pragma unroll
    for (int w = 0; w < kInterpWarps; ++w) v[k] += red[w][k][lane];
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
