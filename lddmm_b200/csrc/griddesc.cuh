// Descriptor of the grid that carries a pair's Gaussian kernel sums at one time step
// (grid.cuh), shared by the grid kernels and the pair sweeps that take over when a pair
// has none (gauss.cuh).
#pragma once

#include "grid.h"
#include "layout.h"

namespace lddmm {

struct GridArgs {
  const PairDesc *pd;
  const int *act;
  const int2 *blocks;     // work list: (pair, index of the tile's first 32 points)
  const int *ord;         // per pair (pt_off): the rows in the tiles' order (k-d order)
  const int *pairs;       // pairs with a grid
  const int *slot;        // per pair: index of its grid, or -1
  const long long *off, *cap;  // per grid: first node (of 6 components), nodes
  const unsigned *box;    // step's box keys [pair][6]
  const unsigned *amax;   // max |a| bits [pair]
  const unsigned *umax;   // max |u| bits [pair] (adjoint)
  unsigned long long *raw;
  double *fld;
  const GridTables *tab;
  int dmax;               // largest extent per axis
};

// Order-preserving key of a float; the largest keys belong to NaNs and infinities.
__device__ __forceinline__ unsigned float_key(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct GridDesc {
  int f[3], n[3];   // first node, nodes per axis (z even)
  long long nodes;
  bool ok;
};

// keys: min of x, y, z, then min of -x, -y, -z.
__device__ __forceinline__ GridDesc grid_desc(const unsigned *keys, long long cap, int dmax,
                                              bool finite) {
  GridDesc g;
  g.ok = finite;
  g.nodes = 1;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float lo = key_float(__ldcg(&keys[d])), hi = -key_float(__ldcg(&keys[3 + d]));
    // a margin of 0.004 nodes: the box is of the FP32 positions, which differ from the
    // FP64 ones by at most 2^-24 of 8192 scaled units (0.002 nodes), and the FP32 scale
    // by half of that
    const float a = lo * 4.0f - 4e-3f, b = hi * 4.0f + 4e-3f;
    const bool fin = fabsf(a) < 32768.0f && fabsf(b) < 32768.0f;  // also false for NaN
    g.f[d] = fin ? (int)floorf(a) - (kWin / 2 - 1) : 0;
    const int last = fin ? (int)floorf(b) + kWin / 2 : 0;
    g.n[d] = last - g.f[d] + 1;
    if (d == 2) g.n[d] += g.n[d] & 1;
    if (!fin || g.n[d] > dmax || g.n[d] < kWin) g.ok = false;
    g.nodes *= g.n[d];
  }
  if (g.nodes > cap) g.ok = false;
  return g;
}

// Whether pair p's kernel sums run on the grid at the step of `a` (adj: with u).
__device__ __forceinline__ bool grid_active(const GridArgs &a, int p, bool adj, GridDesc &g) {
  const int s = a.slot ? a.slot[p] : -1;
  if (s < 0) return false;
  const bool fin = __ldcg(&a.amax[p]) < 0x7f800000u && (!adj || __ldcg(&a.umax[p]) < 0x7f800000u);
  g = grid_desc(a.box + 6 * p, a.cap[s], a.dmax, fin);
  return g.ok;
}

// 2^k with N m 2^k <= 2^61.  In FP64: N m may exceed the largest float.
__device__ __forceinline__ int grid_scale_exp(int N, unsigned mbits) {
  const double b = (double)N * __uint_as_float(mbits);
  return b > 0.0 ? 60 - ilogb(b) : 0;
}

}  // namespace lddmm
