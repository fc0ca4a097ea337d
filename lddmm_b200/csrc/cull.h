// Distance test of the adjoint's Gaussian pair sweep (gauss.cuh), for host and device.
//
// The sweep adds, for every row i of a tile I,
//   (a) sum_j K_ij u_j   and   (b) sum_j K_ij (m_i.r_j + r_i.u_j) (x_i - x_j).
// A 32-column block B at box distance g, of weights U_B = sum |u_j| and R_B = sum |r_j|, adds
// at most 2^-g^2 U_B to (a) and, for g >= 1 (t 2^-t^2 falls from 0.85 on), at most
// 2^-g^2 g (|m_i| R_B + |r_i| U_B) to (b).  It is skipped when
//   2^-g^2 U_B <= e U_I,   2^-g^2 g U_B <= e d U_I   and   2^-g^2 g R_B <= e d R_I,
// e = 2^-26 2^-diag^2 / nblk, d = diag / 4.  K >= 2^-diag^2 inside the tile and the last two
// bound the two parts of (b) one by one, so for every row, whatever its own m_i and r_i, all
// skipped blocks together change
//   (a) by at most 2^-26 of sum_{j in I} K_ij |u_j|,
//   (b) by at most 2^-26 of sum_{j in I} K_ij (|m_i| |r_j| + |r_i| |u_j|) d.
// The second is the size of the row's own-tile terms at a quarter of the tile's diagonal; the
// FP32 products of a compact tile are rounded at 2^-24 of twice that and more.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define LDDMM_HD __host__ __device__ __forceinline__
#else
#define LDDMM_HD inline
#endif

namespace lddmm {

constexpr float kCullBits = 26.0f;

LDDMM_HD float cull_lg2(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return std::log2(x);
#endif
}

// log2 of a tile's weight; -inf (nothing is skipped) when it is not finite.
LDDMM_HD float lg2_finite(float s) { return cull_lg2(s < INFINITY ? s : 0.0f); }

struct AdjointCut {
  float u, r, q;  // log2 of 1 / (e U_I), 1 / (e R_I), 1 / d
};

LDDMM_HD AdjointCut adjoint_cut(float diag2, int nblk, float U_I, float R_I) {
  const float bits = diag2 + kCullBits + cull_lg2((float)nblk);
  return {bits - lg2_finite(U_I), bits - lg2_finite(R_I), 2.0f - 0.5f * cull_lg2(diag2)};
}

// g2: squared box distance (NaN or a weight of infinity: not skipped).
LDDMM_HD bool adjoint_skips(const AdjointCut &c, float g2, float U_B, float R_B) {
  const float gd = 0.5f * cull_lg2(g2) + c.q;  // log2(g / d)
  const float h = g2 - (gd > 0.0f ? gd : 0.0f);
  return g2 >= 1.0f && h >= cull_lg2(U_B) + c.u && h >= cull_lg2(R_B) + c.r;
}

}  // namespace lddmm
