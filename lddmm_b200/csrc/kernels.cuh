// Deformation and varifold kernel functions in scaled coordinates.
//
// The host stores positions pre-multiplied by a per-pair scale s so that the
// exponent needs no multiply inside the pair loop:
//   Gaussian  K = exp(-|dq|^2 / sigma^2)  ->  s = sqrt(log2 e) / sigma,  K = 2^(-r2)
//   Matern    K = P_n(d) exp(-d), d = |dq| / sigma  ->  s = log2 e / sigma,
//             r = |dq_s| = d log2 e,  exp(-d) = 2^(-r),  d = r ln 2
// The gradient weight W satisfies  dK/dq_i = pd_fac * W * dq_scaled,  with pd_fac
// folded in per pair on the host (PairDesc::pd_fac).
//
// Kernel definitions follow Cpp/src/computeKernel.cpp:26-41 (Gaussian),
// :160-238 (3D Matern orders 0..4; the 2D Matern family is MaternBessel2D below) and their derivatives Cpp/src/dqKernel.cpp:56-57,
// :200-300.  Matern order 0 is not differentiable at 0; the reference leaves its
// gradient at zero (dqKernel.cpp has no order-0 case), and so does W here.
#pragma once

#include <cmath>

#include "common.cuh"

namespace lddmm {

enum KernelFamily : int {
  kGauss = -1,
  kMatern0 = 0,
  kMatern1 = 1,
  kMatern2 = 2,
  kMatern3 = 3,
  kMatern4 = 4,
};

template <int ORDER>
struct DefKernel;

// One value or a packed pair: the same operations in the same order, so that the packed
// sweeps are bitwise the scalar ones.
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ void vdup(float c, float &v) { v = c; }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ void vdup(float c, float2 &v) { v = make_float2(c, c); }

template <>
struct DefKernel<-1> {
  static constexpr int kUnroll = 2;  // j pairs unrolled in the persistent sweeps
  static __device__ __forceinline__ float val(float nr2) { return ex2f(nr2); }
  static __device__ __forceinline__ void val_w(float nr2, float &K, float &W) {
    K = ex2f(nr2);
    W = K;
  }
  static __device__ __forceinline__ float2 val2(float2 r2) {
    return make_float2(ex2f(-r2.x), ex2f(-r2.y));
  }
  static __device__ __forceinline__ void val_w2(float2 r2, float2 &K, float2 &W) {
    K = val2(r2);
    W = K;
  }
};

// Matern kernels take the NEGATED squared scaled distance for symmetry with the
// Gaussian (the pair loops produce -r2 with free negation modifiers); the packed forms
// take the squared distance.
template <int ORDER>
struct DefKernel {
  static constexpr int kUnroll = 2;
  // e times the polynomials in d = r ln 2
  template <class V>
  static __device__ __forceinline__ V times_k(V e, V r) {
    if (ORDER == 0) return e;
    V l, c[5];
    vdup(kLn2, l);
    const float k[5][5] = {{1.0f}, {1.0f, 1.0f}, {1.0f, 1.0f, 1.0f / 3.0f},
                           {1.0f, 1.0f, 0.4f, 1.0f / 15.0f},
                           {1.0f, 1.0f, 3.0f / 7.0f, 2.0f / 21.0f, 1.0f / 105.0f}};
#pragma unroll
    for (int n = 0; n <= ORDER; ++n) vdup(k[ORDER][n], c[n]);
    if (ORDER == 1) return vmul(e, vfma(r, l, c[0]));
    const V d = vmul(r, l);
    V s = c[ORDER];
#pragma unroll
    for (int n = ORDER - 1; n >= 0; --n) s = vfma(d, s, c[n]);
    return vmul(e, s);
  }
  template <class V>
  static __device__ __forceinline__ V times_w(V e, V r) {
    if (ORDER <= 1) return e;
    V l, a, b;
    vdup(kLn2, l);
    vdup(ORDER == 2 ? 1.0f : ORDER == 3 ? 3.0f : 6.0f, a);
    V s = vfma(r, l, a);
    if (ORDER >= 3) {
      const V d = vmul(r, l);
      vdup(ORDER == 3 ? 3.0f : 15.0f, b);
      s = vfma(d, s, b);
      if (ORDER == 4) s = vfma(d, s, b);
    }
    return vmul(e, s);
  }
  static __device__ __forceinline__ float val(float nr2) {
    const float r = sqrtf_approx(-nr2);
    return times_k(ex2f(-r), r);
  }
  static __device__ __forceinline__ void val_w(float nr2, float &K, float &W) {
    const float r = sqrtf_approx(-nr2), e = ex2f(-r);
    K = times_k(e, r);
    W = ORDER == 0 ? 0.0f : times_w(e, r);
  }
  static __device__ __forceinline__ float2 val2(float2 r2) {
    const float2 r = make_float2(sqrtf_approx(r2.x), sqrtf_approx(r2.y));
    return times_k(make_float2(ex2f(-r.x), ex2f(-r.y)), r);
  }
  static __device__ __forceinline__ void val_w2(float2 r2, float2 &K, float2 &W) {
    const float2 r = make_float2(sqrtf_approx(r2.x), sqrtf_approx(r2.y)),
                 e = make_float2(ex2f(-r.x), ex2f(-r.y));
    K = times_k(e, r);
    W = ORDER == 0 ? make_float2(0.0f, 0.0f) : times_w(e, r);
  }
};

// ------------------------------------------------------ 2D Matern (Bessel K)
// In 2D the reference's Matern family is built from p0(x) = x^2 K0(x) and
// p1(x) = x K1(x), x = |dq| / sigma (Cpp/src/computeKernel.cpp:44-155,
// Cpp/src/dqKernel.cpp:68-195, with p0Fcn / p1Fcn of Cpp/src/polybesselk.cpp:14-96 and
// their cut-offs: p0(0) = 0, p1(0) = 1).  The kernels of orders 0..4 are
//   K0 = p1,  K1 = p0/2 + p1,  K2 = (4 p0 + (8 + x^2) p1) / 8,
//   K3 = ((24 + x^2) p0 + 8 (6 + x^2) p1) / 48,
//   K4 = (12 (16 + x^2) p0 + (384 + x^2 (72 + x^2)) p1) / 384,
// and the reference's dq factor of order n is -K_{n-1} / (2 n sigma^2), so the gradient
// weight here is W = K_{n-1} / (2 n) with pd_fac = -1 / (sigma^2 kscale), kscale = 1 / sigma.
//
// p0 and p1 are evaluated in FP32 from the mathematics of K0 and K1, not from the
// reference's rational approximations:
//   x <= 2  ascending series (Abramowitz & Stegun 9.6.13 and 9.6.11, n = 1), 8 terms in
//           y = x^2 / 4 (the next is below 2e-9):  K0 = -(ln(x/2) + gamma) I0 + sum_k H_k
//           y^k / (k!)^2,  x K1 = 1 + x ln(x/2) I1 - y sum_k (psi(k+1) + psi(k+2)) y^k /
//           (k! (k+1)!), four polynomials by Horner's rule;
//   x > 2   sqrt(x) e^x K_nu(x) as a polynomial of degree 8 in t = 2 / x on (0, 1]: Chebyshev
//           interpolation of K0 and K1 in double precision, within 2.1e-9.
// In FP32 the relative error against double-precision K0 / K1 is below 3e-7 rms (3e-6 at most,
// K0 near x = 2) up to x = 10 and 7e-7 rms beyond, where the exponential's argument rounds.
// Bound by FMA issue (18 and 28 per point); a trapezoid rule with 14 exponentials for 2 < x
// <= 10 and an asymptotic series beyond took 7.55 instead of 6.73 us per shooting step of 500
// points and 8.54 instead of 7.43 per adjoint step.
__device__ __forceinline__ float lg2f_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void bessel_p01(float x, float &p0, float &p1) {
  constexpr float kGamma = 0.5772156649015329f;
  if (x < 1e-18f) {
    p0 = 0.0f;
    p1 = 1.0f;
    return;
  }
  if (x <= 2.0f) {
    // c_k = 1 / (k!)^2 and e_k = 1 / (k! (k+1)!); H_k c_k; (H_k + H_{k+1} - 2 gamma) e_k
    constexpr float c[8] = {1.0f, 1.0f, 0.25f, 2.77777778e-2f, 1.73611111e-3f, 6.94444444e-5f,
                            1.92901235e-6f, 3.93675989e-8f};
    constexpr float e[8] = {1.0f, 0.5f, 8.33333333e-2f, 6.94444444e-3f, 3.47222222e-4f,
                            1.15740741e-5f, 2.75573192e-7f, 4.92094986e-9f};
    constexpr float H[8] = {0.0f, 1.0f, 1.5f, 1.83333333f, 2.08333333f, 2.28333333f, 2.45f,
                            2.59285714f};
    constexpr float S[8] = {-0.154431330f, 1.34556867f, 2.17890200f, 2.76223534f,
                            3.21223534f, 3.57890200f, 3.88842581f, 4.15628296f};
    const float y = 0.25f * x * x;
    float i0 = c[7], s0 = H[7] * c[7], i1 = e[7], s1 = S[7] * e[7];
#pragma unroll
    for (int k = 6; k >= 0; --k) {
      i0 = fmaf(i0, y, c[k]);
      s0 = fmaf(s0, y, H[k] * c[k]);
      i1 = fmaf(i1, y, e[k]);
      s1 = fmaf(s1, y, S[k] * e[k]);
    }
    const float L = (lg2f_approx(x) - 1.0f) * kLn2;  // ln(x / 2)
    p0 = x * x * fmaf(-(L + kGamma), i0, s0);
    p1 = fmaf(2.0f * y * L, i1, fmaf(-y, s1, 1.0f));
    return;
  }
  constexpr float k0[9] = {1.253314135156027f,   -0.07833176026425974f, 0.022020063119861162f,
                           -0.011349035288939255f, 0.00801971889052289f, -0.006020387370799306f,
                           0.0037290997491742344f, -0.0015056031184785617f,
                           0.0002809539465136094f};
  constexpr float k1[9] = {1.2533141398699563f,  0.23499595959859942f, -0.03670538480055631f,
                           0.01591652569667686f, -0.01039640273343412f, 0.007511644585594581f,
                           -0.0045668498089172106f, 0.001826349388488236f,
                           -0.00033900994429618246f};
  const float t = 2.0f * rcpf_approx(x);
  float a0 = k0[8], a1 = k1[8];
#pragma unroll
  for (int k = 7; k >= 0; --k) {
    a0 = fmaf(a0, t, k0[k]);
    a1 = fmaf(a1, t, k1[k]);
  }
  const float c = sqrtf_approx(x) * ex2f(-x * kLog2e);  // sqrt(x) e^-x
  p0 = x * c * a0;
  p1 = c * a1;
}

template <int ORDER>
struct MaternBessel2D {
  static constexpr int kUnroll = 1;  // of about 200 instructions each
  // K_n(x) of the family in terms of p0, p1 and x^2
  template <int N>
  static __device__ __forceinline__ float form(float p0, float p1, float x2) {
    if (N == 0) return p1;
    if (N == 1) return fmaf(0.5f, p0, p1);
    if (N == 2) return fmaf(0.5f, p0, fmaf(0.125f * x2, p1, p1));
    if (N == 3) return fmaf(fmaf(x2, 1.0f / 48.0f, 0.5f), p0, fmaf(x2, 1.0f / 6.0f, 1.0f) * p1);
    return fmaf(fmaf(x2, 1.0f / 32.0f, 0.5f), p0,
                fmaf(x2 * (72.0f + x2), 1.0f / 384.0f, 1.0f) * p1);
  }
  static __device__ __forceinline__ float val(float nr2) {
    const float x = sqrtf_approx(-nr2);
    float p0, p1;
    bessel_p01(x, p0, p1);
    return form<ORDER>(p0, p1, -nr2);
  }
  static __device__ __forceinline__ void val_w(float nr2, float &K, float &W) {
    const float x = sqrtf_approx(-nr2);
    float p0, p1;
    bessel_p01(x, p0, p1);
    K = form<ORDER>(p0, p1, -nr2);
    W = (ORDER == 0) ? 0.0f : form<(ORDER > 0 ? ORDER - 1 : 0)>(p0, p1, -nr2) *
                                  (1.0f / (2.0f * (ORDER > 0 ? ORDER : 1)));
  }
  static __device__ __forceinline__ float2 val2(float2 r2) {
    return make_float2(val(-r2.x), val(-r2.y));
  }
  static __device__ __forceinline__ void val_w2(float2 r2, float2 &K, float2 &W) {
    val_w(-r2.x, K.x, W.x);
    val_w(-r2.y, K.y, W.y);
  }
};

// Deformation kernel of dimension D and order: the 2D Matern family has its own
// (Bessel K) definition; every other combination uses DefKernel.
template <int D, int ORDER>
struct DefKernelOf {
  using type = DefKernel<ORDER>;
};
template <int ORDER>
struct DefKernelOf<2, ORDER> {
  using type = MaternBessel2D<ORDER>;
};
template <>
struct DefKernelOf<2, -1> {
  using type = DefKernel<-1>;
};

// Host-side scale and gradient factor for a family (see the header comment).
inline void def_kernel_scales(int order, int dim, double width, float *kscale,
                              double *pd_fac) {
  const double log2e = 1.4426950408889634;
  const double w2 = width * width;
  if (order == -1) {
    const double s = std::sqrt(log2e) / width;
    *kscale = (float)s;
    *pd_fac = -2.0 / (w2 * s);
    return;
  }
  if (dim == 2) {  // Bessel forms in x = |dq| / sigma
    const double s = 1.0 / width;
    *kscale = (float)s;
    *pd_fac = order == 0 ? 0.0 : -1.0 / (w2 * s);
    return;
  }
  const double s = log2e / width;
  *kscale = (float)s;
  switch (order) {
    case 1: *pd_fac = -1.0 / (w2 * s); break;
    case 2: *pd_fac = -1.0 / (3.0 * w2 * s); break;
    case 3: *pd_fac = -1.0 / (15.0 * w2 * s); break;
    case 4: *pd_fac = -1.0 / (105.0 * w2 * s); break;
    default: *pd_fac = 0.0; break;
  }
}

// ------------------------------------------------------------ varifold kernels
// Centre kernels (Cpp/src/varifold3D.cpp:41-93), in centres scaled by cscale:
//   'G'  k = exp(-|dc|^2/sigma^2) = 2^(-r2),  cscale = sqrt(log2 e)/sigma,
//        dk/dc_i = -2 k / sigma^2 dc  ->  gradient weight k
//   'C'  k = 1 / (1 + |dc|^2/sigma^2),         cscale = 1/sigma,
//        dk/dc_i = -2 k^2 / sigma^2 dc  ->  gradient weight k^2
// Both share dc_fac = -2 / (sigma^2 cscale) on the host.  cscale is rounded to FP32 except
// with `exact` (vfd.cuh, where that rounding would be the largest systematic error).
template <char CT>
struct CenKernel {
  static __device__ __forceinline__ void val_w(float nr2, float &k, float &kw) {
    if (CT == 'G') {
      k = ex2f(nr2);
      kw = k;
    } else {
      k = rcpf_approx(1.0f - nr2);
      kw = k * k;
    }
  }
};

inline void cen_kernel_scales(char type, double width, bool exact, double *cscale,
                              double *dc_fac) {
  const double log2e = 1.4426950408889634;
  const double s = (type == 'G') ? std::sqrt(log2e) / width : 1.0 / width;
  *cscale = exact ? s : (double)(float)s;
  *dc_fac = -2.0 / (width * width * s);
}

// Direction kernels (Cpp/src/varifold3D.cpp:95-188): value b(ang) and derivative
// b'(ang), ang = n_i . n_j.  ow2 = 2 / dirKnlWidth^2 for the Gaussian kinds.
template <char DT>
struct DirKernel {
  static __device__ __forceinline__ void val_d(float ang, float ow2, float &b, float &db) {
    if (DT == 'B') {
      b = ang * ang;
      db = 2.0f * ang;
    } else if (DT == 'L') {
      b = ang;
      db = 1.0f;
    } else if (DT == 'O') {
      b = ex2f((ang - 1.0f) * ow2 * kLog2e);
      db = ow2 * b;
    } else {  // 'U'
      b = ex2f((ang * ang - 1.0f) * ow2 * kLog2e);
      db = 2.0f * ang * ow2 * b;
    }
  }
};

}  // namespace lddmm
