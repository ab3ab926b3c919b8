// Point-wise numerics of the cell-centered finite-volume hot path, shared by
// every kernel of this library: WENO3/WENO5 face reconstruction (with and
// without the analytic gradient), the Rusanov flux for the Euler and
// shallow-water equations and its analytic Jacobians.
//
// Every expression below keeps the operand order and association of the
// reference implementation so that, compiled without FMA contraction
// (nvcc -fmad=false), each value is bit-identical to the reference's
// double-precision result.  The few places that cannot be bit-identical are
// marked "deviation" and are within the stated parity tolerance.
//
// The gradient and flux-Jacobian functions are templates on the scalar type:
// T = double is the reference's arithmetic (every literal is a T, so the
// double instantiation is the same expression tree); T = float serves the
// reduced-order model's approximate Jacobians.
//
// Reference (pressio-demoapps, include/pressiodemoapps/...):
//   impl/weno5.hpp:56-178   weno5           -> weno5_face
//   impl/weno5.hpp:180-434  weno5WithGrad   -> weno5_face_grad
//   impl/weno3.hpp:56-132   weno3           -> weno3_face
//   impl/weno3.hpp:134-246  weno3WithGrad   -> weno3_face_grad
//   impl/euler_rusanov_flux_values_function.hpp:54-208   -> euler*_flux
//   impl/euler_rusanov_flux_jacobian_function.hpp:54-406 -> euler*_flux_jac
//   impl/swe_rusanov_flux_values_function.hpp:54-97      -> swe_flux
//   impl/swe_rusanov_flux_jacobian_function.hpp:54-137   -> swe_flux_jac
#pragma once

#include <math.h>

#include <type_traits>

#include "fp64_intpipe.cuh"

#if defined(__CUDACC__)
#define PDA_HD __host__ __device__ __forceinline__
#else
#define PDA_HD inline
#endif

namespace pda {

enum Scheme : int { FirstOrder = 0, Weno3 = 1, Weno5 = 2 };

// half-width of the reconstruction stencil: 1, 2, 3
template <int S> struct SchemeTraits;
template <> struct SchemeTraits<FirstOrder> { static constexpr int h = 1; };
template <> struct SchemeTraits<Weno3> { static constexpr int h = 2; };
template <> struct SchemeTraits<Weno5> { static constexpr int h = 3; };

// Division and square root of runtime operands.  Device code computes them
// on the integer pipe (fp64_intpipe.cuh): the IEEE round-to-nearest results,
// bit for bit, without occupying GB300's FP64 pipe (one warp instruction per
// ~64 cycles per SM sub-partition), which is left to the multiplications and
// additions.  INL = true expands them in place (the pivots of the LSPG solve,
// one division in a serial chain); elsewhere they are calls: inlined, the face
// kernels outgrew the instruction cache and ran slower.  Host code uses the
// operators.  Compiling with -DPDA_FP64_PIPE_DIVSQRT selects FP64-pipe divisions,
// roots, and products that go through the functions of this file on the device
// too (the same results), for comparison; the groups of products that the tile
// kernels and the balance check together call ip:: directly and stay on the
// integer pipe.
template <bool INL = false>
PDA_HD double div_rn(double a, double b) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (INL) return ip::div(a, b);
  else return ip::div_call(a, b);
#else
  return a / b;
#endif
}
template <bool INL = false>
PDA_HD double sqrt_rn(double x) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (INL) return ip::sqrt(x);
  else return ip::sqrt_call(x);
#else
  return sqrt(x);
#endif
}
// Several quotients by one divisor: the same IEEE quotients as div_rn, with
// the divisor's reciprocal formed once on the device.
template <bool INL = false>
PDA_HD Quot2 div2_rn(double a0, double a1, double b) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (INL) return ip::div2(a0, a1, b);
  else return ip::div2_call(a0, a1, b);
#else
  return {a0 / b, a1 / b};
#endif
}
template <bool INL = false>
PDA_HD Quot3 div3_rn(double a0, double a1, double a2, double b) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (INL) return ip::div3(a0, a1, a2, b);
  else return ip::div3_call(a0, a1, a2, b);
#else
  return {a0 / b, a1 / b, a2 / b};
#endif
}
template <bool INL = false>
PDA_HD Quot4 div4_rn(double a0, double a1, double a2, double a3, double b) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (INL) return ip::div4(a0, a1, a2, a3, b);
  else return ip::div4_call(a0, a1, a2, a3, b);
#else
  return {a0 / b, a1 / b, a2 / b, a3 / b};
#endif
}
template <bool INL = false>
PDA_HD float div_rn(float a, float b) { return a / b; }
template <bool INL = false>
PDA_HD float sqrt_rn(float x) { return sqrtf(x); }

// The reference's products by small integers (K x) and by 1/2, products of two
// variables, and its density guard r + 1e-30.  Device code forms the double
// results on the integer pipe (fp64_intpipe.cuh: the IEEE round-to-nearest
// values, bit for bit); host code and single precision use the operators.
template <int K, typename T>
PDA_HD T mul_k(T x) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (sizeof(T) == 8) return ip::mul_small<K>(x);
#endif
  return T(K) * x;
}
template <typename T>
PDA_HD T half_of(T x) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  if constexpr (sizeof(T) == 8) return ip::mul_pow2_neg<1>(x);
#endif
  return T(1. / 2.) * x;
}
// RN(x y) on the integer pipe, out of line
PDA_HD double mul_ip_out(double x, double y) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  return ip::mul_out(x, y);
#else
  return x * y;
#endif
}
PDA_HD double plus_es(double r) {
#if defined(__CUDA_ARCH__) && !defined(PDA_FP64_PIPE_DIVSQRT)
  return ip::add_1em30(r);
#else
  return r + 1.e-30;
#endif
}
// Selectable forms of the above: IP = true forms them on the integer pipe (the
// flux in the face tiles, where that pays); IP = false keeps the FP64 operations
// (row and reduced-order kernels, where the extra integer code measured
// slower).  Both give the same bits.
template <bool IP, typename T>
PDA_HD T halfx(T x) {
  if constexpr (IP) return half_of(x);
  else return T(1. / 2.) * x;
}
template <bool IP>
PDA_HD double mx(double x, double y) {
  if constexpr (IP) return mul_ip_out(x, y);
  else return x * y;
}
template <bool IP>
PDA_HD double sqx(double x) {
  if constexpr (IP) return mul_ip_out(x, x);
  else return x * x;
}
template <bool IP>
PDA_HD double esx(double r) {
  if constexpr (IP) return plus_es(r);
  else return r + 1.e-30;
}


template <typename T> PDA_HD T sq(T x) { return x * x; }

// x / d for a constant d with its reciprocal r = RN(1/d), correctly rounded
// (Markstein's correction step, P. Markstein, IBM J. Res. Dev. 34(1), 1990:
// with r within half an ulp of 1/d and q0 = RN(x r) within one ulp of x/d, the
// remainder x - q0 d is exact in one FMA and RN(q0 + r (x - q0 d)) is the
// correctly rounded quotient).  Three FP64 instructions instead of a full
// division; equal to the division for results in the normal range.
PDA_HD double div_const(double x, double d, double r) {
  const double q0 = x * r;
  const double e = fma(-q0, d, x);
  return fma(e, r, q0);
}

// Single precision, for the approximate (inexact Gauss-Newton) Jacobians of
// the reduced-order model: no exact-rounding constructions are needed there.
PDA_HD float div_const(float x, float, float r) { return x * r; }

// k x + c rounded once, for k a power of two.  k x is then exact (for
// |x| >= 2^-1020, far below any state or gradient value here), so the result
// equals RN(RN(k x) + c), the separately rounded product and sum of the
// reference's source, in one FP64 instruction instead of two.
template <typename T>
PDA_HD T fma_p2(T k, T x, T c) { return fma(k, x, c); }

// The reference's WENO5 stencil expressions (impl/weno5.hpp), evaluated left
// to right as in its source, with the power-of-two products fused:
//   w5_curv(a, m, c)   = a - 2 m + c
//   w5_slopeL(a, m, c) = a - 4 m + 3 c
//   w5_slopeR(a, m, c) = 3 a - 4 m + c
//   w5_pFarL(a, b, c)  = 2 a - 7 b + 11 c     (6 x a candidate polynomial)
//   w5_pMidL(a, b, c)  = -a + 5 b + 2 c
//   w5_pMidR(a, b, c)  = 2 a + 5 b - c
//   w5_pFarR(a, b, c)  = 11 a - 7 b + 2 c
template <typename T>
PDA_HD T w5_curv(T a, T m, T c) { return fma_p2(-T(2.), m, a) + c; }
template <typename T>
PDA_HD T w5_slopeL(T a, T m, T c) { return fma_p2(-T(4.), m, a) + T(3.) * c; }
template <typename T>
PDA_HD T w5_slopeR(T a, T m, T c) { return fma_p2(-T(4.), m, T(3.) * a) + c; }
template <typename T>
PDA_HD T w5_pFarL(T a, T b, T c) { return fma_p2(T(2.), a, -T(7.) * b) + T(11.) * c; }
template <typename T>
PDA_HD T w5_pMidL(T a, T b, T c) { return fma_p2(T(2.), c, -a + T(5.) * b); }
template <typename T>
PDA_HD T w5_pMidR(T a, T b, T c) { return fma_p2(T(2.), a, T(5.) * b) - c; }
template <typename T>
PDA_HD T w5_pFarR(T a, T b, T c) { return fma_p2(T(2.), c, T(11.) * a - T(7.) * b); }

// ---------------------------------------------------------------------------
// WENO5, one face i+1/2: uNeg from q_{i-2..i+2}, uPos from q_{i-1..i+3}.
// ---------------------------------------------------------------------------
// one side of weno5_face: uNeg (left-biased, q_{i-2..i+2})
PDA_HD double weno5_neg(double qim2, double qim1, double qi, double qip1, double qip2) {
  constexpr double epsilon = 1e-6;
  constexpr double two = 2., three = 3., four = 4., five = 5., seven = 7.,
                   eleven = 11.;
  constexpr double oneOvfour = 1. / 4., oneOvsix = 1. / 6.,
                   oneOvten = 1. / 10., threeOvten = 3. / 10.,
                   sixOvten = 6. / 10., thirteenOvtwelve = 13. / 12.;
  double uNeg;
  {
    const double p0 = w5_pFarL(qim2, qim1, qi) * oneOvsix;
    const double p1 = w5_pMidL(qim1, qi, qip1) * oneOvsix;
    const double p2 = w5_pMidR(qi, qip1, qip2) * oneOvsix;
    const double X0 = w5_curv(qim2, qim1, qi), Y0 = w5_slopeL(qim2, qim1, qi);
    const double X1 = w5_curv(qim1, qi, qip1), Y1 = qim1 - qip1;
    const double X2 = w5_curv(qi, qip1, qip2), Y2 = w5_slopeR(qi, qip1, qip2);
    const double B0 = thirteenOvtwelve * X0 * X0 + oneOvfour * Y0 * Y0;
    const double B1 = thirteenOvtwelve * X1 * X1 + oneOvfour * Y1 * Y1;
    const double B2 = thirteenOvtwelve * X2 * X2 + oneOvfour * Y2 * Y2;
    const double alpha0 = div_rn(oneOvten, (epsilon * epsilon + 2. * epsilon * B0 + B0 * B0));
    const double alpha1 = div_rn(sixOvten, (epsilon * epsilon + 2. * epsilon * B1 + B1 * B1));
    const double alpha2 = div_rn(threeOvten, (epsilon * epsilon + 2. * epsilon * B2 + B2 * B2));
    const double alphaSInv = div_rn(1., (alpha0 + alpha1 + alpha2));
    const double w0 = alpha0 * alphaSInv;
    const double w1 = alpha1 * alphaSInv;
    const double w2 = alpha2 * alphaSInv;
    uNeg = w0 * p0 + w1 * p1 + w2 * p2;
  }
  return uNeg;
}

// one side of weno5_face: uPos (right-biased, q_{i-1..i+3})
PDA_HD double weno5_pos(double qim1, double qi, double qip1, double qip2, double qip3) {
  constexpr double epsilon = 1e-6;
  constexpr double two = 2., three = 3., four = 4., five = 5., seven = 7.,
                   eleven = 11.;
  constexpr double oneOvfour = 1. / 4., oneOvsix = 1. / 6.,
                   oneOvten = 1. / 10., threeOvten = 3. / 10.,
                   sixOvten = 6. / 10., thirteenOvtwelve = 13. / 12.;
  double uPos;
  {
    const double p0 = w5_pMidL(qim1, qi, qip1) * oneOvsix;
    const double p1 = w5_pMidR(qi, qip1, qip2) * oneOvsix;
    const double p2 = w5_pFarR(qip1, qip2, qip3) * oneOvsix;
    const double X0 = w5_curv(qim1, qi, qip1), Y0 = w5_slopeL(qim1, qi, qip1);
    const double X1 = w5_curv(qi, qip1, qip2), Y1 = qi - qip2;
    const double X2 = w5_curv(qip1, qip2, qip3), Y2 = w5_slopeR(qip1, qip2, qip3);
    const double B0 = thirteenOvtwelve * X0 * X0 + oneOvfour * Y0 * Y0;
    const double B1 = thirteenOvtwelve * X1 * X1 + oneOvfour * Y1 * Y1;
    const double B2 = thirteenOvtwelve * X2 * X2 + oneOvfour * Y2 * Y2;
    const double alpha0 = div_rn(threeOvten, (epsilon * epsilon + 2. * epsilon * B0 + B0 * B0));
    const double alpha1 = div_rn(sixOvten, (epsilon * epsilon + 2. * epsilon * B1 + B1 * B1));
    const double alpha2 = div_rn(oneOvten, (epsilon * epsilon + 2. * epsilon * B2 + B2 * B2));
    const double alphaSInv = div_rn(1., (alpha0 + alpha1 + alpha2));
    const double w0 = alpha0 * alphaSInv;
    const double w1 = alpha1 * alphaSInv;
    const double w2 = alpha2 * alphaSInv;
    uPos = w0 * p0 + w1 * p1 + w2 * p2;
  }
  return uPos;
}

PDA_HD void weno5_face(double &uNeg, double &uPos, double qim2, double qim1,
                       double qi, double qip1, double qip2, double qip3) {
  uNeg = weno5_neg(qim2, qim1, qi, qip1, qip2);
  uPos = weno5_pos(qim1, qi, qip1, qip2, qip3);
}

// How a product of two variables is formed: on the FP64 pipe, or on the
// integer pipe by a call (the same bits; kernels with enough warps to hide
// its longer chain).
struct FpMul {
  template <typename T> static PDA_HD T mul(T x, T y) { return x * y; }
};
struct IpMul {
  static PDA_HD double mul(double x, double y) { return mul_ip_out(x, y); }
};

// What a gradient routine does with its face value, before the gradient itself:
// nothing, or (row kernels) hand it to the warps that form the flux.
struct NoHandOver {
  template <typename T> PDA_HD void operator()(T) const {}
};

// whether x is infinite or NaN, from its bits on the device
PDA_HD bool not_finite(double x) {
#if defined(__CUDA_ARCH__)
  return ((uint32_t)__double2hiint(x) & 0x7FF00000u) == 0x7FF00000u;
#else
  return !(x - x == 0.);
#endif
}
PDA_HD bool not_finite(float x) { return !(x - x == 0.f); }
PDA_HD bool is_zero(double x) {
#if defined(__CUDA_ARCH__)
  return ((uint32_t)__double2hiint(x) << 1 | (uint32_t)__double2loint(x)) == 0u;
#else
  return x == 0.;
#endif
}
// x^3 from x and p = RN(x^2) for the reference's std::pow(x, 3.) (glibc pow,
// correctly rounded in all but pathological near-midpoint cases).  With Dekker's
// exact two-product, x*x = p + e and p*x = c + ce exactly, so x^3 = c + ce + e*x
// with an error of order 2^-106 before the final rounding; the result is the
// correctly rounded cube except when x^3 lies within that distance of a
// rounding midpoint.  Used only on the Jacobian path.
template <class M>
PDA_HD double cube_of(double x, double p) {
  const double e = fma(x, x, -p);
  const double c = M::mul(p, x);
  const double ce = fma(p, x, -c);
  return c + (ce + M::mul(e, x));
}
template <class M>
PDA_HD float cube_of(float x, float p) { return p * x; }

// One side of the WENO5 face value u and its gradient g[0..4] with respect to
// the side's five cells, from its three candidates: p values, smoothness
// indicators B, linear weights na / 10, and the indicators' derivatives (the
// nine that are not zero, impl/weno5.hpp:294-310, :385-401) in the form
//   dB0 = {d0[0], -2 d0[1], d0[2]}, dB1 = {d1[0], -2 d1[1], d1[2]} (cells 1..3),
//   dB2 = {d2[0], -2 d2[1], d2[2]} (cells 2..4);
// t: the candidates' derivatives, three each.  The reference's sums run over
// all five cells of every candidate; the terms left out here are exact zeros
// (their factors are finite unless an indicator is not, and then its c, hence
// cS below, and so every component is NaN, as there), and a factor of -2 is
// exact, so it joins the next sum: 94 FP64 instructions where the full loops
// take 124.
template <class M, typename T, class Out>
PDA_HD void weno5_side_grad(T &u, T *g, const T p[3], const T B[3], const T na[3], const T d0[3], const T d1[3],
                            const T d2[3], const T t[9], const Out &out) {
  constexpr T epsilon = T(1e-6);
  // (a value handed over comes first; else all six quotients stand together, with fewer values alive: the Jacobian
  // tile's kernel, 512^2, 1863 us so, 2061 the other way)
  constexpr bool early = !std::is_same<Out, NoHandOver>::value;
  T al[3], c[3], e[3], s[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    e[k] = B[k] + epsilon;
    s[k] = M::mul(e[k], e[k]);
    al[k] = div_rn(na[k] / T(10.), s[k]);
    if (!early) c[k] = div_rn(-na[k], T(5.) * cube_of<M>(e[k], s[k]));
  }
  const T aS = div_rn(T(1.), (al[0] + al[1] + al[2]));
  T w0, w1, w2;
  auto value = [&] {
    w0 = M::mul(al[0], aS), w1 = M::mul(al[1], aS), w2 = M::mul(al[2], aS);
    u = M::mul(w0, p[0]) + M::mul(w1, p[1]) + M::mul(w2, p[2]);
    out(u);
  };
  if (early) {
    value();
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = div_rn(-na[k], T(5.) * cube_of<M>(e[k], s[k]));
  }
  const T sr = al[2] + al[1] + al[0];
  T cS = div_rn(-T(1.), M::mul(sr, sr));
  if (sizeof(T) == 8 && (not_finite((double)c[0]) || not_finite((double)c[1]) || not_finite((double)c[2])))
    cS = c[0] + c[1] + c[2] + (c[0] - c[0]) + (c[1] - c[1]) + (c[2] - c[2]);  // NaN
  if (!early) value();
  // da0 = {x0, -2 x1, x2}, da1 = {y0, -2 y1, y2}, da2 = {z0, -2 z1, z2}
  const T x0 = M::mul(c[0], d0[0]), x1 = M::mul(c[0], d0[1]), x2 = M::mul(c[0], d0[2]);
  const T y0 = M::mul(c[1], d1[0]), y1 = M::mul(c[1], d1[1]), y2 = M::mul(c[1], d1[2]);
  const T z0 = M::mul(c[2], d2[0]), z1 = M::mul(c[2], d2[1]), z2 = M::mul(c[2], d2[2]);
  {
    const T S = M::mul(cS, x0);
    T r = M::mul(M::mul(x0, aS) + M::mul(S, al[0]), p[0]) + M::mul(t[0], w0);
    r += M::mul(M::mul(S, al[1]), p[1]);
    r += M::mul(M::mul(S, al[2]), p[2]);
    g[0] = r;
  }
  {
    const T S = M::mul(cS, fma_p2(-T(2.), x1, y0));
    T r = M::mul(fma_p2(-T(2.), M::mul(x1, aS), M::mul(S, al[0])), p[0]) + M::mul(t[1], w0);
    r += M::mul(M::mul(y0, aS) + M::mul(S, al[1]), p[1]) + M::mul(t[3], w1);
    r += M::mul(M::mul(S, al[2]), p[2]);
    g[1] = r;
  }
  {
    const T S = M::mul(cS, fma_p2(-T(2.), y1, x2) + z0);
    T r = M::mul(M::mul(x2, aS) + M::mul(S, al[0]), p[0]) + M::mul(t[2], w0);
    r += M::mul(fma_p2(-T(2.), M::mul(y1, aS), M::mul(S, al[1])), p[1]) + M::mul(t[4], w1);
    r += M::mul(M::mul(z0, aS) + M::mul(S, al[2]), p[2]) + M::mul(t[6], w2);
    g[2] = r;
  }
  {
    const T S = M::mul(cS, fma_p2(-T(2.), z1, y2));
    T r = M::mul(M::mul(S, al[0]), p[0]);
    r += M::mul(M::mul(y2, aS) + M::mul(S, al[1]), p[1]) + M::mul(t[5], w1);
    r += M::mul(fma_p2(-T(2.), M::mul(z1, aS), M::mul(S, al[2])), p[2]) + M::mul(t[7], w2);
    g[3] = r;
  }
  {
    const T S = M::mul(cS, z2);
    T r = M::mul(M::mul(S, al[0]), p[0]);
    r += M::mul(M::mul(S, al[1]), p[1]);
    r += M::mul(M::mul(z2, aS) + M::mul(S, al[2]), p[2]) + M::mul(t[8], w2);
    g[4] = r;
  }
}
// an outer candidate's derivatives from 13 x curvature X and slope Y: Y / 2 +
// X / 6, -2 (Y + X / 6), 3 Y / 2 + X / 6 (RN(X / 3) is 2 RN(X / 6))
template <typename T>
PDA_HD void w5_outer_derivs(T &a, T &b, T &c, T X, T Y) {
  const T D = div_const(X, T(6.), T(1.) / T(6.));
  a = fma_p2(T(0.5), Y, D);
  b = Y + D;
  c = fma_p2(T(0.5), T(3.) * Y, D);
}
// the middle candidate's: Y / 2 + X / 6, -2 X / 6, -Y / 2 + X / 6
template <typename T>
PDA_HD void w5_mid_derivs(T &a, T &b, T &c, T X, T Y) {
  const T D = div_const(X, T(6.), T(1.) / T(6.));
  a = fma_p2(T(0.5), Y, D);
  b = D;
  c = fma_p2(-T(0.5), Y, D);
}
// smoothness indicator from curvature X and slope Y (the quarter of a square is exact)
template <class M, typename T>
PDA_HD T w5_indicator(T X, T Y) {
  return fma_p2(T(1.) / T(4.), M::mul(Y, Y), T(13.) / T(12.) * M::mul(X, X));
}

// WENO5 with the gradient of the two face values with respect to the six
// stencil values q_{i-2..i+3}: gNeg[5] == 0, gPos[0] == 0.
// one side of weno5_face_grad: uNeg and its gradient
template <class M = FpMul, typename T, class Out = NoHandOver>
PDA_HD void weno5_neg_grad(T &uNeg, T gNeg[6], T qim2, T qim1, T qi, T qip1, T qip2, T qip3, const Out &out = Out{}) {
  constexpr T oneOvsix = T(1.) / T(6.);
  const T na[3] = {T(1.), T(6.), T(3.)};
  const T t[9] = {T(1.) / T(3.),  -T(7.) / T(6.), T(11.) / T(6.), -T(1.) / T(6.), T(5.) / T(6.),
                  T(1.) / T(3.),  T(1.) / T(3.),  T(5.) / T(6.),  -T(1.) / T(6.)};
  const T p[3] = {w5_pFarL(qim2, qim1, qi) * oneOvsix, w5_pMidL(qim1, qi, qip1) * oneOvsix,
                  w5_pMidR(qi, qip1, qip2) * oneOvsix};
  const T C0 = w5_curv(qim2, qim1, qi), Y0 = w5_slopeL(qim2, qim1, qi), Y1 = qim1 - qip1;
  const T B[3] = {w5_indicator<M>(C0, Y0), w5_indicator<M>(w5_curv(qim1, qi, qip1), Y1),
                  w5_indicator<M>(w5_curv(qi, qip1, qip2), w5_slopeR(qi, qip1, qip2))};
  T d0[3], d1[3], d2[3];
  w5_outer_derivs(d0[0], d0[1], d0[2], T(13.) * C0, Y0);
  w5_mid_derivs(d1[0], d1[1], d1[2], T(13.) * fma_p2(-T(2.), qi, qip1 + qim1), Y1);
  w5_outer_derivs(d2[2], d2[1], d2[0], T(13.) * w5_curv(qip2, qip1, qi), w5_slopeL(qip2, qip1, qi));
  weno5_side_grad<M>(uNeg, gNeg, p, B, na, d0, d1, d2, t, out);
  gNeg[5] = T(0.);
}

// one side of weno5_face_grad: uPos and its gradient
template <class M = FpMul, typename T, class Out = NoHandOver>
PDA_HD void weno5_pos_grad(T &uPos, T gPos[6], T qim2, T qim1, T qi, T qip1, T qip2, T qip3, const Out &out = Out{}) {
  constexpr T oneOvsix = T(1.) / T(6.);
  const T na[3] = {T(3.), T(6.), T(1.)};
  const T t[9] = {-T(1.) / T(6.), T(5.) / T(6.),  T(1.) / T(3.),  T(1.) / T(3.), T(5.) / T(6.),
                  -T(1.) / T(6.), T(11.) / T(6.), -T(7.) / T(6.), T(1.) / T(3.)};
  const T p[3] = {w5_pMidL(qim1, qi, qip1) * oneOvsix, w5_pMidR(qi, qip1, qip2) * oneOvsix,
                  w5_pFarR(qip1, qip2, qip3) * oneOvsix};
  const T Y1 = qi - qip2;
  const T B[3] = {w5_indicator<M>(w5_curv(qim1, qi, qip1), w5_slopeL(qim1, qi, qip1)),
                  w5_indicator<M>(w5_curv(qi, qip1, qip2), Y1),
                  w5_indicator<M>(w5_curv(qip1, qip2, qip3), w5_slopeR(qip1, qip2, qip3))};
  T d0[3], d1[3], d2[3];
  w5_outer_derivs(d0[0], d0[1], d0[2], T(13.) * fma_p2(-T(2.), qi, qip1 + qim1),
                  fma_p2(-T(4.), qi, T(3.) * qip1 + qim1));
  w5_mid_derivs(d1[0], d1[1], d1[2], T(13.) * w5_curv(qip2, qip1, qi), Y1);
  w5_outer_derivs(d2[2], d2[1], d2[0], T(13.) * w5_curv(qip3, qip2, qip1), w5_slopeL(qip3, qip2, qip1));
  weno5_side_grad<M>(uPos, gPos + 1, p, B, na, d0, d1, d2, t, out);
  gPos[0] = T(0.);
}

PDA_HD void weno5_face_grad(double &uNeg, double &uPos, double gNeg[6],
                            double gPos[6], double qim2, double qim1, double qi,
                            double qip1, double qip2, double qip3) {
  weno5_neg_grad(uNeg, gNeg, qim2, qim1, qi, qip1, qip2, qip3);
  weno5_pos_grad(uPos, gPos, qim2, qim1, qi, qip1, qip2, qip3);
}

// ---------------------------------------------------------------------------
// WENO3, one face i+1/2: uNeg from q_{i-1..i+1}, uPos from q_{i..i+2}.
// ---------------------------------------------------------------------------
// one side of weno3_face: uNeg (q_{i-1..i+1})
PDA_HD double weno3_neg(double qim1, double qi, double qip1) {
  constexpr double epsilon = 1.e-6;
  constexpr double two = 2., three = 3.;
  constexpr double oneOvtwo = 1. / 2., oneOvthree = 1. / 3., twoOvthree = 2. / 3.;
  double uNeg;
  {
    const double p0 = (-qim1 + three * qi) * oneOvtwo;
    const double p1 = (qi + qip1) * oneOvtwo;
    const double B0 = (qim1 - qi) * (qim1 - qi);
    const double B1 = (qi - qip1) * (qi - qip1);
    const double alpha0 = div_rn(oneOvthree, (epsilon * epsilon + two * epsilon * B0 + B0 * B0));
    const double alpha1 = div_rn(twoOvthree, (epsilon * epsilon + two * epsilon * B1 + B1 * B1));
    const double alphaSInv = div_rn(1., (alpha0 + alpha1));
    const double w0 = alpha0 * alphaSInv;
    const double w1 = alpha1 * alphaSInv;
    uNeg = w0 * p0 + w1 * p1;
  }
  return uNeg;
}

// one side of weno3_face: uPos (q_{i..i+2})
PDA_HD double weno3_pos(double qi, double qip1, double qip2) {
  constexpr double epsilon = 1.e-6;
  constexpr double two = 2., three = 3.;
  constexpr double oneOvtwo = 1. / 2., oneOvthree = 1. / 3., twoOvthree = 2. / 3.;
  double uPos;
  {
    const double p0 = (qi + qip1) * oneOvtwo;
    const double p1 = (three * qip1 - qip2) * oneOvtwo;
    const double B0 = (qi - qip1) * (qi - qip1);
    const double B1 = (qip1 - qip2) * (qip1 - qip2);
    const double alpha0 = div_rn(twoOvthree, (epsilon * epsilon + two * epsilon * B0 + B0 * B0));
    const double alpha1 = div_rn(oneOvthree, (epsilon * epsilon + two * epsilon * B1 + B1 * B1));
    const double alphaSInv = div_rn(1., (alpha0 + alpha1));
    const double w0 = alpha0 * alphaSInv;
    const double w1 = alpha1 * alphaSInv;
    uPos = w0 * p0 + w1 * p1;
  }
  return uPos;
}

PDA_HD void weno3_face(double &uNeg, double &uPos, double qim1, double qi,
                       double qip1, double qip2) {
  uNeg = weno3_neg(qim1, qi, qip1);
  uPos = weno3_pos(qi, qip1, qip2);
}

// One side of the WENO3 face value u and its gradient g[0..2] with respect to
// the side's three cells a, b, c.  POS: the right side, whose one-sided
// candidate is the second.  As in weno5_side_grad the terms with a known zero
// are left out (w0 and w1, one of which is in every component, are NaN where a
// zero's factor is not finite), and exact factors of 2, 4 and 8 join the next
// sum: with x = D0 / (3 e0^3) and y = D1 / (3 e1^3) the indicators' derivatives
// are k0 {-x, x, 0} and k1 {0, -y, y}, the weights' sum's k0 s0, 4 s1, -k1 s2.
// 33 FP64 instructions, 31 products and 10 quotients where the full loops take
// 48, 52 and 14.
template <bool POS, class M, typename T, class Out>
PDA_HD void weno3_side_grad(T &u, T *g, T a, T b, T c, const Out &out) {
  constexpr T epsilon = T(1e-6);
  constexpr T third = T(1.) / T(3.), twoThirds = T(2.) / T(3.);
  constexpr T k0 = POS ? T(8.) : T(4.), k1 = POS ? T(4.) : T(8.);
  const T p0 = half_of(POS ? a + b : mul_k<3>(b) - a), p1 = half_of(POS ? mul_k<3>(b) - c : b + c);
  const T D0 = a - b, D1 = b - c;
  const T B0 = M::mul(D0, D0), B1 = M::mul(D1, D1);
  const T a0 = div_rn(POS ? twoThirds : third, epsilon * epsilon + M::mul(T(2.) * epsilon, B0) + M::mul(B0, B0));
  const T a1 = div_rn(POS ? third : twoThirds, epsilon * epsilon + M::mul(T(2.) * epsilon, B1) + M::mul(B1, B1));
  const T aS = div_rn(T(1.), (a0 + a1));
  const T w0 = M::mul(a0, aS), w1 = M::mul(a1, aS);
  u = M::mul(w0, p0) + M::mul(w1, p1);
  out(u);
  const T e0 = B0 + epsilon, e1 = B1 + epsilon;
  const T q0 = M::mul(e0, e0), q1 = M::mul(e1, e1);
  const T A = div_rn(POS ? T(1.) : T(2.), mul_k<3>(q1)) + div_rn(POS ? T(2.) : T(1.), mul_k<3>(q0));
  const T A2 = M::mul(A, A), c0 = mul_k<3>(cube_of<M>(e0, q0)), c1 = cube_of<M>(e1, q1);
  const T x = div_rn(D0, c0), y = div_rn(D1, mul_k<3>(c1));
  const T s0 = div_rn(D0, M::mul(c0, A2)), s2 = div_rn(D1, M::mul(mul_k<3>(A2), c1));
  const T s1 = div_rn(POS ? fma_p2(-T(2.), x, y) : fma_p2(T(2.), y, -x), A2);
  const T xa = M::mul(x, aS), ya = M::mul(y, aS);
  {
    const T r = fma_p2(T(2.) * k0, M::mul(M::mul(s0, a0) - xa, p0), POS ? w0 : -w0);
    g[0] = half_of(fma_p2(T(2.) * k0, M::mul(M::mul(s0, a1), p1), r));
  }
  {
    const T s = M::mul(s1, a0), t = M::mul(s1, a1);
    const T r = fma_p2(T(8.), M::mul(POS ? fma_p2(T(2.), xa, s) : xa + s, p0), POS ? w0 : mul_k<3>(w0));
    g[1] = half_of(r + fma_p2(T(8.), M::mul(POS ? t - ya : fma_p2(-T(2.), ya, t), p1), POS ? mul_k<3>(w1) : w1));
  }
  {
    const T r = fma_p2(T(2.) * k1, M::mul(ya - M::mul(s2, a1), p1), POS ? -w1 : w1);
    g[2] = half_of(fma_p2(-T(2.) * k1, M::mul(M::mul(s2, a0), p0), r));
  }
}

// WENO3 with gradients with respect to q_{i-1..i+2}: gNeg[3] == 0, gPos[0] == 0.
// one side of weno3_face_grad: uNeg and its gradient
template <class M = FpMul, typename T, class Out = NoHandOver>
PDA_HD void weno3_neg_grad(T &uNeg, T gNeg[4], T qim1, T qi, T qip1, T, const Out &out = Out{}) {
  weno3_side_grad<false, M>(uNeg, gNeg, qim1, qi, qip1, out);
  gNeg[3] = T(0.);
}

// one side of weno3_face_grad: uPos and its gradient
template <class M = FpMul, typename T, class Out = NoHandOver>
PDA_HD void weno3_pos_grad(T &uPos, T gPos[4], T, T qi, T qip1, T qip2, const Out &out = Out{}) {
  weno3_side_grad<true, M>(uPos, gPos + 1, qi, qip1, qip2, out);
  gPos[0] = T(0.);
}

PDA_HD void weno3_face_grad(double &uNeg, double &uPos, double gNeg[4],
                            double gPos[4], double qim1, double qi, double qip1,
                            double qip2) {
  weno3_neg_grad(uNeg, gNeg, qim1, qi, qip1, qip2);
  weno3_pos_grad(uPos, gPos, qim1, qi, qip1, qip2);
}

// ---------------------------------------------------------------------------
// Rusanov flux for the Euler equations.  The 2D/3D versions are specialised on
// the face normal (axis-aligned unit vectors); products with 0 and 1 are
// elided, which changes no value other than the sign of an exact zero.
// ---------------------------------------------------------------------------
template <bool INL = false, bool IP = false>
PDA_HD void euler3_flux(double F[3], const double qL[3], const double qR[3],
                        double gamma) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double rL = qL[0];
  const double uL = div_rn<INL>(qL[1], esx<IP>(rL));
  const double pL = mx<IP>(gamma - 1, qL[2] - mx<IP>(halfx<IP>(rL), sqx<IP>(uL)));
  const Quot2 hl = div2_rn<INL>((qL[2] + pL), qR[0], rL);  // HL and rR / rL
  const double HL = hl.q0;
  const double FL0 = mx<IP>(rL, uL), FL1 = mx<IP>(FL0, uL) + pL, FL2 = mx<IP>(FL0, HL);
  const double rR = qR[0];
  const double uR = div_rn<INL>(qR[1], esx<IP>(rR));
  const double pR = mx<IP>(gamma - 1, qR[2] - mx<IP>(halfx<IP>(rR), sqx<IP>(uR)));
  const double HR = div_rn<INL>((qR[2] + pR), rR);
  const double FR0 = mx<IP>(rR, uR), FR1 = mx<IP>(FR0, uR) + pR, FR2 = mx<IP>(FR0, HR);
  const double RT = sqrt_rn<INL>(hl.q1);
  const Quot2 roe = div2_rn<INL>((uL + mx<IP>(RT, uR)), (HL + mx<IP>(RT, HR)), (1. + RT));
  const double u = roe.q0, H = roe.q1;
  const double a = sqrt_rn<INL>(mx<IP>(gamma - 1., H - halfx<IP>(sqx<IP>(u))));
  const double smax = fabs(u) + a;
  F[0] = halfx<IP>(FL0 + FR0 + mx<IP>(smax, qL[0] - qR[0]));
  F[1] = halfx<IP>(FL1 + FR1 + mx<IP>(smax, qL[1] - qR[1]));
  F[2] = halfx<IP>(FL2 + FR2 + mx<IP>(smax, qL[2] - qR[2]));
}

template <int AXIS, bool INL = false, bool IP = false>
PDA_HD void euler4_flux(double F[4], const double qL[4], const double qR[4],
                        double gamma) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double rL = qL[0];
  const Quot2 vl = div2_rn<INL>(qL[1], qL[2], esx<IP>(rL));
  const double uL = vl.q0, vL = vl.q1;
  const double unL = AXIS == 0 ? uL : vL;
  const double pL = mx<IP>(gamma - 1, qL[3] - mx<IP>(halfx<IP>(rL), sqx<IP>(uL) + sqx<IP>(vL)));
  const Quot2 hl = div2_rn<INL>((qL[3] + pL), qR[0], rL);  // HL and rR / rL
  const double HL = hl.q0;
  double FL[4];
  FL[0] = mx<IP>(rL, unL);
  FL[1] = AXIS == 0 ? mx<IP>(FL[0], uL) + pL : mx<IP>(FL[0], uL);
  FL[2] = AXIS == 1 ? mx<IP>(FL[0], vL) + pL : mx<IP>(FL[0], vL);
  FL[3] = mx<IP>(FL[0], HL);
  const double rR = qR[0];
  const Quot2 vr = div2_rn<INL>(qR[1], qR[2], esx<IP>(rR));
  const double uR = vr.q0, vR = vr.q1;
  const double unR = AXIS == 0 ? uR : vR;
  const double pR = mx<IP>(gamma - 1, qR[3] - mx<IP>(halfx<IP>(rR), sqx<IP>(uR) + sqx<IP>(vR)));
  const double HR = div_rn<INL>((qR[3] + pR), rR);
  double FR[4];
  FR[0] = mx<IP>(rR, unR);
  FR[1] = AXIS == 0 ? mx<IP>(FR[0], uR) + pR : mx<IP>(FR[0], uR);
  FR[2] = AXIS == 1 ? mx<IP>(FR[0], vR) + pR : mx<IP>(FR[0], vR);
  FR[3] = mx<IP>(FR[0], HR);
  const double RT = sqrt_rn<INL>(hl.q1);
  const Quot3 roe = div3_rn<INL>((uL + mx<IP>(RT, uR)), (vL + mx<IP>(RT, vR)), (HL + mx<IP>(RT, HR)), (1. + RT));
  const double u = roe.q0, v = roe.q1, H = roe.q2;
  const double uu = sqx<IP>(u) + sqx<IP>(v);
  const double a = sqrt_rn<INL>(mx<IP>(gamma - 1., H - halfx<IP>(uu)));
  const double smax = sqrt_rn<INL>(uu) + a;
#pragma unroll
  for (int d = 0; d < 4; ++d) F[d] = halfx<IP>(FL[d] + FR[d] + mx<IP>(smax, qL[d] - qR[d]));
}

template <int AXIS, bool INL = false, bool IP = false>
PDA_HD void euler5_flux(double F[5], const double qL[5], const double qR[5],
                        double gamma) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double rL = qL[0];
  const Quot3 vl = div3_rn<INL>(qL[1], qL[2], qL[3], esx<IP>(rL));
  const double uL = vl.q0, vL = vl.q1, wL = vl.q2;
  const double unL = AXIS == 0 ? uL : (AXIS == 1 ? vL : wL);
  const double pL = mx<IP>(gamma - 1, qL[4] - mx<IP>(halfx<IP>(rL), sqx<IP>(uL) + sqx<IP>(vL) + sqx<IP>(wL)));
  const Quot2 hl = div2_rn<INL>((qL[4] + pL), qR[0], rL);  // HL and rR / rL
  const double HL = hl.q0;
  double FL[5];
  FL[0] = mx<IP>(rL, unL);
  FL[1] = AXIS == 0 ? mx<IP>(FL[0], uL) + pL : mx<IP>(FL[0], uL);
  FL[2] = AXIS == 1 ? mx<IP>(FL[0], vL) + pL : mx<IP>(FL[0], vL);
  FL[3] = AXIS == 2 ? mx<IP>(FL[0], wL) + pL : mx<IP>(FL[0], wL);
  FL[4] = mx<IP>(FL[0], HL);
  const double rR = qR[0];
  const Quot3 vr = div3_rn<INL>(qR[1], qR[2], qR[3], esx<IP>(rR));
  const double uR = vr.q0, vR = vr.q1, wR = vr.q2;
  const double unR = AXIS == 0 ? uR : (AXIS == 1 ? vR : wR);
  const double pR = mx<IP>(gamma - 1, qR[4] - mx<IP>(halfx<IP>(rR), sqx<IP>(uR) + sqx<IP>(vR) + sqx<IP>(wR)));
  const double HR = div_rn<INL>((qR[4] + pR), rR);
  double FR[5];
  FR[0] = mx<IP>(rR, unR);
  FR[1] = AXIS == 0 ? mx<IP>(FR[0], uR) + pR : mx<IP>(FR[0], uR);
  FR[2] = AXIS == 1 ? mx<IP>(FR[0], vR) + pR : mx<IP>(FR[0], vR);
  FR[3] = AXIS == 2 ? mx<IP>(FR[0], wR) + pR : mx<IP>(FR[0], wR);
  FR[4] = mx<IP>(FR[0], HR);
  const double RT = sqrt_rn<INL>(hl.q1);
  const Quot4 roe = div4_rn<INL>((uL + mx<IP>(RT, uR)), (vL + mx<IP>(RT, vR)), (wL + mx<IP>(RT, wR)), (HL + mx<IP>(RT, HR)), (1. + RT));
  const double u = roe.q0, v = roe.q1, w = roe.q2, H = roe.q3;
  const double uu = sqx<IP>(u) + sqx<IP>(v) + sqx<IP>(w);
  const double a = sqrt_rn<INL>(mx<IP>(gamma - 1., H - halfx<IP>(uu)));
  const double smax = sqrt_rn<INL>(uu) + a;
#pragma unroll
  for (int d = 0; d < 5; ++d) F[d] = halfx<IP>(FL[d] + FR[d] + mx<IP>(smax, qL[d] - qR[d]));
}

// RN(sqrt(RN(x^2))): |x| itself where the square neither overflows nor
// underflows (radix 2: S. Boldo, "Stupid is as stupid does", NSV 2015), checked
// by the integer pipe's operand window; a zero too.
template <bool INL = false, bool IP = false>
PDA_HD double root_of_square(double x) {
#if defined(__CUDA_ARCH__)
  if (ip::in_window(x) || is_zero(x)) return fabs(x);
#endif
  return sqrt_rn<INL>(sqx<IP>(x));
}
// Quotients with a dividend that is zero in whole regions (water at rest),
// which the integer pipe's division would leave to its far, slow exit
template <bool INL = false>
PDA_HD double div_or_zero(double a, double b) {
#if defined(__CUDA_ARCH__)
  if (is_zero(a) && ip::in_window(b) && __double2hiint(b) >= 0) return a;
#endif
  return div_rn<INL>(a, b);
}
template <bool INL = false>
PDA_HD Quot2 div2_or_zero(double a0, double a1, double b) {
#if defined(__CUDA_ARCH__)
  if (is_zero(a0) && is_zero(a1) && ip::in_window(b) && __double2hiint(b) >= 0) return {a0, a1};
#endif
  return div2_rn<INL>(a0, a1, b);
}

// Shallow-water Rusanov flux.  deviation: the reference's std::pow(h, 0.5) is
// evaluated as sqrt(h) (correctly rounded; glibc pow agrees except in rare
// near-midpoint cases, a 1-ulp difference).
template <int AXIS, bool INL = false, bool IP = false>
PDA_HD void swe_flux(double F[3], const double qL[3], const double qR[3],
                     double gravity) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double hL = qL[0];
  const Quot2 vl = div2_or_zero<INL>(qL[1], qL[2], esx<IP>(hL));
  const double uL = vl.q0, vL = vl.q1;
  const double unL = AXIS == 0 ? uL : vL;
  const double pL = mx<IP>(mx<IP>(halfx<IP>(gravity), hL), hL);
  double FL[3];
  FL[0] = mx<IP>(hL, unL);
  FL[1] = AXIS == 0 ? mx<IP>(FL[0], uL) + pL : mx<IP>(FL[0], uL);
  FL[2] = AXIS == 1 ? mx<IP>(FL[0], vL) + pL : mx<IP>(FL[0], vL);
  const double hR = qR[0];
  const Quot2 vr = div2_or_zero<INL>(qR[1], qR[2], esx<IP>(hR));
  const double uR = vr.q0, vR = vr.q1;
  const double unR = AXIS == 0 ? uR : vR;
  const double pR = mx<IP>(mx<IP>(halfx<IP>(gravity), hR), hR);
  double FR[3];
  FR[0] = mx<IP>(hR, unR);
  FR[1] = AXIS == 0 ? mx<IP>(FR[0], uR) + pR : mx<IP>(FR[0], uR);
  FR[2] = AXIS == 1 ? mx<IP>(FR[0], vR) + pR : mx<IP>(FR[0], vR);
  const double hm = halfx<IP>(hL + hR);
  const double sL = sqrt_rn<INL>(hL), sR = sqrt_rn<INL>(hR);
  const double um = div_or_zero<INL>((mx<IP>(unL, sL) + mx<IP>(unR, sR)), esx<IP>(sL + sR));
  const double sg = sqrt_rn<INL>(mx<IP>(gravity, hm));
  const double smax = root_of_square<INL, IP>(um) + root_of_square<INL, IP>(sg);
#pragma unroll
  for (int d = 0; d < 3; ++d) F[d] = halfx<IP>(FL[d] + FR[d] + mx<IP>(smax, qL[d] - qR[d]));
}

// ---------------------------------------------------------------------------
// The Rusanov fluxes above in two halves: flux_side (the quantities of one
// face state: its velocities, enthalpy or sqrt(h), and physical flux) and
// flux_combine (the Roe / wave-speed average and the Rusanov sum).  The side
// takes the face normal as a runtime axis (*_side_ax; the templated form
// passes its constant), so threads of one warp that hold faces of different
// axes run one instruction stream; the combination does not depend on the
// axis at all.
// combine(side(qL), side(qR)) evaluates every expression of the *_flux
// function above unchanged, so it is bit-identical; the halves let a kernel
// compute the two states of a face on different warps.
// ---------------------------------------------------------------------------
template <int N> struct FluxSide {
  double F[N];  // the state's physical flux along the axis
  double u, v, w, H;  // Euler: velocities and total enthalpy; shallow water: u = normal velocity, H = sqrt(h)
};

PDA_HD void euler3_side(FluxSide<3> &o, const double q[3], double gamma) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double r = q[0];
  const double u = div_rn(q[1], (r + es));
  const double p = (gamma - 1) * (q[2] - half * r * (u * u));
  const double H = div_rn((q[2] + p), r);
  o.F[0] = r * u;
  o.F[1] = r * u * u + p;
  o.F[2] = r * u * H;
  o.u = u;
  o.H = H;
}
PDA_HD void euler3_combine(double F[3], const double qL[3], const double qR[3], const FluxSide<3> &L,
                           const FluxSide<3> &R, double gamma) {
  constexpr double half = 1. / 2.;
  const double RT = sqrt_rn(div_rn(qR[0], (qL[0])));
  const double u = div_rn((L.u + RT * R.u), (1. + RT));
  const double H = div_rn((L.H + RT * R.H), (1. + RT));
  const double a = sqrt_rn((gamma - 1.) * (H - half * (u * u)));
  const double smax = fabs(u) + a;
#pragma unroll
  for (int d = 0; d < 3; ++d) F[d] = half * (L.F[d] + R.F[d] + smax * (qL[d] - qR[d]));
}

PDA_HD void euler4_side_ax(FluxSide<4> &o, const double q[4], double gamma, int ax) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double r = q[0];
  const double u = div_rn(q[1], (r + es));
  const double v = div_rn(q[2], (r + es));
  const double un = ax == 0 ? u : v;
  const double p = (gamma - 1) * (q[3] - half * r * (u * u + v * v));
  const double H = div_rn((q[3] + p), r);
  o.F[0] = r * un;
  o.F[1] = ax == 0 ? r * un * u + p : r * un * u;
  o.F[2] = ax == 1 ? r * un * v + p : r * un * v;
  o.F[3] = r * un * H;
  o.u = u;
  o.v = v;
  o.H = H;
}
template <int AXIS>
PDA_HD void euler4_side(FluxSide<4> &o, const double q[4], double gamma) {
  euler4_side_ax(o, q, gamma, AXIS);
}
template <int AXIS>
PDA_HD void euler4_combine(double F[4], const double qL[4], const double qR[4], const FluxSide<4> &L,
                           const FluxSide<4> &R, double gamma) {
  constexpr double half = 1. / 2.;
  const double RT = sqrt_rn(div_rn(qR[0], (qL[0])));
  const double u = div_rn((L.u + RT * R.u), (1. + RT));
  const double v = div_rn((L.v + RT * R.v), (1. + RT));
  const double H = div_rn((L.H + RT * R.H), (1. + RT));
  const double a = sqrt_rn((gamma - 1.) * (H - half * (u * u + v * v)));
  const double smax = sqrt_rn(u * u + v * v) + a;
#pragma unroll
  for (int d = 0; d < 4; ++d) F[d] = half * (L.F[d] + R.F[d] + smax * (qL[d] - qR[d]));
}

PDA_HD void euler5_side_ax(FluxSide<5> &o, const double q[5], double gamma, int ax) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double r = q[0];
  const double u = div_rn(q[1], (r + es));
  const double v = div_rn(q[2], (r + es));
  const double w = div_rn(q[3], (r + es));
  const double un = ax == 0 ? u : (ax == 1 ? v : w);
  const double p = (gamma - 1) * (q[4] - half * r * (u * u + v * v + w * w));
  const double H = div_rn((q[4] + p), r);
  o.F[0] = r * un;
  o.F[1] = ax == 0 ? r * un * u + p : r * un * u;
  o.F[2] = ax == 1 ? r * un * v + p : r * un * v;
  o.F[3] = ax == 2 ? r * un * w + p : r * un * w;
  o.F[4] = r * un * H;
  o.u = u;
  o.v = v;
  o.w = w;
  o.H = H;
}
template <int AXIS>
PDA_HD void euler5_side(FluxSide<5> &o, const double q[5], double gamma) {
  euler5_side_ax(o, q, gamma, AXIS);
}
template <int AXIS>
PDA_HD void euler5_combine(double F[5], const double qL[5], const double qR[5], const FluxSide<5> &L,
                           const FluxSide<5> &R, double gamma) {
  constexpr double half = 1. / 2.;
  const double RT = sqrt_rn(div_rn(qR[0], (qL[0])));
  const double u = div_rn((L.u + RT * R.u), (1. + RT));
  const double v = div_rn((L.v + RT * R.v), (1. + RT));
  const double w = div_rn((L.w + RT * R.w), (1. + RT));
  const double H = div_rn((L.H + RT * R.H), (1. + RT));
  const double a = sqrt_rn((gamma - 1.) * (H - half * (u * u + v * v + w * w)));
  const double smax = sqrt_rn(u * u + v * v + w * w) + a;
#pragma unroll
  for (int d = 0; d < 5; ++d) F[d] = half * (L.F[d] + R.F[d] + smax * (qL[d] - qR[d]));
}

PDA_HD void swe_side_ax(FluxSide<3> &o, const double q[3], double gravity, int ax) {
  constexpr double es = 1.e-30;
  const double h = q[0];
  const Quot2 uv = div2_or_zero(q[1], q[2], h + es);
  const double u = uv.q0, v = uv.q1;
  const double un = ax == 0 ? u : v;
  const double p = 0.5 * gravity * h * h;
  o.F[0] = h * un;
  o.F[1] = ax == 0 ? h * un * u + p : h * un * u;
  o.F[2] = ax == 1 ? h * un * v + p : h * un * v;
  o.u = un;
  o.H = sqrt_rn(h);
}
template <int AXIS>
PDA_HD void swe_side(FluxSide<3> &o, const double q[3], double gravity) {
  swe_side_ax(o, q, gravity, AXIS);
}
template <int AXIS>
PDA_HD void swe_combine(double F[3], const double qL[3], const double qR[3], const FluxSide<3> &L,
                        const FluxSide<3> &R, double gravity) {
  constexpr double half = 1. / 2.;
  constexpr double es = 1.e-30;
  const double hm = 0.5 * (qL[0] + qR[0]);
  const double um = div_or_zero((L.u * L.H + R.u * R.H), (L.H + R.H + es));
  const double sg = sqrt_rn(gravity * hm);
  const double smax = root_of_square(um) + root_of_square(sg);
#pragma unroll
  for (int d = 0; d < 3; ++d) F[d] = half * (L.F[d] + R.F[d] + smax * (qL[d] - qR[d]));
}

// ---------------------------------------------------------------------------
// Analytic Rusanov flux Jacobians JL = dF/dqL, JR = dF/dqR (row-major n x n).
// These keep the reference's generic normal vector n, built from a runtime
// axis (*_flux_jac_ax; the templated form passes its constant), so threads
// of one warp that hold faces of different axes run one instruction stream.
// ---------------------------------------------------------------------------
template <typename T>
PDA_HD void euler3_flux_jac(T JL[9], T JR[9], const T qL[3],
                            const T qR[3], T gamma) {
  constexpr T one = T(1.), two = T(2.), three = T(3.), half = T(1.) / T(2.);
  constexpr T es = T(1.e-30);
  const T gm1 = gamma - one;
  const T rL = qL[0];
  const T uL = div_rn(qL[1], (rL + es));
  const T pL = gm1 * (qL[2] - half * rL * (uL * uL));
  const T HL = div_rn((qL[2] + pL), rL);
  const T aL = sqrt_rn(gm1 * (HL - half * (uL * uL)));
  const T rR = qR[0];
  const T uR = div_rn(qR[1], (rR + es));
  const T pR = gm1 * (qR[2] - half * rR * (uR * uR));
  const T HR = div_rn((qR[2] + pR), rR);
  const T aR = sqrt_rn(gm1 * (HR - half * (uR * uR)));
  const T r = sqrt_rn(rR * rL);
  const T RT = sqrt_rn(div_rn(rR, (rL)));
  const T u = div_rn((uL + RT * uR), (one + RT));
  const T H = div_rn((HL + RT * HR), (one + RT));
  const T a = sqrt_rn(gm1 * (H - half * (u * u)));
  const T smax = fabs(u) + a;
  const T VMagSqrRoe = u * u + es;
  const T VMagSqrL = uL * uL;
  const T VVRoeL = uL * u;
  const T VMagSqrR = uR * uR;
  const T VVRoeR = uR * u;
  const T uRelRoe = div_rn(u, sqrt_rn(VMagSqrRoe));
  T gL[3], gR[3];
  gL[0] = div_rn(one, (rL + r)) * (-half * (uL + u) * uRelRoe + div_rn(half * gm1, a) * (fma_p2(half, VMagSqrRoe + VVRoeL, half * (HL - H)) - div_rn(aL * aL, gm1) + half * (gamma - two) * VMagSqrL));
  gL[1] = div_rn(one, (rL + r)) * (uRelRoe - div_rn(half * (gm1 * (u + gm1 * uL)), (a)));
  gL[2] = div_rn(div_rn(half, (rL + r)) * gamma * gm1, (a));
  gR[0] = div_rn(one, (rR + r)) * (-half * (uR + u) * uRelRoe + div_rn(half * gm1, a) * (fma_p2(half, VMagSqrRoe + VVRoeR, half * (HR - H)) - div_rn(aR * aR, gm1) + half * (gamma - two) * VMagSqrR));
  gR[1] = div_rn(one, (rR + r)) * (uRelRoe - div_rn(half * (gm1 * (u + gm1 * uR)), (a)));
  gR[2] = div_rn(div_rn(half, (rR + r)) * gamma * gm1, (a));
  JL[0] = 0;
  JL[1] = half;
  JL[2] = 0;
  JL[3] = half * (half * gm1 * uL * uL - uL * uL);
  JL[4] = half * ((three - gamma) * uL);
  JL[5] = half * gm1;
  JL[6] = half * ((half * gm1 * uL * uL - HL) * uL);
  JL[7] = half * (HL - gm1 * uL * uL);
  JL[8] = half * gamma * uL;
  for (int i = 0; i < 3; i++) {
    JL[i * 3 + i] = fma_p2(half, smax, JL[i * 3 + i]);
    for (int j = 0; j < 3; j++) JL[i * 3 + j] += half * gL[j] * (qL[i] - qR[i]);
  }
  JR[0] = 0;
  JR[1] = half;
  JR[2] = 0;
  JR[3] = half * (half * gm1 * uR * uR - uR * uR);
  JR[4] = half * ((three - gamma) * uR);
  JR[5] = half * gm1;
  JR[6] = half * ((half * gm1 * uR * uR - HR) * uR);
  JR[7] = half * (HR - gm1 * uR * uR);
  JR[8] = half * gamma * uR;
  for (int i = 0; i < 3; i++) {
    JR[i * 3 + i] = fma_p2(-half, smax, JR[i * 3 + i]);
    for (int j = 0; j < 3; j++) JR[i * 3 + j] += half * gR[j] * (qL[i] - qR[i]);
  }
}

template <typename T>
PDA_HD void euler4_flux_jac_ax(T JL[16], T JR[16], const T qL[4],
                            const T qR[4], T gamma, int ax) {
  constexpr T one = T(1.), two = T(2.), half = T(1.) / T(2.);
  constexpr T es = T(1.e-30);
  const T n[2] = {ax == 0 ? T(1.) : T(0.), ax == 1 ? T(1.) : T(0.)};
  const T gm1 = gamma - one;
  const T rL = qL[0];
  const T uL = div_rn(qL[1], (rL + es));
  const T vL = div_rn(qL[2], (rL + es));
  const T unL = uL * n[0] + vL * n[1];
  const T pL = gm1 * (qL[3] - half * rL * (uL * uL + vL * vL));
  const T HL = div_rn((qL[3] + pL), rL);
  const T aL = sqrt_rn(gm1 * (HL - half * (uL * uL + vL * vL)));
  const T rR = qR[0];
  const T uR = div_rn(qR[1], (rR + es));
  const T vR = div_rn(qR[2], (rR + es));
  const T unR = uR * n[0] + vR * n[1];
  const T pR = gm1 * (qR[3] - half * rR * (uR * uR + vR * vR));
  const T HR = div_rn((qR[3] + pR), rR);
  const T aR = sqrt_rn(gm1 * (HR - half * (uR * uR + vR * vR)));
  const T r = sqrt_rn(rR * rL);
  const T RT = sqrt_rn(div_rn(rR, (rL)));
  const T u = div_rn((uL + RT * uR), (one + RT));
  const T v = div_rn((vL + RT * vR), (one + RT));
  const T H = div_rn((HL + RT * HR), (one + RT));
  const T a = sqrt_rn(gm1 * (H - half * (u * u + v * v)));
  const T smax = sqrt_rn(u * u + v * v) + a;
  const T VMagSqrRoe = u * u + v * v + es;
  const T VMagSqrL = uL * uL + vL * vL;
  const T VVRoeL = uL * u + vL * v;
  const T VMagSqrR = uR * uR + vR * vR;
  const T VVRoeR = uR * u + vR * v;
  const T uRelRoe = div_rn(u, sqrt_rn(VMagSqrRoe));
  const T vRelRoe = div_rn(v, sqrt_rn(VMagSqrRoe));
  T gL[4], gR[4];
  gL[0] = div_rn(one, (rL + r)) * (-half * (uL + u) * uRelRoe - half * (vL + v) * vRelRoe + div_rn(half * gm1, a) * (fma_p2(half, VMagSqrRoe + VVRoeL, half * (HL - H)) - div_rn(aL * aL, gm1) + half * (gamma - two) * VMagSqrL));
  gL[1] = div_rn(one, (rL + r)) * (uRelRoe - div_rn(half * (gm1 * (u + gm1 * uL)), (a)));
  gL[2] = div_rn(one, (rL + r)) * (vRelRoe - div_rn(half * (gm1 * (v + gm1 * vL)), (a)));
  gL[3] = div_rn(div_rn(half, (rL + r)) * gamma * gm1, (a));
  gR[0] = div_rn(one, (rR + r)) * (-half * (uR + u) * uRelRoe - half * (vR + v) * vRelRoe + div_rn(half * gm1, a) * (fma_p2(half, VMagSqrRoe + VVRoeR, half * (HR - H)) - div_rn(aR * aR, gm1) + half * (gamma - two) * VMagSqrR));
  gR[1] = div_rn(one, (rR + r)) * (uRelRoe - div_rn(half * (gm1 * (u + gm1 * uR)), (a)));
  gR[2] = div_rn(one, (rR + r)) * (vRelRoe - div_rn(half * (gm1 * (v + gm1 * vR)), (a)));
  gR[3] = div_rn(div_rn(half, (rR + r)) * gamma * gm1, (a));
  // left
  JL[0] = 0;
  JL[1] = half * n[0];
  JL[2] = half * n[1];
  JL[3] = 0;
  JL[4] = half * (half * gm1 * VMagSqrL * n[0] - uL * unL);
  JL[5] = half * (uL * n[0] - gm1 * uL * n[0] + unL);
  JL[6] = half * (uL * n[1] - gm1 * vL * n[0]);
  JL[7] = half * gm1 * n[0];
  JL[8] = half * (half * gm1 * VMagSqrL * n[1] - vL * unL);
  JL[9] = half * (vL * n[0] - gm1 * uL * n[1]);
  JL[10] = half * (vL * n[1] - gm1 * vL * n[1] + unL);
  JL[11] = half * gm1 * n[1];
  JL[12] = half * ((half * gm1 * VMagSqrL - HL) * unL);
  JL[13] = half * (HL * n[0] - gm1 * uL * unL);
  JL[14] = half * (HL * n[1] - gm1 * vL * unL);
  JL[15] = half * gamma * unL;
  for (int i = 0; i < 4; i++) {
    JL[i * 4 + i] = fma_p2(half, smax, JL[i * 4 + i]);
    for (int j = 0; j < 4; j++) JL[i * 4 + j] += half * gL[j] * (qL[i] - qR[i]);
  }
  // right
  JR[0] = 0;
  JR[1] = half * n[0];
  JR[2] = half * n[1];
  JR[3] = 0;
  JR[4] = half * (half * gm1 * VMagSqrR * n[0] - uR * unR);
  JR[5] = half * (uR * n[0] - gm1 * uR * n[0] + unR);
  JR[6] = half * (uR * n[1] - gm1 * vR * n[0]);
  JR[7] = half * gm1 * n[0];
  JR[8] = half * (half * gm1 * VMagSqrR * n[1] - vR * unR);
  JR[9] = half * (vR * n[0] - gm1 * uR * n[1]);
  JR[10] = half * (vR * n[1] - gm1 * vR * n[1] + unR);
  JR[11] = half * gm1 * n[1];
  JR[12] = half * ((half * gm1 * VMagSqrR - HR) * unR);
  JR[13] = half * (HR * n[0] - gm1 * uR * unR);
  JR[14] = half * (HR * n[1] - gm1 * vR * unR);
  JR[15] = half * gamma * unR;
  for (int i = 0; i < 4; i++) {
    JR[i * 4 + i] = fma_p2(-half, smax, JR[i * 4 + i]);
    for (int j = 0; j < 4; j++) JR[i * 4 + j] += half * gR[j] * (qL[i] - qR[i]);
  }
}
template <int AXIS, typename T>
PDA_HD void euler4_flux_jac(T JL[16], T JR[16], const T qL[4],
                            const T qR[4], T gamma) {
  euler4_flux_jac_ax(JL, JR, qL, qR, gamma, AXIS);
}

template <typename T>
PDA_HD void euler5_flux_jac_ax(T JL[25], T JR[25], const T qL[5],
                            const T qR[5], T gamma, int ax) {
  constexpr T one = T(1.), two = T(2.), half = T(1.) / T(2.);
  constexpr T es = T(1.e-30);
  const T n[3] = {ax == 0 ? T(1.) : T(0.), ax == 1 ? T(1.) : T(0.), ax == 2 ? T(1.) : T(0.)};
  const T gm1 = gamma - one;
  const T rL = qL[0];
  const T uL = div_rn(qL[1], (rL + es));
  const T vL = div_rn(qL[2], (rL + es));
  const T wL = div_rn(qL[3], (rL + es));
  const T unL = uL * n[0] + vL * n[1] + wL * n[2];
  const T pL = gm1 * (qL[4] - half * rL * (uL * uL + vL * vL + wL * wL));
  const T HL = div_rn((qL[4] + pL), rL);
  const T aL = sqrt_rn(gm1 * (HL - half * (uL * uL + vL * vL + wL * wL)));
  const T rR = qR[0];
  const T uR = div_rn(qR[1], (rR + es));
  const T vR = div_rn(qR[2], (rR + es));
  const T wR = div_rn(qR[3], (rR + es));
  const T unR = uR * n[0] + vR * n[1] + wR * n[2];
  const T pR = gm1 * (qR[4] - half * rR * (uR * uR + vR * vR + wR * wR));
  const T HR = div_rn((qR[4] + pR), rR);
  const T aR = sqrt_rn(gm1 * (HR - half * (uR * uR + vR * vR + wR * wR)));
  const T r = sqrt_rn(rR * rL);
  const T RT = sqrt_rn(div_rn(rR, (rL)));
  const T u = div_rn((uL + RT * uR), (one + RT));
  const T v = div_rn((vL + RT * vR), (one + RT));
  const T w = div_rn((wL + RT * wR), (one + RT));
  const T H = div_rn((HL + RT * HR), (one + RT));
  const T a = sqrt_rn(gm1 * (H - half * (u * u + v * v + w * w)));
  const T smax = sqrt_rn(u * u + v * v + w * w) + a;
  const T VMagSqrRoe = u * u + v * v + w * w + es;
  const T VMagSqrL = uL * uL + vL * vL + wL * wL;
  const T VVRoeL = uL * u + vL * v + wL * w;
  const T VMagSqrR = uR * uR + vR * vR + wR * wR;
  const T VVRoeR = uR * u + vR * v + wR * w;
  const T uRelRoe = div_rn(u, sqrt_rn(VMagSqrRoe));
  const T vRelRoe = div_rn(v, sqrt_rn(VMagSqrRoe));
  const T wRelRoe = div_rn(w, sqrt_rn(VMagSqrRoe));
  T gL[5], gR[5];
  gL[0] = div_rn(one, (rL + r)) * (-half * (uL + u) * uRelRoe - half * (vL + v) * vRelRoe - half * (wL + w) * wRelRoe + div_rn(half * gm1, a) * (fma_p2(half, VMagSqrRoe + VVRoeL, half * (HL - H)) - div_rn(aL * aL, gm1) + half * (gamma - two) * VMagSqrL));
  gL[1] = div_rn(one, (rL + r)) * (uRelRoe - div_rn(half * (gm1 * (u + gm1 * uL)), (a)));
  gL[2] = div_rn(one, (rL + r)) * (vRelRoe - div_rn(half * (gm1 * (v + gm1 * vL)), (a)));
  gL[3] = div_rn(one, (rL + r)) * (wRelRoe - div_rn(half * (gm1 * (w + gm1 * wL)), (a)));
  gL[4] = div_rn(div_rn(half, (rL + r)) * gamma * gm1, (a));
  gR[0] = div_rn(one, (rR + r)) * (-half * (uR + u) * uRelRoe - half * (vR + v) * vRelRoe - half * (wR + w) * wRelRoe + div_rn(half * gm1, a) * (fma_p2(half, VMagSqrRoe + VVRoeR, half * (HR - H)) - div_rn(aR * aR, gm1) + half * (gamma - two) * VMagSqrR));
  gR[1] = div_rn(one, (rR + r)) * (uRelRoe - div_rn(half * (gm1 * (u + gm1 * uR)), (a)));
  gR[2] = div_rn(one, (rR + r)) * (vRelRoe - div_rn(half * (gm1 * (v + gm1 * vR)), (a)));
  gR[3] = div_rn(one, (rR + r)) * (wRelRoe - div_rn(half * (gm1 * (w + gm1 * wR)), (a)));
  gR[4] = div_rn(div_rn(half, (rR + r)) * gamma * gm1, (a));
  // left and right use the same template; X = L or R
#define PDA_FILL_J5(J, uX, vX, wX, unX, HX, VMagSqrX)                 \
  J[0] = 0;                                                           \
  J[1] = half * n[0];                                                 \
  J[2] = half * n[1];                                                 \
  J[3] = half * n[2];                                                 \
  J[4] = 0;                                                           \
  J[5] = half * (half * gm1 * VMagSqrX * n[0] - uX * unX);            \
  J[6] = half * (uX * n[0] - gm1 * uX * n[0] + unX);                  \
  J[7] = half * (uX * n[1] - gm1 * vX * n[0]);                        \
  J[8] = half * (uX * n[2] - gm1 * wX * n[0]);                        \
  J[9] = half * gm1 * n[0];                                           \
  J[10] = half * (half * gm1 * VMagSqrX * n[1] - vX * unX);           \
  J[11] = half * (vX * n[0] - gm1 * uX * n[1]);                       \
  J[12] = half * (vX * n[1] - gm1 * vX * n[1] + unX);                 \
  J[13] = half * (vX * n[2] - gm1 * wX * n[1]);                       \
  J[14] = half * gm1 * n[1];                                          \
  J[15] = half * (half * gm1 * VMagSqrX * n[2] - wX * unX);           \
  J[16] = half * (wX * n[0] - gm1 * uX * n[2]);                       \
  J[17] = half * (wX * n[1] - gm1 * vX * n[2]);                       \
  J[18] = half * (wX * n[2] - gm1 * wX * n[2] + unX);                 \
  J[19] = half * gm1 * n[2];                                          \
  J[20] = half * ((half * gm1 * VMagSqrX - HX) * unX);                \
  J[21] = half * (HX * n[0] - gm1 * uX * unX);                        \
  J[22] = half * (HX * n[1] - gm1 * vX * unX);                        \
  J[23] = half * (HX * n[2] - gm1 * wX * unX);                        \
  J[24] = half * gamma * unX;
  PDA_FILL_J5(JL, uL, vL, wL, unL, HL, VMagSqrL)
  for (int i = 0; i < 5; i++) {
    JL[i * 5 + i] = fma_p2(half, smax, JL[i * 5 + i]);
    for (int j = 0; j < 5; j++) JL[i * 5 + j] += half * gL[j] * (qL[i] - qR[i]);
  }
  PDA_FILL_J5(JR, uR, vR, wR, unR, HR, VMagSqrR)
#undef PDA_FILL_J5
  for (int i = 0; i < 5; i++) {
    JR[i * 5 + i] = fma_p2(-half, smax, JR[i * 5 + i]);
    for (int j = 0; j < 5; j++) JR[i * 5 + j] += half * gR[j] * (qL[i] - qR[i]);
  }
}
template <int AXIS, typename T>
PDA_HD void euler5_flux_jac(T JL[25], T JR[25], const T qL[5],
                            const T qR[5], T gamma) {
  euler5_flux_jac_ax(JL, JR, qL, qR, gamma, AXIS);
}

// The 2D Euler face's Rusanov flux fl and twice its two Jacobians, J2L = 2
// dF/dqL and J2R = 2 dF/dqR, for a normal along a fixed axis: euler4_flux and
// euler4_flux_jac with the products by the normal's
// zeros and ones left out, what the three have in common formed once, and the
// factors of 1/2 (exact) joined to a sum or left to the caller, who scales by
// half as much; every other rounding is theirs.  One call forms one of the
// two (side 0: J2L and the flux, side 1: J2R), so that two warps share a
// face's work; set(row, column, x) receives the entries.
template <int AXIS, class M, class S>
PDA_HD void euler4_flux_jac2(int which, double *fl, S set, const double *qL, const double *qR, double gamma) {
  constexpr int DIM = 2, N = DIM + 2, E = DIM + 1;
  constexpr double es = 1.e-30;
  const double gm1 = gamma - 1.;
  struct Side {
    double v[DIM], V2, p, H;  // velocities, |v|^2, pressure, enthalpy
  };
  auto side = [&](Side &o, const double *q) {
    const double r = q[0];
#pragma unroll
    for (int k = 0; k < DIM; ++k) o.v[k] = div_rn(q[1 + k], (r + es));
    o.V2 = M::mul(o.v[0], o.v[0]);
#pragma unroll
    for (int k = 1; k < DIM; ++k) o.V2 = o.V2 + M::mul(o.v[k], o.v[k]);
    o.p = M::mul(gm1, fma_p2(-0.5, M::mul(r, o.V2), q[E]));
    o.H = div_rn(q[E] + o.p, r);
  };
  Side L, R;
  side(L, qL);
  side(R, qR);
  const double rL = qL[0], rR = qR[0];
  const double r = sqrt_rn(M::mul(rR, rL));
  const double RT = sqrt_rn(div_rn(rR, rL));
  const double T1 = 1. + RT;
  double v[DIM];
#pragma unroll
  for (int k = 0; k < DIM; ++k) v[k] = div_rn(L.v[k] + M::mul(RT, R.v[k]), T1);
  const double H = div_rn(L.H + M::mul(RT, R.H), T1);
  double V2 = M::mul(v[0], v[0]);
#pragma unroll
  for (int k = 1; k < DIM; ++k) V2 = V2 + M::mul(v[k], v[k]);
  const double a = sqrt_rn(M::mul(gm1, fma_p2(-0.5, V2, H)));
  const double smax = sqrt_rn(V2) + a;
  const double V2es = V2 + es;
  const double sv = sqrt_rn(V2es);
  double rel[DIM];
#pragma unroll
  for (int k = 0; k < DIM; ++k) rel[k] = div_rn(v[k], sv);
  const double ga = div_rn(0.5 * gm1, a);
  double dq[N];
#pragma unroll
  for (int k = 0; k < N; ++k) dq[k] = qL[k] - qR[k];
  if (which == 0) {
    const double mL = M::mul(rL, L.v[AXIS]), mR = M::mul(rR, R.v[AXIS]);
    fl[0] = 0.5 * (mL + mR + M::mul(smax, dq[0]));
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      double fL = M::mul(mL, L.v[k]), fR = M::mul(mR, R.v[k]);
      if (k == AXIS) {
        fL = fL + L.p;
        fR = fR + R.p;
      }
      fl[1 + k] = 0.5 * (fL + fR + M::mul(smax, dq[1 + k]));
    }
    fl[E] = 0.5 * (M::mul(mL, L.H) + M::mul(mR, R.H) + M::mul(smax, dq[E]));
  }
  Side X;
#pragma unroll
  for (int k = 0; k < DIM; ++k) X.v[k] = which == 0 ? L.v[k] : R.v[k];
  X.V2 = which == 0 ? L.V2 : R.V2;
  X.H = which == 0 ? L.H : R.H;
  const double aX = sqrt_rn(M::mul(gm1, fma_p2(-0.5, X.V2, X.H)));
  const double rX = which == 0 ? rL : rR, diag = which == 0 ? smax : -smax;
  const double inv = div_rn(1., rX + r);
  double g[N];
  double m = M::mul(X.v[0] + v[0], rel[0]), VV = M::mul(X.v[0], v[0]);
#pragma unroll
  for (int k = 1; k < DIM; ++k) {
    m = m + M::mul(X.v[k] + v[k], rel[k]);
    VV = VV + M::mul(X.v[k], v[k]);
  }
  const double t = fma_p2(0.5, M::mul(gamma - 2., X.V2),
                          fma_p2(0.5, (V2es + VV) + (X.H - H), -div_rn(M::mul(aX, aX), gm1)));
  g[0] = M::mul(inv, fma_p2(-0.5, m, M::mul(ga, t)));
#pragma unroll
  for (int k = 0; k < DIM; ++k)
    g[1 + k] = M::mul(inv, fma_p2(-0.5, div_rn(M::mul(gm1, v[k] + M::mul(gm1, X.v[k])), a), rel[k]));
  g[E] = 0.5 * div_rn(M::mul(M::mul(inv, gamma), gm1), a);
  const double un = X.v[AXIS], gV2 = M::mul(gm1, X.V2);
  double w[DIM];  // gm1 v
#pragma unroll
  for (int k = 0; k < DIM; ++k) w[k] = M::mul(gm1, X.v[k]);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const double tt = M::mul(g[j], dq[i]);
      bool zero = false;
      double e = 0.;
      if (i == 0) {
        if (j == 1 + AXIS) e = 1.;
        else zero = true;
      } else if (i < E) {
        const int k = i - 1, l = j - 1;
        if (j == 0) e = k == AXIS ? fma_p2(0.5, gV2, -M::mul(X.v[k], un)) : -M::mul(X.v[k], un);
        else if (j == E) {
          if (k == AXIS) e = gm1;
          else zero = true;
        } else if (k == AXIS) e = l == AXIS ? X.v[k] - w[k] + un : -w[l];
        else if (l == AXIS) e = X.v[k];
        else if (l == k) e = un;
        else zero = true;
      } else {
        if (j == 0) e = M::mul(fma_p2(0.5, gV2, -X.H), un);
        else if (j == E) e = M::mul(gamma, un);
        else e = j - 1 == AXIS ? X.H - M::mul(w[j - 1], un) : -M::mul(w[j - 1], un);
      }
      if (i == j) {
        e = zero ? diag : diag + e;
        zero = false;
      }
      set(i, j, zero ? tt : e + tt);
    }
}

// Shallow-water Rusanov flux Jacobian with respect to the left (side 0) or the
// right state; u_n, q_n and u_t, q_t are the normal's and the other component.
// Products with the normal's 0 and 1 are left out: a zero factor's term is zero
// unless a value is not finite, and then, as in the full form, hsum (hence dn,
// dt and every entry) is NaN; the exact halves of a sum's terms are taken once,
// of the sum.  One face costs 45 FP64 instructions and 13 divisions and roots
// a side where the generic form takes 100 and 19.
// deviation: pow(x,0.5) -> sqrt(x); pow(2,3/2) is the correctly rounded
// constant 2*sqrt(2).
template <typename T>
PDA_HD void swe_flux_jac_side(T J[9], int side, const T qL[3], const T qR[3], T g, int ax) {
  constexpr T es = T(1.e-30);
  const T two_pow_1p5 = T(2.) * sqrt(T(2.));
  const T hL = qL[0], hR = qR[0];
  const T qnL = ax == 0 ? qL[1] : qL[2], qtL = ax == 0 ? qL[2] : qL[1];
  const T qnR = ax == 0 ? qR[1] : qR[2], qtR = ax == 0 ? qR[2] : qR[1];
  T unL, utL, unR, utR;
  if constexpr (sizeof(T) == 8) {
    const Quot2 a = div2_rn(qnL, qtL, hL + es), b = div2_rn(qnR, qtR, hR + es);
    unL = a.q0, utL = a.q1, unR = b.q0, utR = b.q1;
  } else {
    unL = div_rn(qnL, hL + es), utL = div_rn(qtL, hL + es);
    unR = div_rn(qnR, hR + es), utR = div_rn(qtR, hR + es);
  }
  const T sL = sqrt_rn(hL), sR = sqrt_rn(hR), sum = sL + sR, hsum = hL + hR;
  T num = unL * sL + unR * sR;
  if (not_finite(utL) || not_finite(utR)) num = (utL - utL) + (utR - utR);  // NaN
  const T um = div_rn(num, sum + es);
  T smax = fabs(um) + fabs(sqrt_rn(g * half_of(hsum)));
  const T hu = num + es, ahu = fabs(hu);
  // this side
  const T h = side == 0 ? hL : hR, s = side == 0 ? sL : sR, un = side == 0 ? unL : unR, ut = side == 0 ? utL : utR;
  const T qn = side == 0 ? qnL : qnR, qt = side == 0 ? qtL : qtR;
  const T term = div_rn(qn, sq(h));
  const T d0 = half_of(div_rn(-ahu, s * sq(sum))) +
               div_rn((div_rn(half_of(un), s) - s * term) * hu, sum * ahu) +
               div_rn(g, two_pow_1p5 * sqrt_rn(g * hsum));
  const T den = s * sum * ahu, dn = div_rn(hu, den);
  T dt = T(0.);
  if (not_finite(dn)) dt = div_rn(dt * hu, den);
  const T dh = hR - hL, dqn = qnR - qnL, dqt = qtR - qtL;
  if (side != 0) smax = -smax;
  const T J0n = half_of(T(1.) - dn * dh);
  const T Jn0 = half_of((g * h - qn * term) - d0 * dqn);
  const T Jnn = fma_p2(-T(0.5), dn * dqn, fma_p2(T(0.5), smax, un));
  const T Jt0 = half_of(-(qt * term) - d0 * dqt);
  const T Jtn = half_of(ut - dn * dqt);
  const T Jtt = not_finite(dt) ? dt : half_of(un + smax);
  J[0] = half_of(((un - h * term) - d0 * dh) + smax);
  J[1] = ax == 0 ? J0n : dt;
  J[2] = ax == 0 ? dt : J0n;
  J[3] = ax == 0 ? Jn0 : Jt0;
  J[4] = ax == 0 ? Jnn : Jtt;
  J[5] = ax == 0 ? dt : Jtn;
  J[6] = ax == 0 ? Jt0 : Jn0;
  J[7] = ax == 0 ? Jtn : dt;
  J[8] = ax == 0 ? Jtt : Jnn;
}
template <typename T>
PDA_HD void swe_flux_jac_ax(T JL[9], T JR[9], const T qL[3], const T qR[3], T g, int ax) {
  swe_flux_jac_side(JL, 0, qL, qR, g, ax);
  swe_flux_jac_side(JR, 1, qL, qR, g, ax);
}
template <int AXIS, typename T>
PDA_HD void swe_flux_jac(T JL[9], T JR[9], const T qL[3],
                         const T qR[3], T g) {
  swe_flux_jac_ax(JL, JR, qL, qR, g, AXIS);
}

}  // namespace pda
