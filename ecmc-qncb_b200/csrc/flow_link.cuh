// flow_link.cuh — one link of one Wilson-flow RK3 stage, from its force.
//
// Reference: GradientFlow (src/flow/gradient_flow.cpp:15-114):
//   Z   = -P_TA(U A)                         (force, gradient_flow.cpp:15-34)
//   s1: X = eps/4 Z0;                acc = Z0                      (compute_w1, :37-53)
//   s2: X = 8/9 eps Z1 - 17/36 eps Z0; acc = 8/9 Z1 - 17/36 Z0    (compute_w2 + replace_force_0, :56-93)
//   s3: X = 3/4 eps Z2 - eps acc                                   (compute_w3, :96-114)
//   U' = exp(X) U   with Luescher's exponential (src/su3/utils.cpp:145-193)
#pragma once
#include "layout.cuh"

namespace qcb {

// Periodic reunitarisation of FP32 links: after the last stage of each RK3 step the new link
// is converted to FP64, its rows 0 and 1 are orthonormalised (row 2 = conj(r0 x r1)), and it
// is rounded back to FP32.  Without it the FP32 links drift off SU(3) linearly in the number
// of steps; with it the FP32-12 flow of a 32^4 configuration to t = 4 stays within
// |dQ| = 4e-6 and |dE|/E = 6e-8 of the FP64 flow (1e-4 and 2e-5 without), for 3.5% more time
// per step.  FP64 links are left as the reference leaves them.
template <typename R>
__device__ __forceinline__ void flow_reunit(m3<R>& U, int stage) {
  if constexpr (is_fp32<R>::value) {
    if (stage == 3) {
      m3<double> d = convert<double>(U);
      reunitarize_rows(d);
      U = convert<R>(d);
    }
  }
}

// U' = exp(X) U from E = flow_exp(X).  FP32: U + (exp(X) - 1) U, whose products are small, so that one
// rounding at the links' size remains (Q after nine RK3 steps on 24^4 against the FP64 flow, rms of
// six lattices: 2.0e-7, with the products of exp(X) itself 3.4e-7; RK3 step 880 -> 884 us).  12-real
// storage keeps rows 0 and 1 only (the FP64 re-orthonormalisation of stage 3 also reads only those), so
// row 2 of the product is not formed.
template <typename F, typename R>
__device__ __forceinline__ m3<R> flow_product(const m3<R>& E, const m3<R>& U) {
  constexpr int ROWS = F::NREAL == 12 ? 2 : 3;
  m3<R> P;
  if constexpr (F::NREAL == 12)
    P = mul_nn_rows01(E, U);
  else
    P = mul_nn(E, U);
  if constexpr (is_fp32<R>::value) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) P.e[r][c] = U.e[r][c] + P.e[r][c];
  }
  return P;
}

// The stage-dependent part: X from the force Z and the accumulator Z0 (unused in stage 1), and
// the accumulator's update.
template <int STAGE, typename ACC, typename R>
__device__ __forceinline__ alg8<R> flow_x(const ACC& acc, const alg8<R>& Z, const alg8<R>& Z0, R eps, int mu, int par,
                                          uint32_t i) {
  alg8<R> X;
  if constexpr (STAGE == 1) {
    const R c = R(0.25) * eps;
#pragma unroll
    for (int k = 0; k < 8; ++k) X.a[k] = c * Z.a[k];
    acc.template store<R>(mu, par, i, Z);
  } else if constexpr (STAGE == 2) {
    const R c1 = R(8.0 / 9.0) * eps, c0 = R(17.0 / 36.0) * eps;
    alg8<R> N;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      X.a[k] = fma(c1, Z.a[k], -(c0 * Z0.a[k]));
      N.a[k] = fma(R(8.0 / 9.0), Z.a[k], -(R(17.0 / 36.0) * Z0.a[k]));
    }
    acc.template store<R>(mu, par, i, N);
  } else {
    const R c1 = R(0.75) * eps;
#pragma unroll
    for (int k = 0; k < 8; ++k) X.a[k] = fma(c1, Z.a[k], -(eps * Z0.a[k]));
  }
  return X;
}

}  // namespace qcb
