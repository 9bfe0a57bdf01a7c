// loops.cuh — plaquette loops, their parallel transport, and what the Wilson flow and the
// clover make of them.
//
// Reference: the force -P_TA(U A) of GradientFlow (src/flow/gradient_flow.cpp:15-34) with the
// staples of GaugeField.cpp:74-97, and the clover leaves of observables_mpi.cpp:61-107.
//
// With L_{mu nu}(y) = U_mu(y) U_nu(y+mu) U_mu(y+nu)^dag U_nu(y)^dag, every term of both is a
// loop at some corner of a plaquette, and a loop moved along a link is conjugated by it; P_TA
// commutes with the conjugation.  So with K_{mu nu} = P_TA(L_{mu nu}), K_{nu mu} = -K_{mu nu}:
//   P_TA(U_mu(x) A_mu(x)) = sum_{nu != mu} [ K_{mu nu}(x) - Ad(U_nu(x-nu)) K_{mu nu}(x-nu) ]
//   clover at x, from its four leaves = K(x) + Ad(U_nu(x-nu)) K(x-nu)
//     + Ad(U_mu(x-mu)) [ K(x-mu) + Ad(U_nu(x-mu-nu)) K(x-mu-nu) ],  K = K_{mu nu}
// with Ad(U) M = U^dag M U.  Each plaquette is multiplied out once (three products) instead of
// seven times for the flow and sixteen for the clover, and a transport of eight reals costs
// about as much as one product.
//
// The conjugated loop ends in U_nu(x-nu)^dag U_nu(x-nu) where the staple and the leaf do not, so this
// holds for unitary links only.  12-real storage keeps two rows and takes the links as SU(3)
// everywhere.  18-real storage holds whatever was written to it (links from a single-precision
// file, say, unitary to 1e-7), so there the loops kernel also tests every link (off_unitary), and a
// loop is moved along a link that fails by multiplying out the product that it stands for (leaf_*).
#pragma once
#include <type_traits>

#include "flow.h"
#include "staple.cuh"

namespace qcb {

// Index of plane (mu, nu), mu < nu: 01, 02, 03, 12, 13, 23.
__device__ __forceinline__ int plane_of(int mu, int nu) { return ((mu * (7 - mu)) >> 1) + nu - mu - 1; }

// The loop field of one lattice.  Time slice tv (-1: the slice before 0) sits in ring slot
// (tv + 1) mod slices, or at its own place when all slices fit.
template <typename S>
struct Loops {
  typedef typename AlgStore<S>::V V;
  static constexpr int NC = AlgStore<S>::NC;
  V* p;
  S* tr;
  uint8_t* off;
  uint32_t stride, half;
  int slices;
  bool full;
  __device__ __forceinline__ Loops(const LoopDev& k, const Geom& g)
      : p(reinterpret_cast<V*>(k.p)), tr(reinterpret_cast<S*>(k.tr)), off(k.off), stride(k.stride),
        half((uint32_t)g.str[3] >> 1), slices(k.slices), full(k.slices >= g.L[3]) {}
  // place of checkerboard site i of time t, read as slice tv
  __device__ __forceinline__ uint32_t at(uint32_t i, int t, int tv) const {
    if (full) return i;
    return i + (uint32_t)((tv + 1) % slices - t) * half;
  }
  __device__ __forceinline__ size_t idx(int plane, int par, int c, uint32_t j) const {
    return ((size_t)((plane * 2 + par) * NC + c)) * stride + j;
  }
  template <typename R>
  __device__ __forceinline__ alg8<R> load(int plane, int par, uint32_t j) const {
    V v[NC];
    const V* at = p + idx(plane, par, 0, j);
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = __ldg(at + c * (size_t)stride);
    const S* q = reinterpret_cast<const S*>(v);
    alg8<R> z;
#pragma unroll
    for (int k = 0; k < 8; ++k) z.a[k] = R(q[k]);
    return z;
  }
  template <typename R>
  __device__ __forceinline__ void store(int plane, int par, uint32_t j, const alg8<R>& z) const {
    V v[NC];
    S* q = reinterpret_cast<S*>(v);
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = S(z.a[k]);
    V* at = p + idx(plane, par, 0, j);
#pragma unroll
    for (int c = 0; c < NC; ++c) at[c * (size_t)stride] = v[c];
  }
  template <typename R>
  __device__ __forceinline__ R load_tr(int plane, int par, uint32_t j) const {
    return R(__ldg(&tr[(size_t)(plane * 2 + par) * stride + j]));
  }
  template <typename R>
  __device__ __forceinline__ void store_tr(int plane, int par, uint32_t j, R v) const {
    tr[(size_t)(plane * 2 + par) * stride + j] = S(v);
  }
  __device__ __forceinline__ bool load_off(int mu, int par, uint32_t j) const {
    return __ldg(&off[(size_t)(mu * 2 + par) * stride + j]) != 0;
  }
  __device__ __forceinline__ void store_off(int mu, int par, uint32_t j, bool v) const {
    off[(size_t)(mu * 2 + par) * stride + j] = v ? 1 : 0;
  }
};

// Whether |U U^dag - 1| is above 2^-40 (FP32: 2^-21) in the Frobenius norm, or not a number; the
// relative error of a loop moved along U is at most about that.  Measured on 16^4, the largest of all
// links: FP64 after 10000 sweeps 1.8e-13, after 1000 RK3 steps 4e-14; FP32 after an RK3 step (which
// ends with re-orthonormalised links) or when SU(3) links are rounded 1.4e-7, after 10 sweeps 5e-6 and
// after 2000 3e-4, all in one direction, so that the clover of FP32 18-real links is multiplied out
// behind sweeps.  (At 2^-22 the bound meets the rounding between the stages of an RK3 step: 20x24x28x36
// FP32 18-real 582 us a step, 540 at 2^-21.)
template <typename S, typename R>
__device__ __forceinline__ bool off_unitary(const m3<R>& U) {
  constexpr double BOUND = sizeof(S) == 8 ? 0x1p-80 : 0x1p-42;
  R s = 0;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    R d = R(-1);
#pragma unroll
    for (int k = 0; k < 3; ++k) d = fma(U.e[r][k].re, U.e[r][k].re, fma(U.e[r][k].im, U.e[r][k].im, d));
    s = fma(d, d, s);
#pragma unroll
    for (int q = r + 1; q < 3; ++q) {
      cx<R> o = mk<R>(R(0), R(0));
#pragma unroll
      for (int k = 0; k < 3; ++k) o = cfma_nc(U.e[r][k], U.e[q][k], o);
      s = fma(R(2), fma(o.re, o.re, o.im * o.im), s);
    }
  }
  return !(s <= R(BOUND));
}

// The leading link of a product: its stored rows (12-real), or all of it.
template <typename F, typename R>
__device__ __forceinline__ m3<R> lead(const F& f, int mu, int par, uint32_t i) {
  if constexpr (F::NREAL == 12)
    return f.template load_rows01<R>(mu, par, i);
  else
    return f.template load<R>(mu, par, i);
}

// L_{mu nu} = (U_mu(x) U_nu(x+mu)) (U_nu(x) U_mu(x+nu))^dag.  12-real storage: rows 0 and 1 of
// the three products from the stored rows of their first factors; row 2 of the second and of L
// from the cross product (each is in SU(3)).
template <typename F, typename R>
__device__ __forceinline__ m3<R> plaquette_loop(const F& f, const m3<R>& Umu, int mu, int nu, int par, uint32_t i,
                                                uint32_t ixmu, uint32_t ixnu) {
  const int opp = par ^ 1;
  const m3<R> Unu = lead<F, R>(f, nu, par, i);
  if constexpr (F::NREAL == 12) {
    const m3<R> G = mul_nn_rows01(Umu, f.template load<R>(nu, opp, ixmu));
    m3<R> H = mul_nn_rows01(Unu, f.template load<R>(mu, opp, ixnu));
    reconstruct_row2(H);
    m3<R> L = mul_na_rows01(G, H);
    reconstruct_row2(L);
    return L;
  } else {
    const m3<R> G = mul_nn(Umu, f.template load<R>(nu, opp, ixmu));
    const m3<R> H = mul_nn(Unu, f.template load<R>(mu, opp, ixnu));
    return mul_na(G, H);
  }
}

// i d v for real d
template <typename R>
__device__ __forceinline__ cx<R> times_i(R d, cx<R> v) {
  return mk(-(d * v.im), d * v.re);
}
// acc - conj(a) b
template <typename R>
__device__ __forceinline__ cx<R> cfms_cn(cx<R> a, cx<R> b, cx<R> acc) {
  acc.re = fma(-a.re, b.re, acc.re);
  acc.re = fma(-a.im, b.im, acc.re);
  acc.im = fma(-a.re, b.im, acc.im);
  acc.im = fma(a.im, b.re, acc.im);
  return acc;
}
// Im(conj(u) . b) over three components
template <typename R>
__device__ __forceinline__ R im_dot3(const cx<R> (&u)[3], const cx<R> (&b)[3]) {
  R p = u[0].re * b[0].im, m = u[0].im * b[0].re;
#pragma unroll
  for (int k = 1; k < 3; ++k) p = fma(u[k].re, b[k].im, p), m = fma(u[k].im, b[k].re, m);
  return p - m;
}
// conj(u) . b over three components
template <typename R>
__device__ __forceinline__ cx<R> dot3(const cx<R> (&u)[3], const cx<R> (&b)[3]) {
  cx<R> s = mk(fma(u[0].re, b[0].re, u[0].im * b[0].im), fma(u[0].re, b[0].im, -(u[0].im * b[0].re)));
  s = cfma_cn(u[1], b[1], s);
  return cfma_cn(u[2], b[2], s);
}

// Ad(U) K = U^dag K U: element (i, j) is conj(u_i) . (K u_j) with the columns u of U.  Columns 0 and 1
// of the result hold all of it (anti-Hermitian, traceless), so K u_2 is not formed: 108 multiply-adds,
// 138 with the upper triangle's three columns.  32^4: RK3 step FP32 12-real 916 -> 884 us, FP64 18-real
// 1890 -> 1810; Q and E of FP64 631 -> 598.
template <typename R>
__device__ __forceinline__ alg8<R> transport(const m3<R>& U, const alg8<R>& K) {
  const cx<R> a = mk(K.a[2], K.a[3]), b = mk(K.a[4], K.a[5]), c = mk(K.a[6], K.a[7]);
  const R d2 = -(K.a[0] + K.a[1]);
  cx<R> u[3][3], w[3];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) u[j][k] = U.e[k][j];
  alg8<R> r;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    // rows of K: (i d0, a, b), (-a*, i d1, c), (-b*, -c*, i d2)
    w[0] = cfma(b, u[j][2], cfma(a, u[j][1], times_i(K.a[0], u[j][0])));
    w[1] = cfma(c, u[j][2], cfms_cn(a, u[j][0], times_i(K.a[1], u[j][1])));
    w[2] = cfms_cn(c, u[j][1], cfms_cn(b, u[j][0], times_i(d2, u[j][2])));
    r.a[j] = im_dot3(u[j], w);
    // elements (1, 0), (2, 0), (2, 1), each minus the conjugate of its mirror image
    const cx<R> q = dot3(u[2], w);
    if (j == 0) {
      const cx<R> o = dot3(u[1], w);
      r.a[2] = -o.re, r.a[3] = o.im;
      r.a[4] = -q.re, r.a[5] = q.im;
    } else {
      r.a[6] = -q.re, r.a[7] = q.im;
    }
  }
  return r;
}

// a + sg b, sg = +-1
template <typename R>
__device__ __forceinline__ void add_alg(alg8<R>& a, const alg8<R>& b, R sg = R(1)) {
#pragma unroll
  for (int q = 0; q < 8; ++q) a.a[q] = fma(sg, b.a[q], a.a[q]);
}

// The loop L_{mu nu}(y) (either order of mu and nu), begun at y+nu instead of y:
// U_nu(y)^dag U_mu(y) U_nu(y+mu) U_mu(y+nu)^dag.  iy, iymu, iynu: y (parity py), y+mu, y+nu.
template <typename F, typename R>
__device__ __forceinline__ m3<R> loop_beside(const F& f, int mu, int nu, int py, uint32_t iy, uint32_t iymu,
                                             uint32_t iynu) {
  m3<R> M = mul_an(f.template load<R>(nu, py, iy), f.template load<R>(mu, py, iy));
  M = mul_nn(M, f.template load<R>(nu, py ^ 1, iymu));
  return mul_na(M, f.template load<R>(mu, py ^ 1, iynu));
}
// The same begun at z+mu+nu: [U_nu(z) U_mu(z+nu)]^dag U_mu(z) U_nu(z+mu).
template <typename F, typename R>
__device__ __forceinline__ m3<R> loop_across(const F& f, int mu, int nu, int pz, uint32_t iz, uint32_t izmu,
                                             uint32_t iznu) {
  const m3<R> H = mul_nn(f.template load<R>(nu, pz, iz), f.template load<R>(mu, pz ^ 1, iznu));
  const m3<R> G = mul_nn(f.template load<R>(mu, pz, iz), f.template load<R>(nu, pz ^ 1, izmu));
  return mul_an(H, G);
}
// P_TA of the two.
template <typename F, typename R>
__device__ __forceinline__ alg8<R> leaf_beside(const F& f, int mu, int nu, int py, uint32_t iy, uint32_t iymu,
                                               uint32_t iynu) {
  return proj_ta(loop_beside<F, R>(f, mu, nu, py, iy, iymu, iynu));
}
template <typename F, typename R>
__device__ __forceinline__ alg8<R> leaf_across(const F& f, int mu, int nu, int pz, uint32_t iz, uint32_t izmu,
                                               uint32_t iznu) {
  return proj_ta(loop_across<F, R>(f, mu, nu, pz, iz, izmu, iznu));
}
// Out of line, so that the products cost the transports beside them no registers (the clover in FP32
// has them in line: 380 us so, 312 in line on 20x24x28x36 with links that need them).
template <typename F, typename R>
__device__ __noinline__ alg8<R> leaf_beside_call(F f, int mu, int nu, int py, uint32_t iy, uint32_t iymu,
                                                 uint32_t iynu) {
  return leaf_beside<F, R>(f, mu, nu, py, iy, iymu, iynu);
}
template <typename F, typename R>
__device__ __noinline__ alg8<R> leaf_across_call(F f, int mu, int nu, int pz, uint32_t iz, uint32_t izmu,
                                                 uint32_t iznu) {
  return leaf_across<F, R>(f, mu, nu, pz, iz, izmu, iznu);
}

// The loops below site x in direction nu, K_{mu nu}(x-nu) of the three mu != nu (mu ascending,
// K_{nu mu} where nu < mu), moved to x: out[k] = Ad(U_nu(x-nu)) K.
template <typename F, typename S, typename R>
__device__ __forceinline__ void transported(const Geom& g, const F& f, const Loops<S>& K, const Coord& x, int nu,
                                            int par, alg8<R> (&out)[3]) {
  const int opp = par ^ 1, t = x.c[3], L = g.L[nu], d = g.str[nu];
  const int32_t sy = (int32_t)x.s + (sel4(x.c, nu) == 0 ? (L - 1) * d : -d);
  const uint32_t iy = cb_index((uint32_t)sy);
  const uint32_t jy = nu == 3 ? K.at(iy, t == 0 ? L - 1 : t - 1, t - 1) : K.at(iy, t, t);
  const int p0 = nu == 0 ? 0 : nu - 1, p1 = nu < 2 ? 3 * nu + (1 - nu) : nu + 1, p2 = nu < 2 ? 2 + 2 * nu : 5;
  const m3<R> U = f.template load<R>(nu, opp, iy);
  const alg8<R> k0 = K.template load<R>(p0, opp, jy), k1 = K.template load<R>(p1, opp, jy),
                k2 = K.template load<R>(p2, opp, jy);
  if constexpr (F::NREAL == 18) {
    if (off_unitary<S>(U)) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int mu = k + (k >= nu);
        const int32_t up = sel4(x.c, mu) + 1 == g.L[mu] ? (1 - g.L[mu]) * g.str[mu] : g.str[mu];
        out[k] = leaf_beside_call<F, R>(f, mu, nu, opp, iy, cb_index((uint32_t)(sy + up)), cb_index(x.s));
        if (mu > nu) {
#pragma unroll
          for (int a = 0; a < 8; ++a) out[k].a[a] = -out[k].a[a];
        }
      }
      return;
    }
  }
  out[0] = transport(U, k0);
  out[1] = transport(U, k1);
  out[2] = transport(U, k2);
}

// Anti-Hermitian 3x3 matrix in 9 reals: F_kk = i d[k], F_ij = o[.] for (i,j) = (0,1),
// (0,2), (1,2), and F_ji = -conj(F_ij).
template <typename R>
struct ah9 {
  R d[3];
  cx<R> o[3];
};

// Re tr(A B) of two anti-Hermitian matrices: -sum_k a_k b_k - 2 sum_{i<j} Re(A_ij conj B_ij).
template <typename R>
__device__ __forceinline__ R re_tr_ah(const ah9<R>& A, const ah9<R>& B) {
  R s = 0, t = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s = fma(A.d[k], B.d[k], s);
    t = fma(A.o[k].re, B.o[k].re, fma(A.o[k].im, B.o[k].im, t));
  }
  return fma(R(-2), t, -s);
}

// |F|^2 = sum_ij |F_ij|^2 = sum_k d_k^2 + 2 sum_{i<j} |F_ij|^2.
template <typename R>
__device__ __forceinline__ R sqnorm_ah(const ah9<R>& A) {
  R s = 0, t = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s = fma(A.d[k], A.d[k], s);
    t = fma(A.o[k].re, A.o[k].re, fma(A.o[k].im, A.o[k].im, t));
  }
  return fma(R(2), t, s);
}

// F_{mu nu}(x) = (C - C^dag) / 8 (observables_mpi.cpp:81-82), C the sum of the four leaves: a
// quarter of the transported loops, their traces (the same at every corner) on the diagonal.  The third
// place takes what the other two leave of the whole trace: three times FP32's 1/3 is not 1, and E came
// out 1.1e-9 too large with a third of the trace in each (5e-10 so).  multiply: one of the three links that loops
// move along here is not unitary.
template <typename F, typename S, typename R>
__device__ __forceinline__ ah9<R> clover_plane(const F& f, const Loops<S>& K, const Coord& x, const NbOff& o, int mu,
                                               int nu, int par, uint32_t i, int Lt, bool multiply) {
  const int opp = par ^ 1, t = x.c[3], plane = plane_of(mu, nu);
  const int tm = t == 0 ? Lt - 1 : t - 1;
  const int32_t s = (int32_t)x.s, dmu = sel4(o.dn, mu), dnu = sel4(o.dn, nu);
  const uint32_t imu = (uint32_t)(s + dmu) >> 1, inu = (uint32_t)(s + dnu) >> 1, imn = (uint32_t)(s + dmu + dnu) >> 1;
  // only nu can be the time direction (mu < nu)
  const int tn = nu == 3 ? tm : t, vn = nu == 3 ? t - 1 : t;
  const uint32_t j0 = K.at(i, t, t), jmu = K.at(imu, t, t), jnu = K.at(inu, tn, vn), jmn = K.at(imn, tn, vn);
  alg8<R> A;
  if (multiply) {
    if constexpr (F::NREAL == 18) {
      const int32_t umu = sel4(o.up, mu), unu = sel4(o.up, nu);
      const uint32_t iun = cb_index((uint32_t)(s + dmu + unu)), ium = cb_index((uint32_t)(s + dnu + umu));
      if constexpr (is_fp32<R>::value) {
        A = leaf_across<F, R>(f, mu, nu, par, imn, inu, imu);
        add_alg(A, leaf_beside<F, R>(f, nu, mu, opp, imu, iun, i), R(-1));
        add_alg(A, leaf_beside<F, R>(f, mu, nu, opp, inu, ium, i));
      } else {
        A = leaf_across_call<F, R>(f, mu, nu, par, imn, inu, imu);
        add_alg(A, leaf_beside_call<F, R>(f, nu, mu, opp, imu, iun, i), R(-1));
        add_alg(A, leaf_beside_call<F, R>(f, mu, nu, opp, inu, ium, i));
      }
    }
  } else {
    alg8<R> B = transport(f.template load<R>(nu, par, imn), K.template load<R>(plane, par, jmn));
    add_alg(B, K.template load<R>(plane, opp, jmu));
    A = transport(f.template load<R>(mu, opp, imu), B);
    add_alg(A, transport(f.template load<R>(nu, opp, inu), K.template load<R>(plane, opp, jnu)));
  }
  add_alg(A, K.template load<R>(plane, par, j0));
  const R tr = (K.template load_tr<R>(plane, par, j0) + K.template load_tr<R>(plane, par, jmn)) +
               (K.template load_tr<R>(plane, opp, jmu) + K.template load_tr<R>(plane, opp, jnu));
  ah9<R> out;
  const R d0 = fma(R(1.0 / 3.0), tr, A.a[0]), d1 = fma(R(1.0 / 3.0), tr, A.a[1]);
  out.d[0] = R(0.25) * d0;
  out.d[1] = R(0.25) * d1;
  out.d[2] = R(0.25) * (tr - (d0 + d1));
#pragma unroll
  for (int k = 0; k < 3; ++k) out.o[k] = mk<R>(R(0.25) * A.a[2 + 2 * k], R(0.25) * A.a[3 + 2 * k]);
  return out;
}

}  // namespace qcb
