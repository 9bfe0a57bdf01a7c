// hb_quad.cuh — one FP64 Cabibbo-Marinari heatbath update of one link by four lanes of a warp.
//
// A pass over a small lattice has fewer links than the chip has lanes and takes as long as one
// link: thousands of dependent FP64 instructions.  Here lanes 0, 1, 2 of a group form a row each
// of the staple sum, and lane sg takes the draw of subgroup sg: what two attempts and the
// direction need of their random words alone (logarithms, sines) is computed before the links
// arrive, the three subgroups side by side.  Every element and every draw is computed by the
// operations of hb_link.cuh in their order, so the links are the same bit for bit.  Pass on 8^4,
// 18-real: one lane 11.6 us, four lanes 9.0 (with the attempts of one draw side by side, behind the
// staple, 10.1); on 12^4 12.3 and 11.9.  (One lane with its words ahead, in shared memory, is
// slower: 32^4 192 us against 185, FP32 8^4 7.0 against 5.7: the loads wait for the words there.)
// In FP32, and with 12-real links (whose third rows take all lanes' rows), four
// lanes were slower on 10^4 already, and on 8^4 in FP32 (5.7 against 8.5 us).
#pragma once
#include "hb_link.cuh"

namespace qcb {

// The group of four lanes a thread belongs to.
struct Quad {
  unsigned mask;
  int lane;  // 0 .. 3
  __device__ __forceinline__ Quad() : mask(0xFu << (threadIdx.x & 28)), lane((int)(threadIdx.x & 3)) {}
  template <typename T>
  __device__ __forceinline__ T get(T v, int from) const {
    return __shfl_sync(mask, v, from, 4);
  }
  __device__ __forceinline__ cx<double> get(cx<double> v, int from) const { return mk(get(v.re, from), get(v.im, from)); }
};

// Row `lane` (lane 3: row 2 again) of the staple sum, by the terms of staple_terms.
template <typename F>
__device__ __forceinline__ row3<double> staple_row(const Quad& q, const Geom& g, const F& f, const Coord& x, int mu,
                                                   int par, uint32_t i) {
  typedef double R;
  const int opp = par ^ 1, row = q.lane < 2 ? q.lane : 2;
  const NbOff o = nb_offsets(g, x);
  const int32_t upmu = sel4(o.up, mu);
  const uint32_t ixmu = cb_index((uint32_t)((int32_t)x.s + upmu));
  row3<R> A;
#pragma unroll
  for (int j = 0; j < 3; ++j) A.e[j] = mk<R>(0, 0);
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    const int nu = k + (k >= mu);
    const int32_t upnu = sel4(o.up, nu), dnnu = sel4(o.dn, nu);
    const uint32_t ixnu = cb_index((uint32_t)((int32_t)x.s + upnu));
    const uint32_t ixmunu = cb_index((uint32_t)((int32_t)x.s + upmu + dnnu));
    const uint32_t ixmnu = cb_index((uint32_t)((int32_t)x.s + dnnu));
    {
      // forward: (U_nu(x+mu) U_mu(x+nu)^dagger) U_nu(x)^dagger
      const row3<R> u0 = f.template load_row<R>(nu, opp, ixmu, row);
      const m3<R> U1 = f.template load<R>(mu, opp, ixnu), U2 = f.template load<R>(nu, par, i);
      row3<R> t;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        t.e[j] = mk<R>(0, 0);
#pragma unroll
        for (int m = 0; m < 3; ++m) t.e[j] = cfma_nc(u0.e[m], U1.e[j][m], t.e[j]);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int m = 0; m < 3; ++m) A.e[j] = cfma_nc(t.e[m], U2.e[j][m], A.e[j]);
    }
    {
      // backward: (U_nu(x+mu-nu)^dagger U_mu(x-nu)^dagger) U_nu(x-nu)
      const row3<R> v0 = f.template load_col<R>(nu, par, ixmunu, row);
      const m3<R> V1 = f.template load<R>(mu, opp, ixmnu), V2 = f.template load<R>(nu, opp, ixmnu);
      row3<R> t;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        t.e[j] = mk<R>(0, 0);
#pragma unroll
        for (int m = 0; m < 3; ++m) t.e[j] = cfma_cc(v0.e[m], V1.e[j][m], t.e[j]);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int m = 0; m < 3; ++m) A.e[j] = cfma(t.e[m], V2.e[m][j], A.e[j]);
    }
  }
  return A;
}

// What lane sg of a group holds of subgroup sg's draw: two attempts and the direction.
struct QuadWords {
  double d2[2], lg[2];
  KpDirection<double> dir;
};
__device__ __forceinline__ QuadWords kp_words_quad(const Quad& q, uint32_t link, uint32_t sweep, uint32_t hb,
                                                   uint32_t k0, uint32_t k1) {
  const uint32_t hsg = hb | (uint32_t)(q.lane < 2 ? q.lane : 2);
  QuadWords d;
#pragma unroll
  for (uint32_t att = 0; att < 2; ++att)
    kp_attempt<double>(kp_words(link, sweep, hsg, att, k0, k1), &d.d2[att], &d.lg[att]);
  d.dir = kp_direction<double>(kp_words(link, sweep, hsg, 0xFFFFFFFFu, k0, k1));
  return d;
}

// kp_draw from the words of lane sg; attempts from 2 on four at a time.
__device__ __forceinline__ bool kp_draw_quad(const Quad& q, const QuadWords& d, double mhalf_over_alpha,
                                             uint32_t link, uint32_t sweep, uint32_t hb, int sg, uint32_t k0,
                                             uint32_t k1, double* x) {
  double lam2, lam2b;
  const bool first = kp_accept(mhalf_over_alpha, d.d2[0], d.lg[0], &lam2);
  const bool second = kp_accept(mhalf_over_alpha, d.d2[1], d.lg[1], &lam2b);
  if (!first) lam2 = lam2b;
  bool ok = q.get((int)(first || second), sg) != 0;
  for (uint32_t att = 2; !ok && att < KP_CAP; att += 4) {
    double d2, lg, l2;
    kp_attempt<double>(kp_words(link, sweep, hb | (uint32_t)sg, att + (uint32_t)q.lane, k0, k1), &d2, &lg);
    const bool good = kp_accept(mhalf_over_alpha, d2, lg, &l2) && att + (uint32_t)q.lane < KP_CAP;
    const unsigned hits = (__ballot_sync(q.mask, good) >> (threadIdx.x & 28)) & 0xFu;
    if (hits) {
      lam2 = q.get(l2, __ffs(hits) - 1);
      ok = true;
    }
  }
  if (!ok) return false;
  kp_quaternion(lam2, d.dir, x);
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = q.get(x[k], sg);
  return true;
}

// hb_update_at by the four lanes of q (every lane holds the link; lane 0 stores it).
template <typename F, bool MEAS>
__device__ __forceinline__ uint32_t hb_update_quad(const Quad& q, const Geom& g, const F& f, const Coord& x, int mu,
                                                   int par, uint32_t i, double beta, uint32_t k0, uint32_t k1,
                                                   uint32_t sweep, int n_hits, double* retr) {
  typedef double R;
  const uint32_t link = (uint32_t)mu * g.Vg + (x.s + g.soff);
  QuadWords d = kp_words_quad(q, link, sweep, RNG_DOMAIN_HB, k0, k1);
  m3<R> U = f.template load<R>(mu, par, i), A;
  {
    const row3<R> a = staple_row(q, g, f, x, mu, par, i);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < 3; ++j) A.e[k][j] = q.get(a.e[j], k);
  }
  uint32_t fails = 0;
  for (int h = 0; h < n_hits; ++h) {
    const uint32_t hb = RNG_DOMAIN_HB | ((uint32_t)h << 2);
    if (h) d = kp_words_quad(q, link, sweep, hb, k0, k1);
    auto draw = [&](int sg) {
      return [&, sg](R mhalf_over_alpha, R* y) {
        return kp_draw_quad(q, d, mhalf_over_alpha, link, sweep, hb, sg, k0, k1, y);
      };
    };
    fails += !cm_subgroup_with<R, 0, 1>(U, A, beta, draw(0));
    fails += !cm_subgroup_with<R, 1, 2>(U, A, beta, draw(1));
    fails += !cm_subgroup_with<R, 0, 2>(U, A, beta, draw(2));
  }
  __syncwarp(q.mask);  // the link is read by all four lanes before it is written
  if (q.lane == 0) f.template store<R>(mu, par, i, U);
  if constexpr (MEAS) *retr = re_tr_nn(U, A);
  return fails;
}

}  // namespace qcb
