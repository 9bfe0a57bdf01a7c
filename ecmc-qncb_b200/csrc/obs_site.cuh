// obs_site.cuh — per-site plaquette contributions, shared by the single-lattice and batched
// reductions.
//
// Reference: mean_plaquette_local (src/observables/observables_mpi.cpp:8-29).
#pragma once
#include "staple.cuh"

namespace qcb {

template <typename F, typename R>
__device__ __forceinline__ R site_plaquette(const Geom& g, const F& f, const Coord& x, int par,
                                            uint32_t i) {
  const int opp = par ^ 1;
  R sum = 0;
#pragma unroll
  for (int mu = 0; mu < 4; ++mu) {
    const m3<R> Umu = f.template load<R>(mu, par, i);
    const uint32_t xmu = cb_index(nb_full(g, x, mu, +1));
#pragma unroll
    for (int nu = mu + 1; nu < 4; ++nu) {
      const uint32_t xnu = cb_index(nb_full(g, x, nu, +1));
      // T1 = U_mu(x) U_nu(x+mu), T2 = U_nu(x) U_mu(x+nu); Re tr(T1 T2^dag)
      m3<R> T1 = mul_nn(Umu, f.template load<R>(nu, opp, xmu));
      m3<R> T2 = mul_nn(f.template load<R>(nu, par, i), f.template load<R>(mu, opp, xnu));
      sum += re_tr_na(T1, T2);
    }
  }
  return sum * R(1.0 / 3.0);
}

// Re tr P_{mu nu}(x) of one plane.
template <typename F, typename R>
__device__ __forceinline__ R plaquette_plane(const Geom& g, const F& f, const Coord& x, int par, uint32_t i, int mu,
                                             int nu) {
  const int opp = par ^ 1;
  const NbOff o = nb_offsets(g, x);
  const uint32_t xmu = cb_index((uint32_t)((int32_t)x.s + sel4(o.up, mu)));
  const uint32_t xnu = cb_index((uint32_t)((int32_t)x.s + sel4(o.up, nu)));
  const m3<R> T1 = mul_nn(f.template load<R>(mu, par, i), f.template load<R>(nu, opp, xmu));
  const m3<R> T2 = mul_nn(f.template load<R>(nu, par, i), f.template load<R>(mu, opp, xnu));
  return re_tr_na(T1, T2);
}

// Sum of Re tr P_ij(x) over the spatial planes i < j < 3 (no 1/3), for the measuring
// heatbath pass.
template <typename F, typename R>
__device__ __forceinline__ R site_plaquette_spatial(const Geom& g, const F& f, const Coord& x, int par,
                                                    uint32_t i) {
  const int opp = par ^ 1;
  R sum = 0;
#pragma unroll
  for (int mu = 0; mu < 2; ++mu) {
    const m3<R> Umu = f.template load<R>(mu, par, i);
    const uint32_t xmu = cb_index(nb_full(g, x, mu, +1));
#pragma unroll
    for (int nu = mu + 1; nu < 3; ++nu) {
      const uint32_t xnu = cb_index(nb_full(g, x, nu, +1));
      m3<R> T1 = mul_nn(Umu, f.template load<R>(nu, opp, xmu));
      m3<R> T2 = mul_nn(f.template load<R>(nu, par, i), f.template load<R>(mu, opp, xnu));
      sum += re_tr_na(T1, T2);
    }
  }
  return sum;
}

}  // namespace qcb
