// obs_site.cuh — per-site plaquette contributions, shared by the single-lattice and batched
// reductions.
//
// Reference: mean_plaquette_local (src/observables/observables_mpi.cpp:8-29).
#pragma once
#include "staple.cuh"

namespace qcb {

// Re tr P_{mu nu}(x) of one plane.
template <typename F, typename R>
__device__ __forceinline__ R plaquette_plane(const Geom& g, const F& f, const Coord& x, int par, uint32_t i, int mu,
                                             int nu) {
  const int opp = par ^ 1;
  const NbOff o = nb_offsets(g, x);
  const uint32_t xmu = cb_index((uint32_t)((int32_t)x.s + sel4(o.up, mu)));
  const uint32_t xnu = cb_index((uint32_t)((int32_t)x.s + sel4(o.up, nu)));
  // T1 = U_mu(x) U_nu(x+mu), T2 = U_nu(x) U_mu(x+nu); Re tr(T1 T2^dag)
  if constexpr (F::NREAL == 12) {  // rows 0 and 1 from the stored rows, row 2 of each from them
    m3<R> T1 = mul_nn_rows01(f.template load_rows01<R>(mu, par, i), f.template load<R>(nu, opp, xmu));
    m3<R> T2 = mul_nn_rows01(f.template load_rows01<R>(nu, par, i), f.template load<R>(mu, opp, xnu));
    reconstruct_row2(T1);
    reconstruct_row2(T2);
    return re_tr_na(T1, T2);
  } else {
    const m3<R> T1 = mul_nn(f.template load<R>(mu, par, i), f.template load<R>(nu, opp, xmu));
    const m3<R> T2 = mul_nn(f.template load<R>(nu, par, i), f.template load<R>(mu, opp, xnu));
    return re_tr_na(T1, T2);
  }
}

// Sum of Re tr P_{mu nu}(x) over planes p0, p0 + dp, ... < np of 01, 02, 12, 03, 13, 23 (the
// spatial ones first), in FP64 whichever planes go together.  One plane body, not unrolled.
template <typename F, typename R>
__device__ __forceinline__ double site_plaquettes(const Geom& g, const F& f, const Coord& x, int par, uint32_t i, int p0,
                                             int dp, int np) {
  double sum = 0.0;
#pragma unroll 1
  for (int p = p0; p < np; p += dp)
    sum += (double)plaquette_plane<F, R>(g, f, x, par, i, p < 2 ? 0 : (p == 2 ? 1 : p - 3),
                                         p < 2 ? p + 1 : (p == 2 ? 2 : 3));
  return sum;
}

}  // namespace qcb
