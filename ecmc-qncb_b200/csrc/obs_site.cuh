// obs_site.cuh — per-site plaquette contributions, shared by the single-lattice and batched
// reductions.
//
// Reference: mean_plaquette_local (src/observables/observables_mpi.cpp:8-29).
#pragma once
#include "staple.cuh"

namespace qcb {

// Re tr P_{mu nu}(x) of one plane.  SU3: the links are in SU(3) to rounding (those of a sweep, whose
// 12-real rows are re-orthonormalised), so that the third row of a product follows from its first two.
// Links that were written to the lattice need not be, and 12-real ones are then multiplied out with
// their third rows completed.  32^4, plaquette alone: FP32 12-real 107 us with SU3, 124 without, FP64 188 and
// 219.
template <typename F, typename R, bool SU3>
__device__ __forceinline__ R plaquette_plane(const Geom& g, const F& f, const Coord& x, int par, uint32_t i, int mu,
                                             int nu) {
  const int opp = par ^ 1;
  const NbOff o = nb_offsets(g, x);
  const uint32_t xmu = cb_index((uint32_t)((int32_t)x.s + sel4(o.up, mu)));
  const uint32_t xnu = cb_index((uint32_t)((int32_t)x.s + sel4(o.up, nu)));
  // T1 = U_mu(x) U_nu(x+mu), T2 = U_nu(x) U_mu(x+nu); Re tr(T1 T2^dag)
  if constexpr (F::NREAL == 12 && SU3) {
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
template <typename F, typename R, bool SU3 = false>
__device__ __forceinline__ double site_plaquettes(const Geom& g, const F& f, const Coord& x, int par, uint32_t i, int p0,
                                             int dp, int np) {
  double sum = 0.0;
#pragma unroll 1
  for (int p = p0; p < np; p += dp)
    sum += (double)plaquette_plane<F, R, SU3>(g, f, x, par, i, p < 2 ? 0 : (p == 2 ? 1 : p - 3),
                                         p < 2 ? p + 1 : (p == 2 ? 2 : 3));
  return sum;
}

}  // namespace qcb
