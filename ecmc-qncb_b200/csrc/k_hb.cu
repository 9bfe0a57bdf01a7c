// k_hb.cu — checkerboarded Cabibbo-Marinari heatbath pass.
//
// Reference path: mpi::heatbathcb::hit (src/heatbath/heatbath_mpi.cpp:11-34) with
// heatbath::su2_step and generate_su2_kp (src/heatbath/heatbath.cpp:8-44), applied by
// mpi::heatbathcb::sweep (heatbath_mpi.cpp:37-56) to every non-frozen link in
// lexicographic order.  Here one pass updates all links U_mu(x) with x of one parity:
// their staples only touch links of other directions or of U_mu at the opposite parity,
// so the updates of a pass are independent and run one thread per link.
//
// Per link: staple A once (it does not change between hits), then for each hit and each
// subgroup (0,1), (1,2), (0,2):
//   W = U A restricted to the 2x2 block, w = quaternion of the block (su2_to_quaternion,
//   src/su3/utils.cpp:47-50), k = |w|, v = w/k; x ~ KP(alpha = 2 beta k / 3);
//   r = x v^dagger (utils.cpp:53-63); U <- embed_ij(r) U (utils.cpp:33-44), touching rows
//   i and j only.
#include "dispatch.cuh"
#include "hb_link.cuh"
#include "hb_quad.cuh"
#include "obs_site.cuh"
#include "reduce.cuh"
#include "sync.cuh"

namespace qcb {

// Blocks of 128 threads.  Resident blocks per SM (the register bound): FP32 5 (96
// registers, measured 2.6% faster than 4 on 32^4), FP64 3 (2.6% faster than 4, 2 slower).
#ifndef QCB_HB_MINB32
#define QCB_HB_MINB32 5
#endif
#ifndef QCB_HB_MINB64
#define QCB_HB_MINB64 3
#endif
template <typename S>
struct HbMinBlocks {
  static constexpr int value = sizeof(S) == 4 ? QCB_HB_MINB32 : QCB_HB_MINB64;
};

// Frozen links of the reference's block decomposition (src/geometry/GeometryCB.cpp:33-56)
// after a cumulative translation of the field by `shift`: link (x, mu) with
// (x_d + shift_d) % lcore == 0 for some d != mu is not updated.  The other links of a pass are
// numbered without gaps, so that no lane idles (with l_core = 6, 42% of a pass's links are frozen):
// along d != mu the positions k lcore + 1 + r, r < lcore - 1, and along mu every second site, by
// the parity of the rest.  A pass on 48^4, FP32 12-real, l_core 6: 261 us with the
// frozen links' lanes idle, 198 so; on 32^4, l_core 4, 51 -> 37, FP64 18-real 129 -> 102; on
// 12x18x24x30, FP32 18-real, two hits, 20.4 -> 17.8 (one partial wave).
struct ActiveLinks {
  int lcore;                // 0: every link is updated
  int shift[4];             // each in [0, lcore)
  uint32_t n;               // links of the pass
  uint32_t ext[3], rcp[3];  // extents along x, y, z, and their reciprocals (divmod_rcp)
  uint32_t rcp_run;         // the reciprocal of lcore - 1
};

static uint32_t rcp_of(uint32_t d) { return d <= 1 ? 0xFFFFFFFFu : (uint32_t)((1ull << 32) / d); }

static ActiveLinks active_links(const Geom& g, int mu, const int* frozen) {
  ActiveLinks m = {};
  m.n = g.Vh;
  if (!frozen || frozen[0] <= 0) return m;
  m.lcore = frozen[0];
  m.n = 1;
  for (int d = 0; d < 4; ++d) {
    m.shift[d] = frozen[1 + d];
    const uint32_t e = (uint32_t)(d == mu ? g.L[d] / 2 : g.L[d] / m.lcore * (m.lcore - 1));
    m.n *= e;
    if (d < 3) m.ext[d] = e, m.rcp[d] = rcp_of(e);
  }
  m.rcp_run = rcp_of((uint32_t)m.lcore - 1);
  return m;
}

// Site of link j of pass (mu, par).
__device__ __forceinline__ Coord active_site(const Geom& g, const ActiveLinks& m, int mu, int par, uint32_t j) {
  uint32_t a[4];
  uint32_t q = j;
#pragma unroll
  for (int d = 0; d < 3; ++d) q = divmod_rcp(q, m.ext[d], m.rcp[d], &a[d]);
  a[3] = q;
  Coord r;
  int sum = par;
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    uint32_t rem;
    const uint32_t k = divmod_rcp(a[d], (uint32_t)m.lcore - 1, m.rcp_run, &rem);
    int x = (int)(k * (uint32_t)m.lcore + 1 + rem) - m.shift[d];
    if (x < 0) x += g.L[d];
    if (d != mu) sum += x;
    r.c[d] = x;
  }
#pragma unroll
  for (int d = 0; d < 4; ++d)
    if (d == mu) r.c[d] = 2 * (int)a[d] + (sum & 1);
  r.s = (uint32_t)r.c[0] + (uint32_t)g.L[0] * ((uint32_t)r.c[1] + (uint32_t)g.L[1] * ((uint32_t)r.c[2] + (uint32_t)g.L[2] * (uint32_t)r.c[3]));
  return r;
}

template <typename S, int NR, int MU, bool FROZEN>
__global__ void __launch_bounds__(128, HbMinBlocks<S>::value) k_hb_pass(Geom g, Links<S, NR> f, int par, S beta, uint32_t k0,
                                                 uint32_t k1, uint32_t sweep, int n_hits, uint32_t* status,
                                                 ActiveLinks act) {
  pdl_wait();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= act.n) return;
  uint32_t fails;
  if (FROZEN) {
    const Coord x = active_site(g, act, MU, par, i);
    fails = hb_update_at<Links<S, NR>, arith_t<S>, NR, MU>(g, f, x, par, cb_index(x.s), arith_t<S>(beta), k0, k1, sweep,
                                                          n_hits);
  } else {
    fails = hb_update_link<Links<S, NR>, arith_t<S>, NR, MU>(g, f, par, i, arith_t<S>(beta), k0, k1, sweep, n_hits);
  }
  if (fails) atomicAdd(status, fails);
}

// Pass (mu, par) with four lanes per link (FP64 18-real), for lattices whose links do not fill the
// chip.  The direction is a run-time value: the time is one link's latency.
template <bool FROZEN>
__global__ void __launch_bounds__(128) k_hb_quad(Geom g, Links<double, 18> f, int mu, int par, double beta, uint32_t k0,
                                                 uint32_t k1, uint32_t sweep, int n_hits, uint32_t* status,
                                                 ActiveLinks act) {
  pdl_wait();
  const uint32_t j = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  if (j >= act.n) return;
  const Coord x = FROZEN ? active_site(g, act, mu, par, j) : cb_coord(g, par, j);
  const uint32_t i = cb_index(x.s);
  if (!own_site(g, x.c[3])) return;  // halo slice of a slab
  const Quad q;
  const uint32_t fails = hb_update_quad<Links<double, 18>, false>(q, g, f, x, mu, par, i, beta, k0, k1, sweep, n_hits,
                                                                  nullptr);
  if (fails && q.lane == 0) atomicAdd(status, fails);
}

// Four lanes per link while all of a pass's links are then resident at once (148 SMs of three
// blocks of 32 links): 12x12x12x16 (13824 links) takes 12.1 us against 12.4,
// 12x12x14x16 (16128) 18.8 against 12.6; 8^4 9.0 against 11.6.
static bool quad_pass(const LatDev& L, uint32_t links) {
  return L.prec == QCB_PREC_FP64 && L.nr == 18 && links <= 148u * 3u * 32u;
}

// Launch with programmatic stream serialization: the pass's blocks become resident while the
// previous kernel drains and wait in pdl_wait() (pass on 16^4 FP32-12, us: 9.6 without, 7.1).
template <typename S, int NR, int MU>
static cudaError_t hb_pass_launch(dim3 grid, int block, cudaStream_t s, const Geom& g, const Links<S, NR>& f, int par,
                                  S beta, uint32_t k0, uint32_t k1, uint32_t sweep, int n_hits, uint32_t* status,
                                  const ActiveLinks& act) {
  if (act.lcore > 0)
    return pdl_launch(k_hb_pass<S, NR, MU, true>, grid, block, s, g, f, par, beta, k0, k1, sweep, n_hits, status, act);
  return pdl_launch(k_hb_pass<S, NR, MU, false>, grid, block, s, g, f, par, beta, k0, k1, sweep, n_hits, status, act);
}

template <typename S, int NR>
static cudaError_t hb_pass_impl(const LatDev& L, int mu, int par, double beta, uint64_t seed, uint32_t sweep,
                                int n_hits, uint32_t* status, cudaStream_t s, int block, const int* frozen) {
  const ActiveLinks act = active_links(L.g, mu, frozen);
  if (act.n == 0) return cudaSuccess;  // l_core 1 freezes every link
  Links<S, NR> f;
  f.p = reinterpret_cast<typename Links<S, NR>::V*>(L.links);
  f.stride = L.g.stride;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  if constexpr (sizeof(S) == 8 && NR == 18)
    if (quad_pass(L, act.n))
      return pdl_launch(act.lcore > 0 ? k_hb_quad<true> : k_hb_quad<false>, dim3(grid_for(4 * (uint64_t)act.n, block)),
                        block, s, L.g, f, mu, par, beta, k0, k1, sweep, n_hits, status, act);
  dim3 grid(grid_for(act.n, block));
  switch (mu) {
    case 0: return hb_pass_launch<S, NR, 0>(grid, block, s, L.g, f, par, S(beta), k0, k1, sweep, n_hits, status, act);
    case 1: return hb_pass_launch<S, NR, 1>(grid, block, s, L.g, f, par, S(beta), k0, k1, sweep, n_hits, status, act);
    case 2: return hb_pass_launch<S, NR, 2>(grid, block, s, L.g, f, par, S(beta), k0, k1, sweep, n_hits, status, act);
    default: return hb_pass_launch<S, NR, 3>(grid, block, s, L.g, f, par, S(beta), k0, k1, sweep, n_hits, status, act);
  }
}

// The last pass (mu = 3, parity 1) of a measured sweep (whole lattices only).  Blocks 0 .. nb - 1: the
// updates of k_hb_pass, and per block the FP64 sum of Re tr(U_3 A_3) of its updated links.  After
// the pass of parity 0 the spatial links and the even U_3 links are final, so this pass sees final
// staples; every temporal plaquette holds exactly one odd U_3 link and is counted once.  The other
// blocks sum the spatial plaquettes, `rows` blocks side by side for the three planes of 128 sites.
// (Summed by the update's threads behind their links, in both passes, they cost on 32^4 FP64
// 18-real 354 us on top of the passes and FP32 12-real 92, more than all six planes of k_plaquette
// do; in blocks of their own 210 and 50.)
template <typename S, int NR>
__global__ void __launch_bounds__(128, HbMinBlocks<S>::value) k_hb_pass_meas(Geom g, Links<S, NR> f, S beta,
                                                                            uint32_t k0, uint32_t k1, uint32_t sweep,
                                                                            int n_hits, uint32_t* status, int nb,
                                                                            int rows, double* __restrict__ parts) {
  typedef arith_t<S> R;
  __shared__ double sh[4];
  pdl_wait();
  double v = 0.0;
  if ((int)blockIdx.x < nb) {
    const uint32_t i = blockIdx.x * 128 + threadIdx.x;
    R retr = 0;
    uint32_t fails = 0;
    if (i < g.Vh)
      fails = hb_update_at<Links<S, NR>, R, NR, 3, true>(g, f, cb_coord(g, 1, i), 1, i, R(beta), k0, k1, sweep, n_hits,
                                                         &retr);
    if (fails) atomicAdd(status, fails);
    v = (double)retr;
  } else {
    const uint32_t b = blockIdx.x - (uint32_t)nb, i = block_site(b / rows);
    const int par = block_parity();
    if (i < g.Vh)
      v = site_plaquettes<Links<S, NR>, R, true>(g, f, cb_coord(g, par, i), par, i, (int)(b % rows), rows, 3);
  }
  const double b = block_sum<128>(v, sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = b;
}

// Both passes mu = 3 with four lanes per link: lanes 0, 1, 2 also take one spatial plane each of the
// pass's sites.
__global__ void __launch_bounds__(128) k_hb_quad_meas(Geom g, Links<double, 18> f, int par, double beta, uint32_t k0,
                                                      uint32_t k1, uint32_t sweep, int n_hits, uint32_t* status,
                                                      double* __restrict__ parts) {
  __shared__ double sh[4];
  pdl_wait();
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
  double v = 0.0;
  uint32_t fails = 0;
  const Quad q;
  if (i < g.Vh) {
    const Coord x = cb_coord(g, par, i);
    double retr = 0;
    fails = hb_update_quad<Links<double, 18>, true>(q, g, f, x, 3, par, i, beta, k0, k1, sweep, n_hits, &retr);
    const double p = plaquette_plane<Links<double, 18>, double, true>(g, f, x, par, i, q.lane == 2 ? 1 : 0, q.lane == 0 ? 1 : 2);
    const double sum = q.get(p, 0) + q.get(p, 1) + q.get(p, 2);
    if (q.lane == 0) {
      v = sum;
      if (par) v += retr;
    }
  }
  if (fails && q.lane == 0) atomicAdd(status, fails);
  const double b = block_sum<128>(v, sh);
  if (threadIdx.x == 0) parts[blockIdx.x] = b;
}

cudaError_t launch_hb_pass(const LatDev& L, int mu, int parity, double beta, uint64_t seed, uint32_t sweep,
                           int n_hits, uint32_t* status, cudaStream_t s, int block, const int* frozen) {
  if (block <= 0) block = 128;
  QCB_DISPATCH_STORE(L, hb_pass_impl, L, mu, parity, beta, seed, sweep, n_hits, status, s, block, frozen);
}

// Planes side by side while all blocks then fit on the chip at once.
static int spatial_rows(const LatDev& L) { return 3 * grid_for(L.g.Vh, 64) <= 148 * 3 ? 3 : 1; }
int hb_meas_parts(const LatDev& L) {
  return quad_pass(L, L.g.Vh) ? 2 * (int)grid_for(4 * (uint64_t)L.g.Vh, 128)
                      : (int)grid_for(L.g.Vh, 128) + spatial_rows(L) * (int)grid_for(L.g.Vh, 64);
}

template <typename S, int NR>
static cudaError_t hb_meas_impl(const LatDev& L, double beta, uint64_t seed, uint32_t sweep, int n_hits,
                                uint32_t* status, double* parts, cudaStream_t s, int block, uint64_t* launches) {
  Links<S, NR> f;
  f.p = reinterpret_cast<typename Links<S, NR>::V*>(L.links);
  f.stride = L.g.stride;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  cudaError_t e = cudaSuccess;
  if constexpr (sizeof(S) == 8 && NR == 18)
    if (quad_pass(L, L.g.Vh)) {
      const dim3 grid(grid_for(4 * (uint64_t)L.g.Vh, 128));
      for (int par = 0; par < 2 && e == cudaSuccess; ++par)
        e = pdl_launch(k_hb_quad_meas, grid, 128, s, L.g, f, par, beta, k0, k1, sweep, n_hits, status,
                       parts + (size_t)par * grid.x);
      *launches += 2;
      return e;
    }
  e = launch_hb_pass(L, 3, 0, beta, seed, sweep, n_hits, status, s, block, nullptr);
  const int nb = (int)grid_for(L.g.Vh, 128), rows = spatial_rows(L);
  if (e == cudaSuccess)
    e = pdl_launch(k_hb_pass_meas<S, NR>, dim3(hb_meas_parts(L)), 128, s, L.g, f, S(beta), k0, k1, sweep, n_hits, status,
                   nb, rows, parts);
  *launches += 2;
  return e;
}

cudaError_t launch_hb_meas(const LatDev& L, double beta, uint64_t seed, uint32_t sweep, int n_hits, uint32_t* status,
                           double* parts, cudaStream_t s, int block, uint64_t* launches) {
  if (L.g.tlo != 0 || L.g.thi != L.g.L[3] - 1) return cudaErrorInvalidValue;  // whole lattices only
  QCB_DISPATCH_STORE(L, hb_meas_impl, L, beta, seed, sweep, n_hits, status, parts, s, block, launches);
}

}  // namespace qcb
