// k_loops.cu — the plaquette-loop field of a lattice, and the clover Q and E summed from it.
//
// References: clover_site, local_q_e_clover and topo_q_e_clover(_global)
// (src/observables/observables_mpi.cpp:61-150) for Q and E; the loops also carry the force of
// the Wilson flow (loops.cuh).
#include <algorithm>

#include "flow_launch.cuh"
#include "reduce.cuh"

namespace qcb {

// ---- the loop buffer --------------------------------------------------------------------
static size_t loops_stride(const Geom& g, int slices) {
  return ((size_t)slices * (size_t)(g.str[3] / 2) + 63) / 64 * 64;
}
static size_t index_bytes(int prec) { return (size_t)(6 * 2 * 9) * (prec == QCB_PREC_FP64 ? 8 : 4) + 4 * 2; }
size_t loops_bytes(const Geom& g, int prec, int slices) { return loops_stride(g, slices) * index_bytes(prec); }
int loops_slices(const Geom& g, int prec, size_t bytes) {
  if (loops_bytes(g, prec, g.L[3]) <= bytes) return g.L[3];
  // the padding of the stride is that of all slices together, so the estimate leaves it out
  const size_t most = bytes / ((size_t)(g.str[3] / 2) * index_bytes(prec));
  int n = (int)std::min(most, (size_t)(g.L[3] - 1));
  while (n >= 2 && loops_bytes(g, prec, n) > bytes) --n;
  return n >= 2 ? n : 0;
}
cudaError_t loops_reserve(LoopBuf* buf, size_t want, size_t least) {
  auto alloc = [](size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, n) == cudaSuccess) return p;
    cudaGetLastError();
    return (void*)nullptr;
  };
  return loops_grow(buf, want, least, alloc, [](void* p) { cudaFree(p); }) ? cudaSuccess : cudaErrorMemoryAllocation;
}
LoopDev loops_view(const LoopBuf& buf, size_t off, const Geom& g, int prec, int slices) {
  const size_t es = prec == QCB_PREC_FP64 ? 8 : 4, st = loops_stride(g, slices);
  LoopDev k = {};
  if (slices == 0) return k;
  k.p = (char*)buf.p + off;
  k.tr = (char*)buf.p + off + 6 * 2 * 8 * st * es;
  k.off = (uint8_t*)buf.p + off + 6 * 2 * 9 * st * es;
  k.stride = (uint32_t)st;
  k.slices = slices;
  return k;
}

std::vector<FlowLat> flow_rounds(const LatDev& L, const LoopDev& k) {
  std::vector<FlowLat> out;
  const Geom& g = L.g;
  const bool whole = g.tlo == 0 && g.thi == g.L[3] - 1;
  FlowLat r;
  r.g = g;
  r.a = L.links;
  r.b = r.acc = nullptr;
  r.k = k;
  r.eps = 0.0;
  r.tile = 32;
  r.nsteps = 1 << 30;
  const bool full = k.slices >= g.L[3];
  if (!k.p) {
    r.t0 = g.tlo;
    r.t1 = g.thi + 1;
    r.kt0 = r.kn = 0;
    return {r};
  }
  for (int t = g.tlo; t <= g.thi;) {
    const int room = full ? g.L[3] : k.slices - 1;  // one slot holds the slice before the round
    r.t0 = t;
    r.t1 = t + room <= g.thi ? t + room : g.thi + 1;
    if (full && whole) {
      r.kt0 = 0;
      r.kn = g.L[3];
    } else {
      r.kt0 = t == g.tlo ? t - 1 : t;
      r.kn = r.t1 - r.kt0;
    }
    out.push_back(r);
    t = r.t1;
  }
  return out;
}

static uint32_t tiles_of(const Geom& g, int slices, uint32_t tile) {
  return ((uint32_t)slices * (uint32_t)(g.str[3] / 2) + tile - 1) / tile;
}
uint32_t loops_blocks(const FlowLat& r) { return tiles_of(r.g, r.kn, FLOW_THREADS / 2); }
uint32_t qe_blocks(const FlowLat& r) { return tiles_of(r.g, r.t1 - r.t0, FLOW_THREADS / 2); }
uint32_t update_blocks(const FlowLat& r) { return 2 * tiles_of(r.g, r.t1 - r.t0, r.tile); }  // both parities

// ---- the loops --------------------------------------------------------------------------
// One thread per site and grid row: row y of n takes planes y, y + n, ...; the planes run
// through one body that is not unrolled.  Measured on 32^4 FP32 12-real: 110 us, 0.37 GB of DRAM
// traffic (the links read and the loops written once), bound by the FP32 pipes and by the latency
// of its sixteen links; FP64 18-real 250 us.  Six rows instead of one make a small lattice's few
// blocks six times as many; from 2048 blocks the chip is full without that, and one row reads
// the site's own links once for all its planes.
template <typename S, int NR, bool TRACE>
__device__ __forceinline__ void loops_site(const FlowLat& L, const Links<S, NR>& f, int par, uint32_t j) {
  typedef arith_t<S> R;
  const Loops<S> K(L.k, L.g);
  int32_t ii = (int32_t)(j + (uint32_t)L.kt0 * K.half);
  const bool before = ii < 0;  // the slice before 0 is the last one
  if (before) ii += (int32_t)L.g.Vh;
  const uint32_t i = (uint32_t)ii;
  const Coord x = cb_coord(L.g, par, i);
  const NbOff o = nb_offsets(L.g, x);
  const uint32_t jx = K.at(i, x.c[3], before ? -1 : x.c[3]);
  m3<R> U;
  int have = -1;
#pragma unroll 1
  for (int p = blockIdx.y; p < 6; p += gridDim.y) {
    const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2), nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
    if (mu != have) U = lead<Links<S, NR>, R>(f, mu, par, i);
    have = mu;
    if constexpr (NR == 18 && TRACE) {  // each link once: U_0, U_3, U_1, U_2
      if (p == 0 || p == 3 || p == 5) K.store_off(mu, par, jx, off_unitary<S>(U));
      if (p == 2) K.store_off(3, par, jx, off_unitary<S>(f.template load<R>(3, par, i)));
    }
    const m3<R> W = plaquette_loop<Links<S, NR>, R>(f, U, mu, nu, par, i, cb_index((uint32_t)((int32_t)x.s + sel4(o.up, mu))),
                                                    cb_index((uint32_t)((int32_t)x.s + sel4(o.up, nu))));
    K.template store<R>(p, par, jx, proj_ta(W));
    if (TRACE) K.template store_tr<R>(p, par, jx, W.e[0][0].im + W.e[1][1].im + W.e[2][2].im);
  }
}

#ifndef QCB_LOOPS_MINB32
#define QCB_LOOPS_MINB32 5
#endif
#ifndef QCB_LOOPS_MINB64
#define QCB_LOOPS_MINB64 3
#endif
template <typename S, int NR, bool TRACE, bool MULTI>
__global__ void __launch_bounds__(FLOW_THREADS, sizeof(S) == 4 ? QCB_LOOPS_MINB32 : QCB_LOOPS_MINB64)
    k_loops(const __grid_constant__ FlowLat one, const FlowLat* __restrict__ lats, const uint32_t* __restrict__ prefix,
            int nlat, int swap, int step) {
  pdl_wait();
  const int l = MULTI ? lattice_of(prefix, nlat, blockIdx.x) : 0;
  const FlowLat& L = MULTI ? lats[l] : one;
  if (MULTI && step >= L.nsteps) return;
  const uint32_t b = MULTI ? blockIdx.x - __ldg(&prefix[l]) : blockIdx.x;
  const Links<S, NR> f = flow_links<S, NR>(L, swap);
  const uint32_t n = (uint32_t)L.kn * (uint32_t)(L.g.str[3] >> 1), k = block_site(b);
  if (k < n) loops_site<S, NR, TRACE>(L, f, block_parity(), k);
}

template <typename S, int NR>
static cudaError_t loops_impl(const FlowSet& s, bool trace, int swap, int step, cudaStream_t st) {
  if (s.blocks == 0) return cudaSuccess;
  auto kern = s.lats ? (trace ? k_loops<S, NR, true, true> : k_loops<S, NR, false, true>)
                     : (trace ? k_loops<S, NR, true, false> : k_loops<S, NR, false, false>);
  const unsigned rows = s.blocks >= 2048 ? 1 : (s.blocks >= 512 ? 3 : 6);
  return pdl_launch(kern, dim3(s.blocks, rows), FLOW_THREADS, st, s.one, s.lats, s.prefix, s.nlat, swap, step);
}

cudaError_t launch_loops(const FlowSet& s, int prec, int nr, bool trace, int swap, int step, cudaStream_t st) {
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  QCB_DISPATCH_STORE(probe, loops_impl, s, trace, swap, step, st);
}

// ---- Q and E ------------------------------------------------------------------------------
// Unscaled clover sums q_site = tr F01 F23 - tr F02 F13 + tr F03 F12 and e_site = sum_{mu<nu}
// |F_mu nu|^2 (the 1/(4 pi^2) and 1/2 are applied to the totals).  The six planes run through
// one body, in the pairs (01, 23), (02, 13), (03, 12); each pair's share is added in FP64.
// Three transports a plane where four leaves were nine products: Q and E of 32^4 alone, loops
// included, FP32 12-real 442 -> 315 us, FP64 18-real 1073 -> 680 us; with the loops already there
// for an RK3 step, FP32 187 us more.
// In 18-real storage the bytes of the links that are not unitary are read first, for all planes
// together: 20x24x28x36 with SU(3) links FP64 296 us without the test, 320 with it (335 with the
// bytes read plane by plane); links that need the products 530, FP32 200, 217 and 312.
template <typename S, int NR>
__device__ __forceinline__ void qe_site(const FlowLat& L, const Links<S, NR>& f, int par, uint32_t i, double* q,
                                        double* e) {
  typedef arith_t<S> R;
  const Loops<S> K(L.k, L.g);
  const Coord x = cb_coord(L.g, par, i);
  const NbOff o = nb_offsets(L.g, x);
  unsigned bad = 0;
  if constexpr (NR == 18) {
    const int t = x.c[3], tm = t == 0 ? L.g.L[3] - 1 : t - 1;
    bool side[4];  // U_d(x-d)
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const uint32_t k = (uint32_t)((int32_t)x.s + o.dn[d]) >> 1;
      side[d] = K.load_off(d, par ^ 1, d == 3 ? K.at(k, tm, t - 1) : K.at(k, t, t));
    }
#pragma unroll
    for (int p = 0; p < 6; ++p) {
      const int mu = p < 3 ? 0 : (p < 5 ? 1 : 2), nu = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
      const uint32_t k = (uint32_t)((int32_t)x.s + o.dn[mu] + o.dn[nu]) >> 1;
      const bool far = K.load_off(nu, par, nu == 3 ? K.at(k, tm, t - 1) : K.at(k, t, t));
      if (side[mu] || side[nu] || far) bad |= 1u << p;
    }
  }
  ah9<R> prev;
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    const int h = p >> 1;
    const int mu = (p & 1) == 0 ? 0 : (h == 0 ? 2 : 1), nu = (p & 1) == 0 ? h + 1 : (h == 2 ? 2 : 3);
    const bool multiply = (bad >> plane_of(mu, nu)) & 1;
    const ah9<R> F = clover_plane<Links<S, NR>, S, R>(f, K, x, o, mu, nu, par, i, L.g.L[3], multiply);
    *e += (double)sqnorm_ah(F);
    if (p & 1) {
      const double t = (double)re_tr_ah(prev, F);
      *q += h == 1 ? -t : t;
    } else {
      prev = F;
    }
  }
}

#ifndef QCB_QE_MINB32
#define QCB_QE_MINB32 5
#endif
#ifndef QCB_QE_MINB64
#define QCB_QE_MINB64 3
#endif
template <typename S, int NR, bool MULTI>
__global__ void __launch_bounds__(FLOW_THREADS, sizeof(S) == 4 ? QCB_QE_MINB32 : QCB_QE_MINB64)
    k_loops_qe(const __grid_constant__ FlowLat one, const FlowLat* __restrict__ lats,
               const uint32_t* __restrict__ prefix, int nlat, int swap, double* __restrict__ parts, uint32_t first,
               uint32_t nparts) {
  __shared__ double sh[FLOW_THREADS / 32];
  pdl_wait();
  const int l = MULTI ? lattice_of(prefix, nlat, blockIdx.x) : 0;
  const FlowLat& L = MULTI ? lats[l] : one;
  const uint32_t b = MULTI ? blockIdx.x - __ldg(&prefix[l]) : blockIdx.x;
  const Links<S, NR> f = flow_links<S, NR>(L, swap);
  const uint32_t half = (uint32_t)(L.g.str[3] >> 1), n = (uint32_t)(L.t1 - L.t0) * half,
                 k = block_site(b);
  double q = 0.0, e = 0.0;
  if (k < n) qe_site<S, NR>(L, f, block_parity(), (uint32_t)L.t0 * half + k, &q, &e);
  const double bq = block_sum<FLOW_THREADS>(q, sh);
  const double be = block_sum<FLOW_THREADS>(e, sh);
  if (threadIdx.x == 0) {
    parts[first + blockIdx.x] = bq;
    parts[nparts + first + blockIdx.x] = be;
  }
}

// F_{mu nu} = (C - C^dag) / 8 of the plaquette leaf M: its share.
template <typename R>
__device__ __forceinline__ void add_leaf(ah9<R>& F, const m3<R>& M, R sg) {
#pragma unroll
  for (int k = 0; k < 3; ++k) F.d[k] = fma(R(0.25) * sg, M.e[k][k].im, F.d[k]);
  const int a[3] = {0, 0, 1}, b[3] = {1, 2, 2};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    F.o[k].re = fma(R(0.125) * sg, M.e[a[k]][b[k]].re - M.e[b[k]][a[k]].re, F.o[k].re);
    F.o[k].im = fma(R(0.125) * sg, M.e[a[k]][b[k]].im + M.e[b[k]][a[k]].im, F.o[k].im);
  }
}

// Q and E without loops: the four leaves of every plane multiplied out (twelve products).  20x24x28x36:
// FP64 18-real 467 us (323 with loops), FP32 12-real 298 (172).
template <typename S, int NR>
__global__ void __launch_bounds__(FLOW_THREADS, sizeof(S) == 4 ? 4 : 2)
    k_clover(const __grid_constant__ FlowLat L, int swap, double* __restrict__ parts, uint32_t first, uint32_t nparts) {
  typedef arith_t<S> R;
  typedef Links<S, NR> F;
  __shared__ double sh[FLOW_THREADS / 32];
  pdl_wait();
  const F f = flow_links<S, NR>(L, swap);
  const uint32_t half = (uint32_t)(L.g.str[3] >> 1), n = (uint32_t)(L.t1 - L.t0) * half, k = block_site(blockIdx.x);
  const int par = block_parity(), opp = par ^ 1;
  double q = 0.0, e = 0.0;
  if (k < n) {
    const uint32_t i = (uint32_t)L.t0 * half + k;
    const Coord x = cb_coord(L.g, par, i);
    const NbOff o = nb_offsets(L.g, x);
    const int32_t s = (int32_t)x.s;
    ah9<R> prev;
#pragma unroll 1
    for (int p = 0; p < 6; ++p) {
      const int h = p >> 1;
      const int mu = (p & 1) == 0 ? 0 : (h == 0 ? 2 : 1), nu = (p & 1) == 0 ? h + 1 : (h == 2 ? 2 : 3);
      const int32_t umu = sel4(o.up, mu), unu = sel4(o.up, nu), dmu = sel4(o.dn, mu), dnu = sel4(o.dn, nu);
      const uint32_t imu = cb_index((uint32_t)(s + dmu)), inu = cb_index((uint32_t)(s + dnu)),
                     imn = cb_index((uint32_t)(s + dmu + dnu)), iun = cb_index((uint32_t)(s + dmu + unu)),
                     ium = cb_index((uint32_t)(s + dnu + umu));
      ah9<R> A = {};
      const m3<R> G = mul_nn(f.template load<R>(mu, par, i), f.template load<R>(nu, opp, cb_index((uint32_t)(s + umu))));
      const m3<R> H = mul_nn(f.template load<R>(nu, par, i), f.template load<R>(mu, opp, cb_index((uint32_t)(s + unu))));
      add_leaf(A, mul_na(G, H), R(1));
      add_leaf(A, loop_beside<F, R>(f, nu, mu, opp, imu, iun, i), R(-1));
      add_leaf(A, loop_across<F, R>(f, mu, nu, par, imn, inu, imu), R(1));
      add_leaf(A, loop_beside<F, R>(f, mu, nu, opp, inu, ium, i), R(1));
      e += (double)sqnorm_ah(A);
      if (p & 1) {
        const double t = (double)re_tr_ah(prev, A);
        q += h == 1 ? -t : t;
      } else {
        prev = A;
      }
    }
  }
  const double bq = block_sum<FLOW_THREADS>(q, sh);
  const double be = block_sum<FLOW_THREADS>(e, sh);
  if (threadIdx.x == 0) {
    parts[first + blockIdx.x] = bq;
    parts[nparts + first + blockIdx.x] = be;
  }
}

template <typename S, int NR>
static cudaError_t clover_impl(const FlowLat& r, int swap, double* parts, uint32_t first, uint32_t n, cudaStream_t st) {
  return pdl_launch(k_clover<S, NR>, dim3(qe_blocks(r)), FLOW_THREADS, st, r, swap, parts, first, n);
}

cudaError_t launch_clover(const FlowLat& r, int prec, int nr, int swap, double* parts, uint32_t first, uint32_t n,
                          cudaStream_t st) {
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  QCB_DISPATCH_STORE(probe, clover_impl, r, swap, parts, first, n, st);
}

template <typename S, int NR>
static cudaError_t loops_qe_impl(const FlowSet& s, int swap, double* parts, uint32_t first, uint32_t n,
                                 cudaStream_t st) {
  if (s.blocks == 0) return cudaSuccess;
  auto kern = s.lats ? k_loops_qe<S, NR, true> : k_loops_qe<S, NR, false>;
  return pdl_launch(kern, dim3(s.blocks), FLOW_THREADS, st, s.one, s.lats, s.prefix, s.nlat, swap, parts, first, n);
}

cudaError_t launch_loops_qe(const FlowSet& s, int prec, int nr, int swap, double* parts, uint32_t first, uint32_t n,
                            cudaStream_t st) {
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  QCB_DISPATCH_STORE(probe, loops_qe_impl, s, swap, parts, first, n, st);
}

}  // namespace qcb
