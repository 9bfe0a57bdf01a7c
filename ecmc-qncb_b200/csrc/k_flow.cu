// k_flow.cu — the update of a Wilson-flow RK3 stage, from the loops of its source links.
//
// Reference: GradientFlow (src/flow/gradient_flow.cpp:15-128) runs five full-lattice loops
// per step (compute_force, compute_w1, compute_force, compute_w2, replace_force_0,
// compute_force, compute_w3) over three full GaugeField copies, with a halo exchange after
// every W update.  Each stage here is two kernels: the plaquette loops of the links (k_loops.cu),
// and this one, which takes each link's force from them and applies the stage (flow_link.cuh).
// Links are double-buffered (src -> dst) because every stage reads neighbours of the
// previous stage; the force accumulator holds 8 reals per link.
//
// Measured per RK3 step on 32^4, against kernels that multiplied out the staples of every link
// (twelve products each; in FP32 ten, with one product shared by a plane's two links), in turn on one
// box: FP64 18-real 2.71 -> 2.00 ms, FP32 12-real 1.05 -> 0.91 ms.  Of an FP32 stage, the loops take
// 110 us and the update 187 to 214 (0.71-0.85 GB of DRAM traffic, 68% issue).  A smaller loop buffer, whose
// rounds of slices would stay in L2, costs more in half-filled last waves than it saves: 110, 70 and
// 24 MB made the FP32 step 1.05, 1.09 and 1.24 ms where 1 GiB made it 0.97.
#include "flow_launch.cuh"
#include "flow_link.cuh"

namespace qcb {

// Four warps work on 32 sites of one parity.  Warp nu first moves the three loops K_{mu nu}(x-nu) up
// along U_nu(x-nu), which it loads and completes once, into shared memory; then warp mu sums its link's
// force from them and applies the stage.  (18-real: the test whether U_nu(x-nu) is unitary is hidden, RK3
// step of 20x24x28x36 FP64 880 us with and without; with every link off, 1400 us.)
#ifndef QCB_FLOW_MINB32
#define QCB_FLOW_MINB32 5
#endif
#ifndef QCB_FLOW_MINB64
#define QCB_FLOW_MINB64 3
#endif
template <typename S, int NR, int STAGE, bool MULTI>
__global__ void __launch_bounds__(FLOW_THREADS, sizeof(S) == 4 ? QCB_FLOW_MINB32 : QCB_FLOW_MINB64)
    k_flow_update(const __grid_constant__ FlowLat one, const FlowLat* __restrict__ lats,
                  const uint32_t* __restrict__ prefix, int nlat, int swap, int step) {
  typedef arith_t<S> R;
  typedef Links<S, NR> F;
  pdl_wait();
  const int l = MULTI ? lattice_of(prefix, nlat, blockIdx.x) : 0;
  const FlowLat& L = MULTI ? lats[l] : one;
  if (MULTI && step >= L.nsteps) return;
  const uint32_t b = MULTI ? blockIdx.x - __ldg(&prefix[l]) : blockIdx.x;
  const F src = flow_links<S, NR>(L, swap), dst = flow_links<S, NR>(L, swap ^ 1);
  AlgField<S> acc;
  acc.p = reinterpret_cast<typename AlgField<S>::V*>(L.acc);
  acc.stride = L.g.stride;
  const Loops<S> K(L.k, L.g);
  typedef typename AlgStore<S>::V V;
  constexpr int NC = AlgStore<S>::NC;
  __shared__ V moved[12][NC][32];  // [3 nu + k]: loop k of direction nu, moved to x
  const uint32_t n = (uint32_t)(L.t1 - L.t0) * K.half, first = (b >> 1) * L.tile;
  const int par = (int)(b & 1), w = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const R eps = R(S(L.eps));
  for (uint32_t k0 = 0; k0 < L.tile && first + k0 < n; k0 += 32) {
    const uint32_t k = first + k0 + lane;
    const uint32_t i = (uint32_t)L.t0 * K.half + k;
    const bool on = k < n;
    if (k0) __syncthreads();
    alg8<R> Z, Z0;
    m3<R> U;
    if (on) {
      const Coord x = cb_coord(L.g, par, i);
      {
        alg8<R> m[3];
        transported<F, S, R>(L.g, src, K, x, w, par, m);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          V v[NC];
          S* q = reinterpret_cast<S*>(v);
#pragma unroll
          for (int a = 0; a < 8; ++a) q[a] = S(m[j].a[a]);
#pragma unroll
          for (int c = 0; c < NC; ++c) moved[3 * w + j][c][lane] = v[c];
        }
      }
      // -sum_nu of K_{mu nu}(x), mu = w
      const uint32_t jx = K.at(i, x.c[3], x.c[3]);
#pragma unroll
      for (int a = 0; a < 8; ++a) Z.a[a] = R(0);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int nu = j + (j >= w);
        const alg8<R> A = K.template load<R>(nu > w ? plane_of(w, nu) : plane_of(nu, w), par, jx);
        add_alg(Z, A, nu > w ? R(-1) : R(1));
      }
      if (STAGE != 1) Z0 = acc.template load<R>(w, par, i);
      U = src.template load<R>(w, par, i);
    }
    __syncthreads();
    if (on) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int nu = j + (j >= w);
        V v[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) v[c] = moved[3 * nu + w - (w > nu)][c][lane];
        const S* q = reinterpret_cast<const S*>(v);
        alg8<R> B;
#pragma unroll
        for (int a = 0; a < 8; ++a) B.a[a] = R(q[a]);
        add_alg(Z, B, nu > w ? R(1) : R(-1));
      }
      const alg8<R> X = flow_x<STAGE, AlgField<S>, R>(acc, Z, Z0, eps, w, par, i);
      m3<R> Un = flow_product<F, R>(flow_exp(X), U);
      flow_reunit<R>(Un, STAGE);
      dst.template store<R>(w, par, i, Un);
    }
  }
}

// The stage without loops: one thread per link, its staples multiplied out.  RK3 step of 20x24x28x36:
// FP64 18-real 1350 us (880 with loops), FP32 12-real 555 (440).
template <typename S, int NR>
__global__ void __launch_bounds__(FLOW_THREADS, sizeof(S) == 4 ? 4 : 2)
    k_flow_links(const __grid_constant__ FlowLat L, int swap, int stage) {
  typedef arith_t<S> R;
  typedef Links<S, NR> F;
  pdl_wait();
  const uint32_t half = (uint32_t)(L.g.str[3] >> 1), n = (uint32_t)(L.t1 - L.t0) * half,
                 k = (blockIdx.x >> 1) * FLOW_THREADS + threadIdx.x;
  if (k >= n) return;
  const int par = (int)(blockIdx.x & 1), mu = (int)blockIdx.y;
  const uint32_t i = (uint32_t)L.t0 * half + k;
  const F src = flow_links<S, NR>(L, swap), dst = flow_links<S, NR>(L, swap ^ 1);
  AlgField<S> acc;
  acc.p = reinterpret_cast<typename AlgField<S>::V*>(L.acc);
  acc.stride = L.g.stride;
  const m3<R> A = staple_sum_rt<F, R>(L.g, src, cb_coord(L.g, par, i), mu, par, i);
  const m3<R> U = src.template load<R>(mu, par, i);
  alg8<R> Z = proj_ta(mul_nn(U, A)), Z0;
#pragma unroll
  for (int a = 0; a < 8; ++a) Z.a[a] = -Z.a[a];
  if (stage != 1) Z0 = acc.template load<R>(mu, par, i);
  const R eps = R(S(L.eps));
  alg8<R> X;
  if (stage == 1)
    X = flow_x<1, AlgField<S>, R>(acc, Z, Z0, eps, mu, par, i);
  else if (stage == 2)
    X = flow_x<2, AlgField<S>, R>(acc, Z, Z0, eps, mu, par, i);
  else
    X = flow_x<3, AlgField<S>, R>(acc, Z, Z0, eps, mu, par, i);
  m3<R> Un = flow_product<F, R>(flow_exp(X), U);
  flow_reunit<R>(Un, stage);
  dst.template store<R>(mu, par, i, Un);
}

template <typename S, int NR>
static cudaError_t flow_links_impl(const FlowLat& r, int stage, int swap, cudaStream_t st) {
  const uint32_t n = (uint32_t)(r.t1 - r.t0) * (uint32_t)(r.g.str[3] >> 1);
  return pdl_launch(k_flow_links<S, NR>, dim3(2 * ((n + FLOW_THREADS - 1) / FLOW_THREADS), 4), FLOW_THREADS, st, r, swap,
                    stage);
}

cudaError_t launch_flow_links(const FlowLat& r, int prec, int nr, int stage, int swap, cudaStream_t st) {
  if (stage < 1 || stage > 3) return cudaErrorInvalidValue;
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  QCB_DISPATCH_STORE(probe, flow_links_impl, r, stage, swap, st);
}

template <typename S, int NR>
static cudaError_t update_impl(const FlowSet& s, int stage, int swap, int step, cudaStream_t st) {
  if (s.blocks == 0) return cudaSuccess;
  void (*kern)(const FlowLat, const FlowLat*, const uint32_t*, int, int, int) =
      s.lats ? (stage == 1 ? k_flow_update<S, NR, 1, true>
                           : (stage == 2 ? k_flow_update<S, NR, 2, true> : k_flow_update<S, NR, 3, true>))
             : (stage == 1 ? k_flow_update<S, NR, 1, false>
                           : (stage == 2 ? k_flow_update<S, NR, 2, false> : k_flow_update<S, NR, 3, false>));
  return pdl_launch(kern, dim3(s.blocks), FLOW_THREADS, st, s.one, s.lats, s.prefix, s.nlat, swap, step);
}

cudaError_t launch_flow_update(const FlowSet& s, int prec, int nr, int stage, int swap, int step, cudaStream_t st) {
  if (stage < 1 || stage > 3) return cudaErrorInvalidValue;
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  QCB_DISPATCH_STORE(probe, update_impl, s, stage, swap, step, st);
}

}  // namespace qcb
