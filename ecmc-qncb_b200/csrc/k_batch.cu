// k_batch.cu — the persistent heatbath kernel that advances many independent lattices in one
// launch, and the sums of their observables.
//
// The reference runs one lattice per process (src/bin/gauge_hb_ncb.cpp:18-201).  Here a
// batch of lattices of different sizes and couplings shares one cooperative launch: the
// work of every lattice is cut into levels (checkerboard heatbath passes) and each level into
// tiles of sites.  Work items are ordered level-major across lattices, item j = (level, lattice,
// tile), and warp w of W processes items w, w+W, w+2W, ... in order.  Before an item of level k of lattice l starts, all tiles of level k-1 of the
// same lattice must be finished: a per-lattice counter done[l] counts finished tiles, and
// the warp waits (acquire) until done[l] >= k * ntiles[l].  Levels of different lattices
// overlap freely, so small lattices do not serialise the GPU.
//
// Progress: every item's dependencies have smaller indices, warps take their items in
// increasing order, and the cooperative launch makes all of them co-resident; so the
// smallest unfinished item always has its dependencies done.  Every wait is bounded by
// wall-clock time (WAIT_NS); a warp that gives up raises an abort flag that makes every
// other warp return, and the host reports the error.  Links are read with L2-coherent loads
// (LD_CG), because warps read links that other warps wrote in the same launch.
//
// Bound: at large batches the FP32 pipes, as a single lattice's pass; at small ones the latency of
// a level (one link's chain, then the counter's round trip).  An item is a warp's, not a block's:
// with block barriers around every item the slowest of four warps' draws held up the others, a
// default tile put two links behind one another on every thread, and the search for the item's
// lattice went through lines that the acquire had dropped from L1 (the prefix sums and the
// descriptor now lie in shared memory).  Six sweeps, FP32 12-real, items of a block -> of a warp:
// 54 lattices of 8^4 to 16^4 9.35 -> 8.45 ms, 64 of 8^4 to 12^4 2.85 -> 2.64 ms, one of 32^4
// 4.08 -> 3.91 ms, eight of 8^4 711 -> 323 us, 4^4 with 6^4 627 -> 314 us; FP64 18-real 64 of 8^4
// to 12^4 10.1 -> 8.8 ms, 32^4 13.7 -> 12.2 ms, eight of 8^4 1475 -> 780 us.
#include "batch.h"
#include "dispatch.cuh"
#include "hb_link.cuh"
#include "obs_site.cuh"
#include "reduce.cuh"
#include "sync.cuh"

// Resident blocks of 128 threads per SM (the register bound).  FP32: 4, where nothing spills; 5
// spills 100 bytes and took 10.2 ms where 4 takes 8.6, 3 takes 9.1 (54 lattices of 8^4 to 16^4).
// FP64: 2; 3 spills (8x8^4 835 us, 2: 780).
#ifndef QCB_BATCH_MINB32
#define QCB_BATCH_MINB32 4
#endif
#ifndef QCB_BATCH_MINB64
#define QCB_BATCH_MINB64 2
#endif

namespace qcb {

// Decode item r (within one level) into (lattice, tile) by binary search of prefix[].
__device__ __forceinline__ int find_lattice(const uint32_t* prefix, int nlat, uint32_t r) {
  int lo = 0, hi = nlat;  // prefix[lo] <= r < prefix[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= r)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// The calling warp waits until *done >= target; false (for the whole warp) on abort or timeout
// (limit_ns of wall-clock time or WAIT_MAX_ITERS polls).  status[1] counts timeouts, status[2] is
// the abort flag.
__device__ __forceinline__ bool warp_wait(const uint32_t* done, uint32_t target, uint32_t* status,
                                          uint64_t limit_ns = WAIT_NS) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = wait_geq(done, target, status, limit_ns) ? 1 : 0;
  __syncwarp();
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// Publish one finished tile of lattice l.
__device__ __forceinline__ void warp_release(uint32_t* done) {
  __threadfence();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) atomicAdd(done, 1u);
}

// ---- one work item ----------------------------------------------------------------------
// Heatbath level k: pass k % 8 (mu = pass / 2, parity = pass % 2) of sweep sweep0 + k / 8;
// item tile = a tile of that pass's sites.
template <typename S, int NR>
__device__ __forceinline__ uint32_t hb_item(const BatchRun& run, const BatchLat& B, uint32_t level, uint32_t tile) {
  typedef Links<S, NR, LD_CG> F;
  const uint32_t sweep = B.sweep0 + level / 8;
  const int pass = (int)(level & 7), mu = pass >> 1, par = pass & 1;
  F f;
  f.p = reinterpret_cast<typename F::V*>(B.links);
  f.stride = B.g.stride;
  const arith_t<S> beta = arith_t<S>(S(B.beta));
  const int n_hits = B.n_hits > 0 ? B.n_hits : run.n_hits;
  uint32_t fails = 0;
  for (uint32_t k = threadIdx.x & 31; k < B.tile; k += 32) {
    const uint32_t i = tile * B.tile + k;
    if (i >= B.g.Vh) break;
    fails += hb_update_link_rt<F, arith_t<S>, NR>(B.g, f, mu, par, i, beta, B.k0, B.k1, sweep, n_hits);
  }
  return fails;
}

// ---- the persistent kernel -----------------------------------------------------------------
// A lattice with B.nlev != 0 takes part in its first B.nlev levels only; its items at later
// levels are skipped (no wait, no release).  Only as many warps run as a level has items: then
// every warp keeps its item from level to level, and few poll.  They are spread over the blocks;
// where all warps have work, a block's warps take neighbouring items (their links share lines of
// L2: 8.44 ms, spread 8.65).
constexpr int PREFIX_SH = 1024;  // prefix sums kept in shared memory
template <typename S, int NR>
__global__ void __launch_bounds__(128, sizeof(S) == 4 ? QCB_BATCH_MINB32 : QCB_BATCH_MINB64) k_batch(BatchRun run) {
  __shared__ BatchLat slots[4];  // the descriptor of each warp's lattice
  __shared__ uint32_t prefix_sh[PREFIX_SH];
  const uint32_t* prefix = run.prefix;
  if (run.nlat < PREFIX_SH) {
    for (uint32_t k = threadIdx.x; k <= (uint32_t)run.nlat; k += blockDim.x) prefix_sh[k] = run.prefix[k];
    prefix = prefix_sh;
  }
  __syncthreads();
  const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  BatchLat& B = slots[w];
  const uint32_t warps = gridDim.x * nw, step = warps < run.per_level ? warps : run.per_level;
  uint32_t r = warps > run.per_level ? w * gridDim.x + blockIdx.x : blockIdx.x * nw + w;
  if (r >= step) return;
  uint32_t fails = 0, known = ~0u, local = 0, level = 0;
  int l = -1;
  for (;; r += step) {
    while (r >= run.per_level) {
      r -= run.per_level;
      ++level;
    }
    if (level >= run.nlevels) break;
    if (r != known) {
      const int k = find_lattice(prefix, run.nlat, r);
      if (k != l) {
        __syncwarp();
        for (uint32_t c = lane; c < sizeof(BatchLat) / 4; c += 32)
          reinterpret_cast<uint32_t*>(&B)[c] = reinterpret_cast<const uint32_t*>(&run.lats[k])[c];
        __syncwarp();
        l = k;
      }
      local = r - prefix[l];
      known = r;
    }
    if (B.nlev != 0 && level >= B.nlev) continue;
    if (level > 0 && !warp_wait(&run.done[l], level * B.ntiles, run.status)) break;
    fails += hb_item<S, NR>(run, B, level, local);
    warp_release(&run.done[l]);
  }
  if (fails) atomicAdd(&run.status[0], fails);
}

// An item costs about 3 us besides its links (the counter's round trips), so a warp should have few
// items a level; but its links run one after another, so the level ends with the warp that has
// most.  FP64 (a link takes three times as long): 32 links, always (32^4 12.2 ms against 13.2 with
// 256).  FP32: a lattice that is most of the batch runs its levels one by one, and the length that
// gives the fewest links in a row, the longest of those, wins (24^4: 96 links 1.29 ms, 32: 1.70, 256: 2.34;
// 32^4: 224 links 3.91 ms, 32: 4.21, 192: 5.65); lattices that overlap fill each other's gaps, and
// every warp takes one item a level, of 160 links at most (54 lattices of 8^4 to 16^4: 32 links
// 10.4 ms, 128: 8.55, 160: 8.44, 256: 8.67; 32 of 8^4 to 12^4: 64 links 1.25 ms, 32: 1.63, 96: 1.47).
uint32_t batch_tile(uint32_t most, uint64_t groups, uint64_t largest, int prec) {
  if (prec == QCB_PREC_FP64) return 32;
  const uint64_t warps = 148u * QCB_BATCH_MINB32 * 4u, cap = most / 32;
  uint64_t best = 1;
  if (2 * largest > groups) {
    uint64_t cost = ~0ull;
    for (uint64_t u = 1; u <= cap && u <= 1 + groups / warps; ++u) {
      const uint64_t c = u * ((groups + u * warps - 1) / (u * warps));
      if (c <= cost) cost = c, best = u;
    }
  } else {
    best = (groups + warps / 2) / warps;
    if (best > 5) best = 5;
    if (best > cap) best = cap;
    if (best < 1) best = 1;
  }
  return 32 * (uint32_t)best;
}

// ---- launch -------------------------------------------------------------------------------
template <typename S, int NR>
static cudaError_t batch_launch_impl(const BatchRun& run, int block, int max_blocks, cudaStream_t s) {
  void* fn = (void*)k_batch<S, NR>;
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, 0);
  if (e != cudaSuccess) return e;
  e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const uint64_t total = (uint64_t)run.nlevels * run.per_level;
  uint64_t grid = (uint64_t)per_sm * (uint64_t)sms;
  if (max_blocks > 0 && (uint64_t)max_blocks < grid) grid = (uint64_t)max_blocks;
  if (grid > total) grid = total;
  if (grid > run.per_level) grid = run.per_level;
  if (grid == 0) return cudaSuccess;
  BatchRun r = run;
  void* args[] = {&r};
  return cudaLaunchCooperativeKernel(fn, dim3((unsigned)grid), dim3(block), args, 0, s);
}

cudaError_t launch_batch(const BatchRun& run, int prec, int nr, int block, int max_blocks, cudaStream_t s) {
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  if (block <= 0) block = 128;
  if (block > 128 || (block & 31)) return cudaErrorInvalidValue;
  QCB_DISPATCH_STORE(probe, batch_launch_impl, run, block, max_blocks, s);
}

// ---- wait self-test -------------------------------------------------------------------------
// Block 0 waits for flag[0] >= 1, which nothing sets, until its limit; it then counts a
// timeout and raises the abort flag.  The other blocks wait for the same flag with a longer
// limit and return when they see the abort flag.  Exercises the bounded wait and abort path
// of the persistent kernels without a fault.
__global__ void k_wait_probe(const uint32_t* flag, uint32_t* status, uint64_t limit_ns) {
  const uint64_t lim = blockIdx.x == 0 ? limit_ns : 4 * limit_ns;
  if (!warp_wait(flag, 1u, status, lim)) return;
  if (threadIdx.x == 0) atomicAdd(&status[3], 1u);  // a wait that succeeded (not expected)
}

cudaError_t launch_wait_probe(const uint32_t* flag, uint32_t* status, uint64_t limit_ns, int blocks,
                              cudaStream_t s) {
  void* args[] = {(void*)&flag, (void*)&status, (void*)&limit_ns};
  return cudaLaunchCooperativeKernel((void*)k_wait_probe, dim3(blocks), dim3(32), args, 0, s);
}

// ---- batched observables --------------------------------------------------------------------
// Plaquette: one reduction item per (lattice, tile of RED_SITES sites, half of each parity), partial
// sums parts[item].  Plaquette and clover partials are then added by one block per lattice in a fixed
// order with Neumaier compensation.
constexpr int RED_SITES = 128;
int batch_red_sites() { return RED_SITES; }

template <typename S, int NR>
__global__ void __launch_bounds__(RED_SITES, sizeof(S) == 4 ? 5 : 3) k_batch_plaquette(const BatchLat* __restrict__ lats,
                                                         const uint32_t* __restrict__ rprefix, int nlat,
                                                         double* __restrict__ parts) {
  __shared__ double sh[RED_SITES / 32];
  const uint32_t item = blockIdx.x;
  const int l = find_lattice(rprefix, nlat, item);
  const BatchLat& B = lats[l];
  const uint32_t i = block_site(item - rprefix[l]);
  const int par = block_parity();
  Links<S, NR> f;
  f.p = reinterpret_cast<typename Links<S, NR>::V*>(B.links);
  f.stride = B.g.stride;
  double v = 0.0;
  if (i < B.g.Vh) {
    const Coord x = cb_coord(B.g, par, i);
    v = site_plaquettes<Links<S, NR>, arith_t<S>>(B.g, f, x, par, i, 0, 1, 6) * (1.0 / 3.0);
  }
  const double b = block_sum<RED_SITES>(v, sh);
  if (threadIdx.x == 0) parts[item] = b;
}

// One block per lattice: thread j sums items j, j+128, ... of the lattice; thread 0 adds the 128
// sums in order.  (One warp a lattice took 40 us for the 8192 partials of 32^4.)  WHAT 0:
// out[l] = sum / (6 V); WHAT 1: out[2l] = Q, out[2l+1] = E.
template <int WHAT>
__global__ void __launch_bounds__(128) k_batch_red_finalize(const BatchLat* __restrict__ lats,
                                                            const uint32_t* __restrict__ rprefix, uint32_t nitems,
                                                            const double* __restrict__ parts, double* __restrict__ out) {
  __shared__ double sh[2][128];
  const int l = blockIdx.x;
  const uint32_t a = rprefix[l], b = rprefix[l + 1];
  const double V = (double)lats[l].g.V;
  for (int q = 0; q < (WHAT == 0 ? 1 : 2); ++q) {
    double s = 0.0, c = 0.0;
    for (uint32_t k = a + threadIdx.x; k < b; k += 128) neumaier_add(s, c, parts[(size_t)q * nitems + k]);
    __syncthreads();
    sh[0][threadIdx.x] = s;
    sh[1][threadIdx.x] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
      const int n = b - a < 128 ? (int)(b - a) : 128;
      double S = 0.0, Cc = 0.0;
      for (int j = 0; j < n; ++j) {
        neumaier_add(S, Cc, sh[0][j]);
        Cc += sh[1][j];
      }
      const double tot = S + Cc;
      if (WHAT == 0)
        out[l] = tot / (6.0 * V);
      else if (q == 0)
        out[2 * l] = tot * (1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846));
      else
        out[2 * l + 1] = 0.5 * tot / V;
    }
  }
}

template <typename S, int NR>
static cudaError_t batch_plaq_impl(const BatchLat* lats, const uint32_t* rprefix, int nlat, uint32_t nitems,
                                   double* scratch, double* out, cudaStream_t s) {
  if (nitems == 0) return cudaSuccess;
  k_batch_plaquette<S, NR><<<nitems, RED_SITES, 0, s>>>(lats, rprefix, nlat, scratch);
  k_batch_red_finalize<0><<<nlat, 128, 0, s>>>(lats, rprefix, nitems, scratch, out);
  return cudaGetLastError();
}

cudaError_t launch_batch_plaquette(const BatchLat* lats, const uint32_t* rprefix, int nlat, uint32_t nitems,
                                   int prec, int nr, double* scratch, double* out, cudaStream_t s) {
  LatDev probe;
  probe.prec = prec;
  probe.nr = nr;
  QCB_DISPATCH_STORE(probe, batch_plaq_impl, lats, rprefix, nlat, nitems, scratch, out, s);
}
cudaError_t launch_batch_qe(const BatchLat* lats, const uint32_t* rprefix, int nlat, uint32_t nitems,
                            const double* parts, double* out2, cudaStream_t s) {
  if (nitems == 0) return cudaSuccess;
  k_batch_red_finalize<1><<<nlat, 128, 0, s>>>(lats, rprefix, nitems, parts, out2);
  return cudaGetLastError();
}

}  // namespace qcb
