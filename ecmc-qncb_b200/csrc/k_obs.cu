// k_obs.cu — mean plaquette reduction, and the sums of per-block partials.
//
// Reference: mean_plaquette_local / _global (src/observables/observables_mpi.cpp:8-43): serial
// sum of Re tr(U_mu(x) U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag)/3 over x and mu < nu, / (6V).
// Here: one thread per site (a slab skips its halo slices), the site's value in the lattice's
// arithmetic type, converted to FP64, and an FP64 tree in each block; k_total adds the block sums in a fixed
// order with Neumaier compensation.  The grid has a block for 64 checkerboard indices up to a bound
// (the library's RED_BLOCKS, or the caller's scratch), beyond which blocks stride.
#include <algorithm>

#include "dispatch.cuh"
#include "obs_site.cuh"
#include "reduce.cuh"
#include "sync.cuh"

namespace qcb {

constexpr int RED_THREADS = 128;
// One block per 64 checkerboard indices up to 60 per SM (32^4: 8192), from there a grid-stride loop.
constexpr int RED_BLOCKS = 148 * 60;

// Minimum resident blocks per SM of the reduction (32^4, 18-real: FP64 3 224 us, 2 267, 4 235; FP32
// 12-real with the third rows of products rebuilt: 5 114 us, 4 121).
template <typename S>
struct RedMinBlocks {
  static constexpr int value = sizeof(S) == 4 ? 5 : 3;
};

int reduce_blocks() { return RED_BLOCKS; }

// Totals of quantities of n partials each (block q: parts[q n .. q n + n)), Neumaier-compensated and
// in a fixed order: thread j sums k = j, j + 1024, ..., then a tree of the compensated sums.  out[q] =
// total * (q ? scale1 : scale0).  With host_status, block 0 also copies the four status words
// there; out and host_status may be pinned host memory, and the caller then needs no copy and no
// other launch before it synchronises.  One warp on 1184 partials, a scaling kernel and two
// copies took 13 us behind a plaquette of 8^4 (this: 4), 16 behind a sweep.
constexpr int TOTAL_THREADS = 1024;
__global__ void __launch_bounds__(TOTAL_THREADS) k_total(const double* __restrict__ parts, int n, double scale0,
                                                         double scale1, double* __restrict__ out,
                                                         const uint32_t* __restrict__ status,
                                                         uint32_t* __restrict__ host_status) {
  __shared__ double ls[TOTAL_THREADS / 32], lc[TOTAL_THREADS / 32];
  pdl_wait();
  const double* p = parts + (size_t)blockIdx.x * n;
  double s = 0.0, c = 0.0;
  for (int k = threadIdx.x; k < n; k += TOTAL_THREADS) neumaier_add(s, c, p[k]);
  auto tree = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, c, o);
      neumaier_add(s, c, s2);
      c += c2;
    }
  };
  tree();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) ls[w] = s, lc[w] = c;
  __syncthreads();
  if (w == 0) {
    s = ls[lane], c = lc[lane];
    tree();
    if (lane == 0) out[blockIdx.x] = (s + c) * (blockIdx.x ? scale1 : scale0);
    if (host_status && blockIdx.x == 0 && lane < 4) host_status[lane] = status[lane];
  }
}

static cudaError_t total(const double* parts, int n, int nq, double scale0, double scale1, double* out,
                         const StatusCopy& st, cudaStream_t s) {
  return pdl_launch(k_total, dim3(nq), TOTAL_THREADS, s, parts, n, scale0, scale1, out, st.device, st.host);
}

// Per block, the sum of Re tr P / 3 over planes blockIdx.y, blockIdx.y + gridDim.y, ... of its sites.
template <typename S, int NR>
__global__ void __launch_bounds__(RED_THREADS, RedMinBlocks<S>::value) k_plaquette(Geom g, Links<S, NR> f,
                                                                                   double* __restrict__ parts) {
  __shared__ double sh[RED_THREADS / 32];
  pdl_wait();
  double acc = 0.0;
  const int par = block_parity();
  for (uint32_t b = blockIdx.x; b * 64 < g.Vh; b += gridDim.x) {
    const uint32_t i = block_site(b);
    if (i >= g.Vh) continue;
    const Coord x = cb_coord(g, par, i);
    if (own_site(g, x.c[3]))
      acc += site_plaquettes<Links<S, NR>, arith_t<S>>(g, f, x, par, i, blockIdx.y, gridDim.y, 6);
  }
  const double b = block_sum<RED_THREADS>(acc * (1.0 / 3.0), sh);
  if (threadIdx.x == 0) parts[blockIdx.y * gridDim.x + blockIdx.x] = b;
}

// Planes side by side while the sites' blocks are fewer than fill the chip.
static dim3 plaquette_grid(const Geom& g, int most) {
  const int nb = (int)std::min<uint64_t>(((uint64_t)g.Vh + 63) / 64, (uint64_t)most);
  return dim3(nb, nb * 6 <= std::min(most, 148 * 8) ? 6 : 1);
}

template <typename S, int NR>
static cudaError_t plaquette_impl(const LatDev& L, int most, double* scratch, double* out, const StatusCopy& st,
                                  cudaStream_t s) {
  Links<S, NR> f;
  f.p = reinterpret_cast<typename Links<S, NR>::V*>(L.links);
  f.stride = L.g.stride;
  const dim3 grid = plaquette_grid(L.g, most);
  const cudaError_t e = pdl_launch(k_plaquette<S, NR>, grid, RED_THREADS, s, L.g, f, scratch);
  return e != cudaSuccess ? e : total(scratch, (int)(grid.x * grid.y), 1, 1.0, 1.0, out, st, s);
}

cudaError_t launch_plaquette(const LatDev& L, double* scratch, double* out, const StatusCopy& st, cudaStream_t s) {
  QCB_DISPATCH_STORE(L, plaquette_impl, L, RED_BLOCKS, scratch, out, st, s);
}

cudaError_t launch_plaquette_partials(const LatDev& L, int nblocks, double* scratch, double* out, cudaStream_t s) {
  if (nblocks < 1) return cudaErrorInvalidValue;
  QCB_DISPATCH_STORE(L, plaquette_impl, L, nblocks, scratch, out, StatusCopy(), s);
}

int reduce_threads() { return RED_THREADS; }

// First level of a deterministic sum of nq quantities of n partials each (quantity q at
// parts[q * n ..]): block (b, q) sums the chunk [b * chunk, min((b + 1) * chunk, n)) of quantity
// q (thread-strided in index order, then the block tree) into out[q * gridDim.x + b].
__global__ void __launch_bounds__(RED_THREADS) k_sum_chunks(const double* __restrict__ parts, int n, int chunk,
                                                           double* __restrict__ out) {
  __shared__ double sh[RED_THREADS / 32];
  const double* p = parts + (size_t)blockIdx.y * n;
  const int lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  double s = 0.0, c = 0.0;
  for (int k = lo + threadIdx.x; k < hi; k += RED_THREADS) neumaier_add(s, c, p[k]);
  const double b = block_sum<RED_THREADS>(s + c, sh);
  if (threadIdx.x == 0) out[blockIdx.y * gridDim.x + blockIdx.x] = b;
}

// The totals of nq <= 2 quantities, in a fixed order whatever the device: at most SUM_ONE partials by
// k_total alone, more in chunks first (64^4's 131072: 60 us in one block, 6 in two launches).
constexpr int SUM_ONE = 16384;
static cudaError_t sum_parts(const double* parts, int n, int nq, double scale0, double scale1, double* tmp, double* out,
                             const StatusCopy& st, cudaStream_t s, uint64_t* launches) {
  if (n < 1 || nq < 1 || nq > 2) return cudaErrorInvalidValue;
  ++*launches;
  if (n <= SUM_ONE) return total(parts, n, nq, scale0, scale1, out, st, s);
  ++*launches;
  const int nb = 256, chunk = (n + nb - 1) / nb;
  k_sum_chunks<<<dim3(nb, nq), RED_THREADS, 0, s>>>(parts, n, chunk, tmp);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? e : total(tmp, nb, nq, scale0, scale1, out, st, s);
}

cudaError_t launch_sum_parts(const double* parts, int n, double* tmp, double* out, const StatusCopy& st, cudaStream_t s,
                             uint64_t* launches) {
  return sum_parts(parts, n, 1, 1.0, 1.0, tmp, out, st, s, launches);
}

cudaError_t launch_qe_from_parts(const double* parts, int n, double* tmp, double* out2, double inv_vol,
                                 const StatusCopy& st, cudaStream_t s, uint64_t* launches) {
  const double q = 1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846);
  return sum_parts(parts, n, 2, q, 0.5 * inv_vol, tmp, out2, st, s, launches);
}

}  // namespace qcb
