// flow_launch.cuh — what the kernels of the loops, the flow update and the clover share: which
// lattice a block works on, and their launch.
#pragma once
#include "dispatch.cuh"
#include "flow.h"
#include "loops.cuh"
#include "sync.cuh"

namespace qcb {

constexpr int FLOW_THREADS = 128;  // and sites of one parity per block where a thread has a site

// The lattice l with prefix[l] <= b < prefix[l + 1], found by a whole warp: one load and one
// ballot for each 32 lattices.
__device__ __forceinline__ int lattice_of(const uint32_t* __restrict__ prefix, int nlat, uint32_t b) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < nlat; base += 32) {
    const uint32_t end = base + lane < nlat ? __ldg(&prefix[base + lane + 1]) : 0xFFFFFFFFu;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, end <= b);
    if (m != 0xFFFFFFFFu) return base + __popc(m);
  }
  return nlat - 1;
}

template <typename S, int NR>
__device__ __forceinline__ Links<S, NR> flow_links(const FlowLat& L, int swap) {
  Links<S, NR> f;
  f.p = reinterpret_cast<typename Links<S, NR>::V*>(swap ? L.b : L.a);
  f.stride = L.g.stride;
  return f;
}

}  // namespace qcb
