// flow.h — device descriptors and launchers of the Wilson flow and the clover observables.
//
// Both are built from one field of plaquette loops (loops.cuh): K_{mu nu}(x) = P_TA(U_mu(x)
// U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag), mu < nu, eight reals for each plane, and for the
// clover the traces that P_TA takes out.  A flow stage computes the loops of its source links
// (launch_loops) and then updates every link from them (launch_flow_update); Q and E sum the
// transported loops of each site (launch_loops_qe).
//
// The loops live in a buffer of a bounded number of time slices (LoopBuf).  A lattice whose
// loops do not fit is worked through in rounds of consecutive slices; the buffer then is a
// ring in which the slice before a round's first stays from the round before.  Where not even two
// slices fit (device memory is full, or the user's limit is smaller), the round has no loops
// (k.p == nullptr): staples and leaves are multiplied out link by link (launch_flow_links,
// launch_clover), which takes no work space.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "kernels.h"
#include "loop_buf.h"

namespace qcb {

// The loop buffer as the kernels see it: slices time slices of 6 planes x 2 parities, chunk
// arrays of `stride` elements (the algebra layout of AlgField), then the traces, then (18-real
// links) a byte for each of the 4 x 2 links of a checkerboard index that is set where the link is not
// unitary.
struct LoopDev {
  void* p;
  void* tr;
  uint8_t* off;
  uint32_t stride;
  int slices;
};

// One round of one lattice.
struct FlowLat {
  Geom g;
  void* a;    // links of even steps (stage 1 reads a, writes b; stage 2 back; stage 3 a -> b)
  void* b;    // links of odd steps
  void* acc;  // force accumulator
  LoopDev k;
  double eps;
  int t0, t1;     // time slices the round updates or measures
  int kt0, kn;    // time slices whose loops it computes first: kn from kt0 (-1: the last slice)
  uint32_t tile;  // sites of one parity per block of the update (the other kernels: at least 128)
  int nsteps;     // RK3 steps the lattice takes part in
};

// Bytes of the loops of `slices` time slices.
size_t loops_bytes(const Geom& g, int prec, int slices);
// Slices of g that fit into `bytes` (at most L_t; 0 if fewer than the two a round needs).
int loops_slices(const Geom& g, int prec, size_t bytes);
// Grows buf on the device (loops_grow); cudaErrorMemoryAllocation when it holds less than least.
// The caller has no work in flight that uses the buffer it replaces, or lets cudaFree wait for it.
cudaError_t loops_reserve(LoopBuf* buf, size_t want, size_t least);
// The buffer from offset `off` as lattice g's loops (slices as loops_slices gives them).
LoopDev loops_view(const LoopBuf& buf, size_t off, const Geom& g, int prec, int slices);

// The rounds of lattice L with loops k, or one without loops (a, b, acc, eps, tile and nsteps are the caller's).
std::vector<FlowLat> flow_rounds(const LatDev& L, const LoopDev& k);

// Blocks of a round's three kernels.
uint32_t loops_blocks(const FlowLat& r);
uint32_t update_blocks(const FlowLat& r);
uint32_t qe_blocks(const FlowLat& r);

// The lattices of one launch: one round by value (lats == nullptr), or nlat descriptors on the
// device with the prefix sums of their block counts.
struct FlowSet {
  FlowLat one;
  const FlowLat* lats = nullptr;
  const uint32_t* prefix = nullptr;  // nlat + 1
  int nlat = 1;
  uint32_t blocks = 0;  // prefix[nlat]
};

// swap = 0: the loops of a, 1: of b.  Lattices with nsteps <= step are passed over.
cudaError_t launch_loops(const FlowSet& s, int prec, int nr, bool trace, int swap, int step, cudaStream_t st);
// RK3 stage (1, 2, 3) from the loops of the source: a -> b (swap = 0) or b -> a (swap = 1).
cudaError_t launch_flow_update(const FlowSet& s, int prec, int nr, int stage, int swap, int step, cudaStream_t st);
// Unscaled clover sums of each block, parts[first + block] (q) and parts[n + first + block] (e),
// from loops computed with trace = true.
cudaError_t launch_loops_qe(const FlowSet& s, int prec, int nr, int swap, double* parts, uint32_t first, uint32_t n,
                            cudaStream_t st);
// The same for a round without loops, from the links alone.
cudaError_t launch_flow_links(const FlowLat& r, int prec, int nr, int stage, int swap, cudaStream_t st);
cudaError_t launch_clover(const FlowLat& r, int prec, int nr, int swap, double* parts, uint32_t first, uint32_t n,
                          cudaStream_t st);

// ---- many lattices ------------------------------------------------------------------------
// One lattice of a plan: links (L.links = a), the other buffer b and the accumulator (flow
// only), the step size, sites of one parity per block, RK3 steps it takes part in.
struct FlowItem {
  LatDev L;
  void* b;
  void* acc;
  double eps;
  uint32_t tile;
  int nsteps;
};

// Lattices worked through together: groups whose loops fit into the buffer at once, one after
// another, each group's kernels covering all its lattices; a lattice whose loops do not fit is
// a group of its own with several rounds, or one without loops.
struct FlowPlan {
  struct Round {
    int first, n;            // lats[first .. first + n)
    uint32_t at;             // prefix + at: loops, update and qe prefix sums, n + 1 each
    uint32_t loops, update, qe;  // their totals
    uint32_t qe_first;       // place of the round's first clover partial
  };
  std::vector<FlowLat> lats;
  std::vector<uint32_t> prefix;
  std::vector<std::vector<Round>> groups;
  std::vector<uint32_t> qe_prefix;  // clover partials of item l: [qe_prefix[l], qe_prefix[l + 1])
};
// Buffer sizes for these lattices: all loops at once, and the least one round of each needs.
void flow_plan_bytes(const std::vector<FlowItem>& items, size_t* want, size_t* least);
// Most sites per work item of a plan; an item's own tile only makes it smaller.
uint32_t flow_tile_most(const std::vector<FlowItem>& items);
FlowPlan flow_plan(const std::vector<FlowItem>& items, const LoopBuf& buf);
// n RK3 steps of every lattice from its links a (odd = 0) or b (odd = 1), and the clover sums
// of the links; d_lats and d_prefix are the plan's arrays on the device.  *launches counts.
cudaError_t run_flow_plan(const FlowPlan& p, const FlowLat* d_lats, const uint32_t* d_prefix, int prec, int nr, int odd,
                          int n, cudaStream_t st, uint64_t* launches);
cudaError_t run_qe_plan(const FlowPlan& p, const FlowLat* d_lats, const uint32_t* d_prefix, int prec, int nr, int odd,
                        double* parts, cudaStream_t st, uint64_t* launches);

}  // namespace qcb
