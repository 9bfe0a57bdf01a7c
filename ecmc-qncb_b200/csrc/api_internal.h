// api_internal.h — the C ABI's opaque objects and shared host helpers (library-internal).
#pragma once
#include <mutex>
#include <string>

#include "../../include/qcb.h"
#include "flow.h"
#include "kernels.h"

struct qcb_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int block = 0;
  uint32_t* d_status = nullptr;  // [0] KP cap hits
  uint32_t* h_status = nullptr;  // pinned mirror
  // Partial sums of the reductions.  It grows with the largest lattice (ensure_scratch, at its creation),
  // so the first measurement of a lattice does not allocate.
  double* d_scratch = nullptr;
  size_t scratch_n = 0;
  double* d_out = nullptr;       // small results
  double* h_out = nullptr;       // pinned mirror
  double* d_stage[2] = {nullptr, nullptr};
  size_t stage_bytes = 0;
  double* h_stage = nullptr;  // pinned, for file I/O
  // Plaquette loops of the flow and the clover, shared by the context's lattices and batches (its calls
  // run in stream order); allocated on first use, at most LOOPS_MAX_BYTES or two time slices.
  qcb::LoopBuf loops;
  uint64_t launches = 0;
  std::mutex mu;
  // Objects created on this context (lattices, batches, servers).  qcb_ctx_destroy with
  // live objects only marks the context; the last object's destroy frees it, so no child
  // ever uses a freed context.
  int refs = 0;
  bool doomed = false;
};

struct qcb_lattice {
  qcb_ctx* ctx = nullptr;
  qcb::LatDev dev;
  size_t bytes = 0;
  // Wilson-flow work space, allocated on first use: two link buffers + accumulator.
  void* fw[2] = {nullptr, nullptr};
  void* fz = nullptr;
  // Slab of a larger lattice (qcb_lattice_create_slab): global extents and the global time
  // of local time 1; slab_tl == 0 for a whole lattice.
  int gdims[4] = {0, 0, 0, 0};
  int slab_t0 = 0, slab_tl = 0;
};

namespace qcb {
// Reference counting of a context's child objects (see qcb_ctx::refs).
void ctx_ref(qcb_ctx* c);
void ctx_unref(qcb_ctx* c);
// Allocates a lattice's Wilson-flow work space (two link buffers + accumulator) once.
int ensure_flow_space(qcb_lattice* L);
// Makes the context's loop buffer answer a request as far as the memory goes (loops_reserve).
void reserve_loops(qcb_ctx* c, size_t want, size_t least);
// Reads and clears the context's device status words (after synchronising its stream).
int check_status(qcb_ctx* c);
int wait_status(qcb_ctx* c);
}  // namespace qcb
