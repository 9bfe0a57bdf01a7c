// batch.h — device descriptors and launchers of the persistent multi-lattice kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"

namespace qcb {

// One lattice of a batched launch (device array).
struct BatchLat {
  Geom g;
  void* links;
  double beta;      // coupling
  uint32_t k0, k1;  // Philox key (seed)
  uint32_t sweep0;  // sweep counter of the launch's first sweep
  uint32_t tile;    // sites per work item (a multiple of 32)
  uint32_t ntiles;  // work items of this lattice per level (0: none)
  uint32_t nlev;    // levels this lattice takes part in (0 = all levels of the launch)
  int n_hits;       // hits (0 = the launch's value)
};

// One persistent heatbath launch: nlevels levels of per_level items each.
struct BatchRun {
  const BatchLat* lats;    // nlat descriptors
  const uint32_t* prefix;  // nlat+1 prefix sums of ntiles; prefix[nlat] = per_level
  int nlat;
  uint32_t nlevels;
  uint32_t per_level;
  uint32_t* done;    // nlat finished-tile counters, zero at launch
  uint32_t* status;  // [0] KP cap hits, [1] wait timeouts, [2] abort flag
  int n_hits;
};

// Sites per work item of a launch whose lattices hold `groups` groups of 32 links a pass, the
// largest of them `largest`: at most `most`.
uint32_t batch_tile(uint32_t most, uint64_t groups, uint64_t largest, int prec);

// Cooperative persistent launch: the grid is the co-resident maximum (capped by max_blocks
// when > 0) for the given block size.
cudaError_t launch_batch(const BatchRun& run, int prec, int nr, int block, int max_blocks, cudaStream_t s);

// Bounded-wait self-test: `blocks` co-resident blocks wait on flag[0] (never set); block 0
// gives up after limit_ns.  status[1] = timeouts, status[2] = abort flag, status[3] = waits
// that succeeded.
cudaError_t launch_wait_probe(const uint32_t* flag, uint32_t* status, uint64_t limit_ns, int blocks,
                              cudaStream_t s);

// Batched plaquette: one item per (lattice, tile of batch_red_sites() sites), item r of lattice
// l in [rprefix[l], rprefix[l+1]); out[l] = mean plaquette.  scratch holds rprefix[nlat] doubles.
int batch_red_sites();
cudaError_t launch_batch_plaquette(const BatchLat* lats, const uint32_t* rprefix, int nlat, uint32_t nitems,
                                   int prec, int nr, double* scratch, double* out, cudaStream_t s);
// out2[2l], out2[2l+1] = (Q, E) from the clover partials of run_qe_plan: lattice l's are
// parts[rprefix[l] .. rprefix[l+1]) (q) and the same places after nitems (e).
cudaError_t launch_batch_qe(const BatchLat* lats, const uint32_t* rprefix, int nlat, uint32_t nitems,
                            const double* parts, double* out2, cudaStream_t s);

}  // namespace qcb
