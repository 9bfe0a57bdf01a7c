// counter.h — comparison of the progress counters of the persistent kernels.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define QCB_HD __host__ __device__ __forceinline__
#else
#define QCB_HD inline
#endif

namespace qcb {

// Whether a 32-bit counter that only grows has come to `target`; both are taken mod 2^32, so a counter
// may go round.  A lattice's counter of finished tiles does: 64^4 in tiles of 32 links counts 2^32
// within 2048 sweeps of one launch.  The two are never 2^31 apart (a waiting tile is one level, at most 2^24
// tiles, behind).
QCB_HD bool counter_reached(uint32_t have, uint32_t target) { return (int32_t)(have - target) >= 0; }

}  // namespace qcb
