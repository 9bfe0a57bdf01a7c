// loop_buf.h — the size of a plaquette-loop buffer and how it grows (no CUDA: the caller allocates).
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace qcb {

// Largest loop buffer unless two time slices of a lattice need more, or the user set a limit.  1 GiB
// holds a whole 32^4 (FP64 461 MB); 64^4 runs in rounds of 17 slices in FP32 and 8 in FP64 (one slice
// of the buffer stays from the round before), each of over two million sites, so that a round's
// launches fill the device.
constexpr size_t LOOPS_MAX_BYTES = 1ull << 30;
constexpr size_t LOOPS_NO_LIMIT = ~(size_t)0;

// A loop buffer (of a context, used by its lattices and batches, or of a server).
struct LoopBuf {
  void* p = nullptr;
  size_t bytes = 0;
  size_t wanted = 0;  // the largest size asked for (not tried again once it did not fit)
  uint64_t gen = 0;   // goes up when p is replaced: plans made on the old one are then remade
  size_t limit = LOOPS_NO_LIMIT;  // set by the user
};

// The size that a request for `want` bytes, of which `least` are needed at once, aims at.
inline size_t loops_target(const LoopBuf& b, size_t want, size_t least) {
  if (b.limit != LOOPS_NO_LIMIT) return want < b.limit ? want : b.limit;
  if (want > LOOPS_MAX_BYTES) want = LOOPS_MAX_BYTES;
  return want < least ? least : want;
}
// Whether b answers the request as it is.
inline bool loops_covered(const LoopBuf& b, size_t want, size_t least) {
  const size_t t = loops_target(b, want, least);
  return b.bytes >= least && (b.bytes >= t || b.wanted >= t);
}
template <typename Free>
void loops_drop(LoopBuf* b, const Free& free) {
  if (!b->p) return;
  free(b->p);
  b->p = nullptr;
  b->bytes = b->wanted = 0;
  b->gen++;
}
// Replaces b's memory by the target size, or by the most that alloc (null: failed) gives of its
// halves, but no less than least.  False when that fails too (b is empty then), or when the user's limit
// is below least (b is left as it is).
template <typename Alloc, typename Free>
bool loops_grow(LoopBuf* b, size_t want, size_t least, const Alloc& alloc, const Free& free) {
  if (loops_covered(*b, want, least)) return true;
  const size_t target = loops_target(*b, want, least);
  if (target < least) return false;
  loops_drop(b, free);
  b->wanted = target;
  for (size_t n = target;; n = n / 2 > least ? n / 2 : least) {
    if ((b->p = alloc(n)) != nullptr) {
      b->bytes = n;
      b->gen++;
      return true;
    }
    if (n <= least) return false;
  }
}

}  // namespace qcb
