// flow_plan.cu — which lattices share a launch of the flow and the clover, and the launches.
#include "flow.h"

namespace qcb {

static size_t aligned(size_t n) { return (n + 255) & ~(size_t)255; }

void flow_plan_bytes(const std::vector<FlowItem>& items, size_t* want, size_t* least) {
  *want = *least = 0;
  for (const FlowItem& it : items) {
    *want += aligned(loops_bytes(it.L.g, it.L.prec, it.L.g.L[3]));
    const size_t two = aligned(loops_bytes(it.L.g, it.L.prec, 2));
    if (two > *least) *least = two;
  }
}

// At most 128 (a block's threads), and 32 while the whole plan then has fewer than 4096 update blocks.
// Four RK3 steps, FP32 12-real: 4^4 with 6^4 89 us with 32, 159 with 128, 258 with 256; eight of 8^4 207,
// 315, 474; four of 12^4 380, 396, 614; 54 of 8^4 to 16^4 9.14 ms, 8.93, 9.03.
uint32_t flow_tile_most(const std::vector<FlowItem>& items) {
  uint64_t blocks = 0;
  for (const FlowItem& it : items) blocks += 2 * ((uint64_t)(it.L.g.Vh + 31) / 32);
  return blocks < 4096 ? 32u : 128u;
}

FlowPlan flow_plan(const std::vector<FlowItem>& items, const LoopBuf& buf) {
  const uint32_t most = flow_tile_most(items);
  FlowPlan p;
  p.qe_prefix.push_back(0);
  auto add = [&](const FlowItem& it, FlowLat r) {
    r.b = it.b;
    r.acc = it.acc;
    r.eps = it.eps;
    r.tile = it.tile < most ? it.tile : most;
    r.nsteps = it.nsteps;
    p.lats.push_back(r);
  };
  auto close_round = [&](int first) {
    FlowPlan::Round rd;
    rd.first = first;
    rd.n = (int)p.lats.size() - first;
    rd.at = (uint32_t)p.prefix.size();
    uint32_t* total[3] = {&rd.loops, &rd.update, &rd.qe};
    uint32_t (*blocks[3])(const FlowLat&) = {loops_blocks, update_blocks, qe_blocks};
    for (int k = 0; k < 3; ++k) {
      uint32_t sum = 0;
      p.prefix.push_back(0);
      for (int l = first; l < first + rd.n; ++l) p.prefix.push_back(sum += blocks[k](p.lats[l]));
      *total[k] = sum;
    }
    rd.qe_first = 0;
    p.groups.back().push_back(rd);
  };
  size_t used = 0;
  int first = 0;
  bool open = false;
  for (const FlowItem& it : items) {
    const size_t all = aligned(loops_bytes(it.L.g, it.L.prec, it.L.g.L[3]));
    if (open && used + all > buf.bytes) {
      close_round(first);
      open = false;
    }
    if (!open) {
      p.groups.emplace_back();
      used = 0;
      first = (int)p.lats.size();
    }
    const int slices = loops_slices(it.L.g, it.L.prec, buf.bytes - used);
    const std::vector<FlowLat> rounds = flow_rounds(it.L, loops_view(buf, used, it.L.g, it.L.prec, slices));
    if (rounds.size() == 1 && rounds[0].k.p) {
      add(it, rounds[0]);
      used += all;
      open = true;
    } else {
      for (const FlowLat& r : rounds) {
        add(it, r);
        close_round((int)p.lats.size() - 1);
      }
    }
    uint32_t n = 0;
    for (size_t k = 0; k < rounds.size(); ++k) n += qe_blocks(p.lats[p.lats.size() - 1 - k]);
    p.qe_prefix.push_back(p.qe_prefix.back() + n);
  }
  if (open) close_round(first);
  uint32_t at = 0;
  for (auto& g : p.groups)
    for (FlowPlan::Round& rd : g) {
      rd.qe_first = at;
      at += rd.qe;
    }
  return p;
}

static FlowSet set_of(const FlowPlan::Round& rd, const FlowLat* d_lats, const uint32_t* d_prefix, int which,
                      uint32_t blocks) {
  FlowSet s;
  s.one = FlowLat();
  s.lats = d_lats + rd.first;
  s.prefix = d_prefix + rd.at + (size_t)which * (rd.n + 1);
  s.nlat = rd.n;
  s.blocks = blocks;
  return s;
}

cudaError_t run_flow_plan(const FlowPlan& p, const FlowLat* d_lats, const uint32_t* d_prefix, int prec, int nr, int odd,
                          int n, cudaStream_t st, uint64_t* launches) {
  for (const auto& g : p.groups)
    for (int step = 0; step < n; ++step)
      for (int stage = 1; stage <= 3; ++stage) {
        const int swap = (odd ^ (step & 1)) ^ (stage == 2 ? 1 : 0);
        for (const FlowPlan::Round& rd : g) {
          const FlowLat& only = p.lats[rd.first];
          if (!only.k.p) {
            if (step >= only.nsteps) continue;
            const cudaError_t e = launch_flow_links(only, prec, nr, stage, swap, st);
            if (e != cudaSuccess) return e;
            ++*launches;
            continue;
          }
          cudaError_t e = launch_loops(set_of(rd, d_lats, d_prefix, 0, rd.loops), prec, nr, false, swap, step, st);
          if (e == cudaSuccess)
            e = launch_flow_update(set_of(rd, d_lats, d_prefix, 1, rd.update), prec, nr, stage, swap, step, st);
          if (e != cudaSuccess) return e;
          *launches += 2;
        }
      }
  return cudaSuccess;
}

cudaError_t run_qe_plan(const FlowPlan& p, const FlowLat* d_lats, const uint32_t* d_prefix, int prec, int nr, int odd,
                        double* parts, cudaStream_t st, uint64_t* launches) {
  const uint32_t n = p.qe_prefix.back();
  for (const auto& g : p.groups)
    for (const FlowPlan::Round& rd : g) {
      if (!p.lats[rd.first].k.p) {
        const cudaError_t e = launch_clover(p.lats[rd.first], prec, nr, odd, parts, rd.qe_first, n, st);
        if (e != cudaSuccess) return e;
        ++*launches;
        continue;
      }
      cudaError_t e = launch_loops(set_of(rd, d_lats, d_prefix, 0, rd.loops), prec, nr, true, odd, 0, st);
      if (e == cudaSuccess)
        e = launch_loops_qe(set_of(rd, d_lats, d_prefix, 2, rd.qe), prec, nr, odd, parts, rd.qe_first, n, st);
      if (e != cudaSuccess) return e;
      *launches += 2;
    }
  return cudaSuccess;
}

}  // namespace qcb
