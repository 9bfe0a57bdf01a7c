// api_batch.cu — C ABI of lattice batches (include/qcb.h, "batches of lattices"):
// persistent multi-lattice launches, batched observables, the graph-captured workload
// and the tile autotuner.
#include <string.h>

#include <algorithm>
#include <chrono>
#include <fstream>
#include <map>
#include <new>
#include <sstream>
#include <string>
#include <vector>

#include "api_internal.h"
#include "batch.h"
#include "flow.h"

using namespace qcb;

namespace {

constexpr int DEFAULT_TILE = 256;

}  // namespace

struct qcb_batch {
  qcb_ctx* ctx = nullptr;
  int n = 0, prec = 0, nr = 0;
  std::vector<qcb_lattice*> lats;
  std::vector<uint32_t> hb_tile, flow_tile;
  BatchLat* d_desc = nullptr;  // n, of the lattices' links
  BatchLat* h_desc = nullptr;  // pinned mirror
  cudaEvent_t uploaded = nullptr;  // behind the latest copy from h_desc
  uint32_t* d_prefix = nullptr;  // hb (n+1) | plaquette (n+1)
  std::vector<uint32_t> h_prefix;
  uint32_t per_hb = 0, nred = 0;
  // Flow and clover: on the links with the copy fw0 as the other buffer, and on copies (fw0 with fw1).
  // The plans differ in their descriptors only.  They point into the context's loop buffer of
  // generation loops_gen, and are remade when that has been replaced.
  bool have_flow = false;
  uint64_t loops_gen = 0;
  FlowPlan flow[2];
  FlowLat* d_flow[2] = {nullptr, nullptr};
  uint32_t* d_flow_prefix = nullptr;  // the plan's prefix, then its qe_prefix
  double* d_qe = nullptr;             // clover partials
  uint32_t* d_done = nullptr;
  uint32_t* d_status = nullptr;  // [0] KP cap hits, [1] wait timeouts, [2] abort
  uint32_t* h_status = nullptr;
  double* d_scratch = nullptr;  // nred
  double* d_out = nullptr;
  double* h_out = nullptr;
  size_t out_cap = 0;
  cudaGraphExec_t exec = nullptr;
  qcb_batch_plan plan{};
  bool have_plan = false;
  bool graph_ok = true;
};

namespace {

int bfail(int code, const std::string& msg) { return qcb::set_error(code, msg.c_str()); }
int bcuda(cudaError_t e, const char* what) {
  return qcb::set_error(QCB_ERR_CUDA, (std::string(what) + ": " + cudaGetErrorString(e)).c_str());
}
#define BCU(call, what)                                 \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return bcuda(e_, what);      \
  } while (0)
#define BTRY(x)                  \
  do {                           \
    int r_ = (x);                \
    if (r_ != QCB_OK) return r_; \
  } while (0)

uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

void drop_flow(qcb_batch* b) {
  for (FlowLat*& d : b->d_flow) {
    cudaFree(d);
    d = nullptr;
  }
  cudaFree(b->d_flow_prefix);
  cudaFree(b->d_qe);
  b->d_flow_prefix = nullptr;
  b->d_qe = nullptr;
  b->have_flow = false;
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  b->have_plan = false;
}

// Groups of 32 links in a heatbath pass over the lattices, and those of the largest lattice.
void pass_groups(const std::vector<qcb_lattice*>& lats, uint64_t* groups, uint64_t* largest) {
  *groups = *largest = 0;
  for (const qcb_lattice* L : lats) {
    const uint64_t n = ceil_div(L->dev.g.Vh, 32u);
    *groups += n;
    *largest = std::max(*largest, n);
  }
}

// Copies the descriptors to the device, on the stream; the next change of the mirror waits for the copy
// (open_desc), which may be queued behind earlier launches.
int upload_desc(qcb_batch* b) {
  BCU(cudaMemcpyAsync(b->d_desc, b->h_desc, (size_t)b->n * sizeof(BatchLat), cudaMemcpyHostToDevice, b->ctx->stream),
      "descriptor upload");
  BCU(cudaEventRecord(b->uploaded, b->ctx->stream), "event");
  return QCB_OK;
}
int open_desc(qcb_batch* b) {
  BCU(cudaEventSynchronize(b->uploaded), "descriptor upload");
  return QCB_OK;
}

int ensure_flow_plan(qcb_batch* b);

// Rebuild descriptors and prefix sums from the lattices and tiles, upload them, and make the flow's plans.
int upload_layout(qcb_batch* b) {
  const int n = b->n;
  BTRY(open_desc(b));
  b->h_prefix.assign(2 * (n + 1), 0);
  uint32_t* ph = &b->h_prefix[0];
  uint32_t* pr = &b->h_prefix[n + 1];
  uint64_t groups = 0, largest = 0;
  pass_groups(b->lats, &groups, &largest);
  for (int l = 0; l < n; ++l) {
    const qcb_lattice* L = b->lats[l];
    const uint32_t tile = batch_tile(b->hb_tile[l], groups, largest, b->prec), nth = ceil_div(L->dev.g.Vh, tile);
    ph[l + 1] = ph[l] + nth;
    pr[l + 1] = pr[l] + ceil_div(L->dev.g.V, (uint32_t)batch_red_sites());
    BatchLat& d = b->h_desc[l];
    memset(&d, 0, sizeof d);
    d.g = L->dev.g;
    d.links = L->dev.links;
    d.tile = tile;
    d.ntiles = nth;
  }
  b->per_hb = ph[n];
  b->nred = pr[n];
  if (!b->d_scratch)  // its size is that of the lattices, whatever the tiles
    BCU(cudaMalloc(&b->d_scratch, (size_t)b->nred * sizeof(double)), "batch scratch");
  BCU(cudaMemcpyAsync(b->d_prefix, b->h_prefix.data(), b->h_prefix.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                      b->ctx->stream),
      "prefix upload");
  BTRY(upload_desc(b));
  BCU(cudaStreamSynchronize(b->ctx->stream), "sync");
  drop_flow(b);
  if (ensure_flow_plan(b) != QCB_OK) drop_flow(b);  // the call that needs it tries again
  return QCB_OK;
}

// Heatbath parameters go into the descriptors (host mirror + async upload).
int set_hb_params(qcb_batch* b, const double* betas, const uint64_t* seeds, const uint64_t* sweep_offsets) {
  for (int l = 0; l < b->n; ++l)
    if (!(betas[l] > 0.0)) return bfail(QCB_ERR_INVALID, "beta must be positive");
  BTRY(open_desc(b));
  for (int l = 0; l < b->n; ++l) {
    BatchLat& d = b->h_desc[l];
    d.beta = betas[l];
    d.k0 = (uint32_t)seeds[l];
    d.k1 = (uint32_t)(seeds[l] >> 32);
    d.sweep0 = (uint32_t)sweep_offsets[l];
  }
  return upload_desc(b);
}

// The lattices as items of a flow plan: on the links, or (copies) on fw0.
std::vector<FlowItem> flow_items(const std::vector<qcb_lattice*>& lats, const std::vector<uint32_t>& tile, int copies) {
  std::vector<FlowItem> items;
  for (size_t l = 0; l < lats.size(); ++l) {
    const qcb_lattice* L = lats[l];
    FlowItem it;
    it.L = L->dev;
    it.b = L->fw[0];
    if (copies) {
      it.L.links = L->fw[0];
      it.b = L->fw[1];
    }
    it.acc = L->fz;
    it.eps = 0.0;
    it.tile = tile[l];
    it.nsteps = 1 << 30;
    items.push_back(it);
  }
  return items;
}

// Plans and their device arrays on the context's loop buffer, made at the batch's creation and again
// when the tiles or the buffer have changed.
int ensure_flow_plan(qcb_batch* b) {
  size_t want = 0, least = 0;
  flow_plan_bytes(flow_items(b->lats, b->flow_tile, 0), &want, &least);
  reserve_loops(b->ctx, want, least);
  const LoopBuf& loops = b->ctx->loops;
  if (b->have_flow && b->loops_gen == loops.gen) return QCB_OK;
  drop_flow(b);
  b->loops_gen = loops.gen;
  for (int k = 0; k < 2; ++k) {
    b->flow[k] = flow_plan(flow_items(b->lats, b->flow_tile, k), loops);
    BCU(cudaMalloc(&b->d_flow[k], b->flow[k].lats.size() * sizeof(FlowLat)), "flow descriptors");
  }
  std::vector<uint32_t> pre = b->flow[0].prefix;
  pre.insert(pre.end(), b->flow[0].qe_prefix.begin(), b->flow[0].qe_prefix.end());
  BCU(cudaMalloc(&b->d_flow_prefix, pre.size() * sizeof(uint32_t)), "flow prefix");
  BCU(cudaMalloc(&b->d_qe, 2 * (size_t)b->flow[0].qe_prefix.back() * sizeof(double)), "clover partials");
  BCU(cudaMemcpyAsync(b->d_flow_prefix, pre.data(), pre.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                      b->ctx->stream),
      "flow prefix upload");
  BCU(cudaStreamSynchronize(b->ctx->stream), "sync");
  b->have_flow = true;
  return QCB_OK;
}

// Step size of the next launches into the descriptors of plan k (host and device).
int set_flow_eps(qcb_batch* b, int k, double eps) {
  for (FlowLat& r : b->flow[k].lats) r.eps = eps;
  BCU(cudaMemcpyAsync(b->d_flow[k], b->flow[k].lats.data(), b->flow[k].lats.size() * sizeof(FlowLat),
                      cudaMemcpyHostToDevice, b->ctx->stream),
      "flow descriptor upload");
  return QCB_OK;
}

int launch_hb(qcb_batch* b, int n_sweeps, int n_hits) {
  if (n_sweeps <= 0) return QCB_OK;
  BCU(cudaMemsetAsync(b->d_done, 0, b->n * sizeof(uint32_t), b->ctx->stream), "memset");
  BatchRun r;
  r.lats = b->d_desc;
  r.prefix = b->d_prefix;
  r.nlat = b->n;
  r.nlevels = 8u * (uint32_t)n_sweeps;
  r.per_level = b->per_hb;
  r.done = b->d_done;
  r.status = b->d_status;
  r.n_hits = n_hits;
  BCU(launch_batch(r, b->prec, b->nr, 128, 0, b->ctx->stream), "batched heatbath");
  b->ctx->launches++;
  return QCB_OK;
}

// n RK3 steps of plan k, from the links that `odd` selects.
int launch_flow(qcb_batch* b, int k, int odd, int n_steps) {
  BCU(run_flow_plan(b->flow[k], b->d_flow[k], b->d_flow_prefix, b->prec, b->nr, odd, n_steps, b->ctx->stream,
                    &b->ctx->launches),
      "batched flow");
  return QCB_OK;
}

int launch_plaq(qcb_batch* b, double* out) {
  BCU(launch_batch_plaquette(b->d_desc, b->d_prefix + b->n + 1, b->n, b->nred, b->prec, b->nr, b->d_scratch, out,
                             b->ctx->stream),
      "batched plaquette");
  b->ctx->launches += 2;
  return QCB_OK;
}
int launch_qe(qcb_batch* b, int k, int odd, double* out2) {
  BCU(run_qe_plan(b->flow[k], b->d_flow[k], b->d_flow_prefix, b->prec, b->nr, odd, b->d_qe, b->ctx->stream,
                  &b->ctx->launches),
      "batched clover");
  BCU(launch_batch_qe(b->d_desc, b->d_flow_prefix + b->flow[k].prefix.size(), b->n, b->flow[k].qe_prefix.back(),
                      b->d_qe, out2, b->ctx->stream),
      "batched clover Q/E");
  b->ctx->launches++;
  return QCB_OK;
}

int ensure_out(qcb_batch* b, size_t count) {
  if (b->out_cap >= count) return QCB_OK;
  cudaFree(b->d_out);
  cudaFreeHost(b->h_out);
  b->d_out = nullptr;
  b->h_out = nullptr;
  b->out_cap = 0;
  if (cudaMalloc(&b->d_out, count * sizeof(double)) != cudaSuccess ||
      cudaMallocHost(&b->h_out, count * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    return bfail(QCB_ERR_NOMEM, "cannot allocate batch result buffers");
  }
  b->out_cap = count;
  return QCB_OK;
}

// Read back status words of the batch (KP cap hits, wait timeouts) after a sync.
int batch_status(qcb_batch* b) {
  BCU(cudaMemcpyAsync(b->h_status, b->d_status, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, b->ctx->stream),
      "status copy");
  BCU(cudaStreamSynchronize(b->ctx->stream), "sync");
  const uint32_t kp = b->h_status[0], to = b->h_status[1];
  if (kp || to || b->h_status[2]) {
    BCU(cudaMemsetAsync(b->d_status, 0, 4 * sizeof(uint32_t), b->ctx->stream), "status reset");
    BCU(cudaStreamSynchronize(b->ctx->stream), "sync");
    if (to || b->h_status[2])
      return bfail(QCB_ERR_STATE, "batched kernel: a dependency wait timed out (" + std::to_string(to) +
                                      "); the launch was abandoned");
    return bfail(QCB_ERR_KP_CAP, "Kennedy-Pendleton draw hit its attempt cap " + std::to_string(kp) + " time(s)");
  }
  return QCB_OK;
}

// The whole plan (heatbath, plaquette, flow on copies with records) as stream work.
int enqueue_plan(qcb_batch* b, const qcb_batch_plan& p) {
  const int n = b->n;
  BTRY(launch_hb(b, p.n_sweeps, p.n_hits));
  // plaquette -> d_out[0 .. n)
  BTRY(launch_plaq(b, b->d_out));
  for (int l = 0; l < n; ++l) {
    qcb_lattice* L = b->lats[l];
    BCU(cudaMemcpyAsync(L->fw[0], L->dev.links, L->bytes, cudaMemcpyDeviceToDevice, b->ctx->stream), "copy");
  }
  // records: (Q, E) of group g -> d_out[n + 2 (g n + l)]
  int cum = 0;
  for (int g = 0; g <= p.n_groups; ++g) {
    BTRY(launch_qe(b, 1, cum & 1, b->d_out + n + 2 * (size_t)g * n));
    if (g < p.n_groups) {
      BTRY(launch_flow(b, 1, cum & 1, p.rk_per_group));
      cum += p.rk_per_group;
    }
  }
  BCU(cudaMemcpyAsync(b->h_out, b->d_out, (n + 2 * (size_t)(p.n_groups + 1) * n) * sizeof(double),
                      cudaMemcpyDeviceToHost, b->ctx->stream),
      "result copy");
  return QCB_OK;
}

void batch_free(qcb_batch* b);

bool same_plan(const qcb_batch_plan& a, const qcb_batch_plan& c) {
  return a.n_sweeps == c.n_sweeps && a.n_hits == c.n_hits && a.eps == c.eps && a.n_groups == c.n_groups &&
         a.rk_per_group == c.rk_per_group;
}

}  // namespace

extern "C" {

int qcb_batch_create(qcb_ctx* ctx, int n, qcb_lattice* const* lats, qcb_batch** out) {
  if (!ctx || !lats || !out || n <= 0) return bfail(QCB_ERR_INVALID, "bad batch arguments");
  *out = nullptr;
  for (int l = 0; l < n; ++l) {
    if (!lats[l]) return bfail(QCB_ERR_INVALID, "null lattice in batch");
    if (lats[l]->slab_tl) return bfail(QCB_ERR_INVALID, "a slab cannot join a batch (it needs halo exchanges)");
    if (lats[l]->ctx != ctx) return bfail(QCB_ERR_INVALID, "batch lattices must share the context");
    if (lats[l]->dev.prec != lats[0]->dev.prec || lats[l]->dev.nr != lats[0]->dev.nr)
      return bfail(QCB_ERR_INVALID, "batch lattices must share precision and storage");
  }
  std::lock_guard<std::mutex> lk(ctx->mu);
  BCU(cudaSetDevice(ctx->device), "cudaSetDevice");
  qcb_batch* b = new (std::nothrow) qcb_batch();
  if (!b) return bfail(QCB_ERR_NOMEM, "host allocation failed");
  b->ctx = ctx;
  b->n = n;
  b->prec = lats[0]->dev.prec;
  b->nr = lats[0]->dev.nr;
  b->lats.assign(lats, lats + n);
  b->hb_tile.assign(n, DEFAULT_TILE);
  b->flow_tile.assign(n, DEFAULT_TILE);
  auto fail_all = [&](int code) {
    b->ctx = nullptr;  // not counted yet
    batch_free(b);
    return code;
  };
  for (int l = 0; l < n; ++l) {
    int r = ensure_flow_space(b->lats[l]);
    if (r != QCB_OK) return fail_all(r);
  }
  if (cudaMalloc(&b->d_desc, (size_t)n * sizeof(BatchLat)) != cudaSuccess ||
      cudaMallocHost(&b->h_desc, (size_t)n * sizeof(BatchLat)) != cudaSuccess ||
      cudaEventCreateWithFlags(&b->uploaded, cudaEventDisableTiming) != cudaSuccess ||
      cudaMalloc(&b->d_prefix, 2 * (size_t)(n + 1) * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&b->d_done, (size_t)n * sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&b->d_status, 4 * sizeof(uint32_t)) != cudaSuccess ||
      cudaMallocHost(&b->h_status, 4 * sizeof(uint32_t)) != cudaSuccess) {
    cudaGetLastError();
    bfail(QCB_ERR_NOMEM, "cannot allocate batch descriptors");
    return fail_all(QCB_ERR_NOMEM);
  }
  if (cudaMemset(b->d_status, 0, 4 * sizeof(uint32_t)) != cudaSuccess) return fail_all(QCB_ERR_CUDA);
  int r = upload_layout(b);
  if (r != QCB_OK) return fail_all(r);
  ctx->refs++;  // under the context lock
  *out = b;
  return QCB_OK;
}

int qcb_batch_destroy(qcb_batch* b) {
  if (!b) return QCB_OK;
  qcb_ctx* c = b->ctx;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  batch_free(b);
  ctx_unref(c);
  return QCB_OK;
}

}  // extern "C"

namespace {
void batch_free(qcb_batch* b) {
  drop_flow(b);
  cudaFree(b->d_desc);
  cudaFreeHost(b->h_desc);
  if (b->uploaded) cudaEventDestroy(b->uploaded);
  cudaFree(b->d_prefix);
  cudaFree(b->d_done);
  cudaFree(b->d_status);
  cudaFreeHost(b->h_status);
  cudaFree(b->d_scratch);
  cudaFree(b->d_out);
  cudaFreeHost(b->h_out);
  cudaGetLastError();
  delete b;
}
}  // namespace

extern "C" {

int qcb_batch_set_tiles(qcb_batch* b, const int* hb_tile, const int* flow_tile) {
  if (!b) return bfail(QCB_ERR_INVALID, "null batch");
  for (int l = 0; l < b->n; ++l) {
    for (const int* t : {hb_tile, flow_tile})
      if (t && (t[l] < 32 || t[l] > 65536 || (t[l] & 31)))
        return bfail(QCB_ERR_INVALID, "tiles must be multiples of 32 in [32, 65536]");
  }
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  for (int l = 0; l < b->n; ++l) {
    if (hb_tile) b->hb_tile[l] = (uint32_t)hb_tile[l];
    if (flow_tile) b->flow_tile[l] = (uint32_t)flow_tile[l];
  }
  return upload_layout(b);
}

int qcb_batch_get_tiles(qcb_batch* b, int* hb_tile, int* flow_tile) {
  if (!b) return bfail(QCB_ERR_INVALID, "null batch");
  for (int l = 0; l < b->n; ++l) {
    if (hb_tile) hb_tile[l] = (int)b->hb_tile[l];
    if (flow_tile) flow_tile[l] = (int)b->flow_tile[l];
  }
  return QCB_OK;
}

int qcb_batch_heatbath(qcb_batch* b, const double* betas, int n_sweeps, int n_hits, const uint64_t* seeds,
                       const uint64_t* sweep_offsets) {
  if (!b || !betas || !seeds || !sweep_offsets) return bfail(QCB_ERR_INVALID, "null argument");
  if (n_sweeps < 0 || n_hits < 0 || n_hits > (1 << 20)) return bfail(QCB_ERR_INVALID, "bad sweep or hit count");
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  BTRY(set_hb_params(b, betas, seeds, sweep_offsets));
  return launch_hb(b, n_sweeps, n_hits);
}

int qcb_batch_flow_steps(qcb_batch* b, double eps, int n_steps) {
  if (!b) return bfail(QCB_ERR_INVALID, "null batch");
  if (n_steps < 0) return bfail(QCB_ERR_INVALID, "negative step count");
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  if (n_steps == 0) return QCB_OK;
  BTRY(ensure_flow_plan(b));
  BTRY(set_flow_eps(b, 0, eps));
  BTRY(launch_flow(b, 0, 0, n_steps));
  if (n_steps & 1)  // the result is in fw0
    for (int l = 0; l < b->n; ++l) {
      qcb_lattice* L = b->lats[l];
      BCU(cudaMemcpyAsync(L->dev.links, L->fw[0], L->bytes, cudaMemcpyDeviceToDevice, b->ctx->stream), "copy back");
    }
  return QCB_OK;
}

int qcb_batch_plaquette(qcb_batch* b, double* out) {
  if (!b || !out) return bfail(QCB_ERR_INVALID, "null argument");
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  BTRY(ensure_out(b, (size_t)b->n * 2));
  BTRY(launch_plaq(b, b->d_out));
  BCU(cudaMemcpyAsync(b->h_out, b->d_out, b->n * sizeof(double), cudaMemcpyDeviceToHost, b->ctx->stream), "D2H");
  BTRY(batch_status(b));
  memcpy(out, b->h_out, b->n * sizeof(double));
  return QCB_OK;
}

int qcb_batch_topo_qe(qcb_batch* b, double* q, double* e) {
  if (!b || !q || !e) return bfail(QCB_ERR_INVALID, "null argument");
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  BTRY(ensure_out(b, (size_t)b->n * 2));
  BTRY(ensure_flow_plan(b));
  BTRY(set_flow_eps(b, 0, 0.0));
  BTRY(launch_qe(b, 0, 0, b->d_out));
  BCU(cudaMemcpyAsync(b->h_out, b->d_out, 2 * b->n * sizeof(double), cudaMemcpyDeviceToHost, b->ctx->stream), "D2H");
  BTRY(batch_status(b));
  for (int l = 0; l < b->n; ++l) {
    q[l] = b->h_out[2 * l];
    e[l] = b->h_out[2 * l + 1];
  }
  return QCB_OK;
}

int qcb_batch_run(qcb_batch* b, const qcb_batch_plan* plan, const double* betas, const uint64_t* seeds,
                  const uint64_t* sweep_offsets, double* results, int* used_graph) {
  if (!b || !plan || !betas || !seeds || !sweep_offsets || !results) return bfail(QCB_ERR_INVALID, "null argument");
  const qcb_batch_plan& p = *plan;
  if (p.n_sweeps < 0 || p.n_hits < 0 || p.n_groups < 0 || p.rk_per_group < 0 || p.n_hits > (1 << 20))
    return bfail(QCB_ERR_INVALID, "bad plan");
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  const int n = b->n;
  BTRY(ensure_out(b, (size_t)n + 2 * (size_t)(p.n_groups + 1) * n));
  BTRY(set_hb_params(b, betas, seeds, sweep_offsets));
  BTRY(ensure_flow_plan(b));
  BTRY(set_flow_eps(b, 1, p.eps));
  bool graph = false;
  if (b->graph_ok) {
    if (!b->have_plan || !same_plan(b->plan, p) || !b->exec) {
      if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
      }
      // Capture the plan; on any capture failure fall back to direct launches.
      cudaGraph_t g = nullptr;
      cudaError_t e = cudaStreamBeginCapture(b->ctx->stream, cudaStreamCaptureModeThreadLocal);
      int r = QCB_OK;
      if (e == cudaSuccess) {
        r = enqueue_plan(b, p);
        e = cudaStreamEndCapture(b->ctx->stream, &g);
      }
      if (e == cudaSuccess && r == QCB_OK && g) e = cudaGraphInstantiate(&b->exec, g, 0);
      if (g) cudaGraphDestroy(g);
      if (e != cudaSuccess || r != QCB_OK || !b->exec) {
        cudaGetLastError();
        b->exec = nullptr;
        b->graph_ok = false;
      } else {
        b->plan = p;
        b->have_plan = true;
      }
    }
    if (b->exec) {
      BCU(cudaGraphLaunch(b->exec, b->ctx->stream), "graph launch");
      graph = true;
    }
  }
  if (!graph) BTRY(enqueue_plan(b, p));
  BTRY(batch_status(b));
  const int per = 1 + 3 * (p.n_groups + 1);
  for (int l = 0; l < n; ++l) {
    results[(size_t)l * per] = b->h_out[l];
    for (int g = 0; g <= p.n_groups; ++g) {
      double* rec = results + (size_t)l * per + 1 + 3 * g;
      rec[0] = (double)g * (double)p.rk_per_group * p.eps;
      rec[1] = b->h_out[n + 2 * ((size_t)g * n + l)];
      rec[2] = b->h_out[n + 2 * ((size_t)g * n + l) + 1];
    }
  }
  if (used_graph) *used_graph = graph ? 1 : 0;
  return QCB_OK;
}

int qcb_wait_selftest(qcb_ctx* ctx, double limit_s, uint32_t* timeouts, uint32_t* aborted) {
  if (!ctx || !timeouts || !aborted) return bfail(QCB_ERR_INVALID, "null argument");
  if (!(limit_s > 0.0 && limit_s <= 5.0)) return bfail(QCB_ERR_INVALID, "limit_s must be in (0, 5]");
  std::lock_guard<std::mutex> lk(ctx->mu);
  BCU(cudaSetDevice(ctx->device), "cudaSetDevice");
  uint32_t* d = nullptr;  // [0] the flag nothing sets, [1..4] status words
  BCU(cudaMalloc(&d, 8 * sizeof(uint32_t)), "self-test buffer");
  uint32_t h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  cudaError_t e = cudaMemsetAsync(d, 0, 8 * sizeof(uint32_t), ctx->stream);
  if (e == cudaSuccess) e = launch_wait_probe(d, d + 1, (uint64_t)(limit_s * 1e9), 4, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, 8 * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cudaFree(d);
  if (e != cudaSuccess) return bcuda(e, "wait self-test");
  ctx->launches++;
  *timeouts = h[2];
  *aborted = h[3];
  if (h[4] != 0) return bfail(QCB_ERR_STATE, "a wait on a flag that nothing sets succeeded");
  return QCB_OK;
}

}  // extern "C"

// ---- autotuner --------------------------------------------------------------------------
namespace {

std::map<std::string, int> read_cache(const char* path) {
  std::map<std::string, int> m;
  if (!path) return m;
  std::ifstream f(path);
  std::string line;
  while (std::getline(f, line)) {
    // lines of the form   "key": value,
    size_t a = line.find('"'), b2 = (a == std::string::npos) ? a : line.find('"', a + 1);
    if (a == std::string::npos || b2 == std::string::npos) continue;
    size_t c = line.find(':', b2);
    if (c == std::string::npos) continue;
    m[line.substr(a + 1, b2 - a - 1)] = atoi(line.c_str() + c + 1);
  }
  return m;
}

void write_cache(const char* path, const std::map<std::string, int>& m) {
  if (!path) return;
  std::ofstream f(path);
  f << "{\n";
  size_t k = 0;
  for (auto& kv : m) f << "  \"" << kv.first << "\": " << kv.second << (++k < m.size() ? ",\n" : "\n");
  f << "}\n";
}

}  // namespace

namespace {

// Times the whole batch on scratch copies of its lattices (heatbath on fw1, flow on fw1 and fw0), four
// sweeps (one alone favours smaller items than a long run) or an RK3 step, with given work items: the
// best of three runs, or the first that is not below `limit`.
struct Tuner {
  qcb_batch* b;
  BatchLat* d_dsc = nullptr;
  FlowLat* d_flow = nullptr;
  uint32_t* d_pre = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  uint64_t groups = 0, largest = 0;

  explicit Tuner(qcb_batch* batch) : b(batch) { pass_groups(b->lats, &groups, &largest); }
  Tuner(const Tuner&) = delete;
  ~Tuner() {
    cudaFree(d_dsc);
    cudaFree(d_flow);
    cudaFree(d_pre);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  }
  int open() {
    BTRY(ensure_flow_plan(b));
    const size_t rounds = b->flow[0].lats.size();
    BCU(cudaMalloc(&d_dsc, b->n * sizeof(BatchLat)), "tune alloc");
    BCU(cudaMalloc(&d_flow, rounds * sizeof(FlowLat)), "tune alloc");
    BCU(cudaMalloc(&d_pre, 6 * rounds * sizeof(uint32_t)), "tune alloc");  // at least n + 1 for the heatbath
    BCU(cudaEventCreate(&e0), "event");
    BCU(cudaEventCreate(&e1), "event");
    for (qcb_lattice* L : b->lats)
      BCU(cudaMemcpyAsync(L->fw[1], L->dev.links, L->bytes, cudaMemcpyDeviceToDevice, b->ctx->stream), "copy");
    return QCB_OK;
  }
  uint32_t hb_item(uint32_t most) const { return batch_tile(most, groups, largest, b->prec); }

  template <typename F>
  int best_of(const F& launch, float limit, float* ms) {
    *ms = 1e30f;
    for (int rep = 0; rep < 3; ++rep) {
      BCU(cudaMemsetAsync(b->d_done, 0, b->n * sizeof(uint32_t), b->ctx->stream), "memset");
      BCU(cudaEventRecord(e0, b->ctx->stream), "event");
      BTRY(launch());
      BCU(cudaEventRecord(e1, b->ctx->stream), "event");
      BCU(cudaEventSynchronize(e1), "event sync");
      float t = 0;
      BCU(cudaEventElapsedTime(&t, e0, e1), "elapsed");
      *ms = std::min(*ms, t);
      if (t >= limit) break;
    }
    return QCB_OK;
  }
  int heatbath(const std::vector<uint32_t>& tile, float limit, float* ms) {
    std::vector<BatchLat> dsc(b->n);
    std::vector<uint32_t> pre(b->n + 1, 0);
    for (int l = 0; l < b->n; ++l) {
      BatchLat& d = dsc[l];
      memset(&d, 0, sizeof d);
      d.g = b->lats[l]->dev.g;
      d.links = b->lats[l]->fw[1];
      d.beta = 6.0;
      d.k0 = 12345u;
      d.tile = hb_item(tile[l]);
      d.ntiles = ceil_div(d.g.Vh, d.tile);
      pre[l + 1] = pre[l] + d.ntiles;
    }
    BCU(cudaMemcpyAsync(d_dsc, dsc.data(), b->n * sizeof(BatchLat), cudaMemcpyHostToDevice, b->ctx->stream), "H2D");
    BCU(cudaMemcpyAsync(d_pre, pre.data(), pre.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, b->ctx->stream), "H2D");
    BatchRun r;
    r.lats = d_dsc;
    r.prefix = d_pre;
    r.nlat = b->n;
    r.per_level = pre[b->n];
    r.done = b->d_done;
    r.status = b->d_status;
    r.n_hits = 1;
    r.nlevels = 32;
    return best_of([&]() -> int {
      BCU(launch_batch(r, b->prec, b->nr, 128, 0, b->ctx->stream), "tune launch");
      b->ctx->launches++;
      return QCB_OK;
    }, limit, ms);
  }
  int flow(const std::vector<uint32_t>& tile, float limit, float* ms) {
    std::vector<FlowItem> items = flow_items(b->lats, tile, 0);
    for (int l = 0; l < b->n; ++l) {
      items[l].L.links = b->lats[l]->fw[1];
      items[l].b = b->lats[l]->fw[0];
      items[l].eps = 0.02;
    }
    const FlowPlan fp = flow_plan(items, b->ctx->loops);
    BCU(cudaMemcpyAsync(d_flow, fp.lats.data(), fp.lats.size() * sizeof(FlowLat), cudaMemcpyHostToDevice,
                        b->ctx->stream),
        "H2D");
    BCU(cudaMemcpyAsync(d_pre, fp.prefix.data(), fp.prefix.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                        b->ctx->stream),
        "H2D");
    return best_of([&]() -> int {
      BCU(run_flow_plan(fp, d_flow, d_pre, b->prec, b->nr, 0, 1, b->ctx->stream, &b->ctx->launches), "tune launch");
      return QCB_OK;
    }, limit, ms);
  }
};

}  // namespace

extern "C" int qcb_batch_autotune(qcb_batch* b, const char* cache_path) {
  if (!b) return bfail(QCB_ERR_INVALID, "null batch");
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  BCU(cudaSetDevice(b->ctx->device), "cudaSetDevice");
  cudaDeviceProp prop;
  BCU(cudaGetDeviceProperties(&prop, b->ctx->device), "device properties");
  const std::string pfx = std::string(prop.name) + "|" + (b->prec == QCB_FP64 ? "fp64" : "fp32") + "-" +
                          std::to_string(b->nr) + "|";
  auto cache = read_cache(cache_path);
  // distinct sizes
  std::map<std::string, std::vector<int>> by_size;
  for (int l = 0; l < b->n; ++l) {
    const Geom& g = b->lats[l]->dev.g;
    by_size[std::to_string(g.L[0]) + "x" + std::to_string(g.L[1]) + "x" + std::to_string(g.L[2]) + "x" +
            std::to_string(g.L[3])]
        .push_back(l);
  }
  // What is not bounded by a choice stays at the default bound, under which the launch's own rule
  // (batch_tile, flow_plan) decides.
  std::vector<uint32_t> tile[2] = {std::vector<uint32_t>(b->n, DEFAULT_TILE), std::vector<uint32_t>(b->n, DEFAULT_TILE)};
  std::vector<std::string> open;
  for (auto& kv : by_size) {
    if (cache.count(pfx + "hb|" + kv.first) && cache.count(pfx + "flow|" + kv.first)) {
      for (int l : kv.second) {
        tile[0][l] = (uint32_t)cache[pfx + "hb|" + kv.first];
        tile[1][l] = (uint32_t)cache[pfx + "flow|" + kv.first];
      }
    } else {
      open.push_back(kv.first);
    }
  }
  if (!open.empty()) {
    Tuner t(b);
    BTRY(t.open());
    for (int kind = 0; kind < 2; ++kind) {
      // the bounds under which the launch differs from the one under the default bound, one for each item
      // size, from half of the rule's on (FP32 heatbath, 54 lattices: 32 links take 10.4 ms, 160 8.4)
      const uint32_t rule = kind == 0 ? t.hb_item(DEFAULT_TILE) : flow_tile_most(flow_items(b->lats, tile[1], 0));
      std::vector<uint32_t> cands;
      uint32_t last = 0;
      for (uint32_t c = 32; c < rule; c += 32) {
        const uint32_t item = kind == 0 ? t.hb_item(c) : c;
        if (item != last && item != rule && 2 * item >= rule) cands.push_back(c);
        last = item;
      }
      auto time = [&](float limit, float* ms) {
        return kind == 0 ? t.heatbath(tile[0], limit, ms) : t.flow(tile[1], limit, ms);
      };
      float base = 0;
      if (!cands.empty()) BTRY(time(1e30f, &base));
      for (const std::string& size : open) {
        uint32_t pick = DEFAULT_TILE;
        for (uint32_t c : cands) {
          for (int l : by_size[size]) tile[kind][l] = c;
          const float below = 0.98f * base;  // by more than repeated runs differ
          float ms = 0;
          BTRY(time(below, &ms));
          if (ms < below) {
            base = ms;
            pick = c;
          }
        }
        for (int l : by_size[size]) tile[kind][l] = pick;
        cache[pfx + (kind == 0 ? "hb|" : "flow|") + size] = (int)pick;
      }
    }
  }
  BTRY(batch_status(b));
  write_cache(cache_path, cache);
  b->hb_tile = tile[0];
  b->flow_tile = tile[1];
  return upload_layout(b);
}
