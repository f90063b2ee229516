// Batched and served explicit Euler (include/subfv.h, subfv_ns_batch_*): many independent
// problems, each on its own device mesh, advanced together in shared persistent launches
// (launch_ns_batch_step) with the step loop captured once in a CUDA graph. No counterpart
// in the reference, whose ns_main.F90:83-107 loop advances one mesh per process.
//
// Concurrency model. All step work runs on the batch stream. Admission work (state
// allocation, upload, packing) runs on the admitted mesh's own stream and is joined to
// the batch stream by an event, so a request can be admitted while earlier chunks are
// still running. The table of in-flight problems lives in device memory and is rewritten
// in stream order; the captured graph reads its size from the device, so it stays valid
// as problems join and leave. Removed slots are reused only after the batch stream has
// passed the point where they left the table; their memory is freed stream-ordered.
#include <algorithm>
#include <cstring>
#include <deque>
#include <vector>

#include "handles.cuh"
#include "ns.cuh"
#include "pool.cuh"

using namespace subfv;

namespace {

struct Slot {
  subfv_mesh* mesh = nullptr;
  int owns_mesh = 0;
  int tiles = 0;           // admitted with its mesh's node codes, which the admission's event covers
  int live = 0;            // holds a problem (in the table or waiting to be removed)
  cudaEvent_t free_ev = nullptr;  // recorded on the batch stream when the slot left the table
  double *U0 = nullptr, *U1 = nullptr, *fs = nullptr, *rhs1 = nullptr, *rhs2 = nullptr;
  double *ngrad = nullptr, *grad = nullptr, *delta = nullptr, *partial = nullptr;
  int64_t bytes = 0;       // state + mesh bytes charged against the budget
  int64_t caches = 0;      // bytes of mesh caches built for its admission, beside the charge
  unsigned long long seen_epoch = 0;  // the mesh geometry the table's copy of the mesh belongs to
  unsigned long long first_snap = 0;  // the first snapshot that includes this problem
  double t0 = 0.0;
};

struct Snapshot {
  NsScalars* sc = nullptr;   // pinned
  unsigned* status = nullptr;
  cudaEvent_t ev = nullptr;
  int pending = 0;
  unsigned long long seq = 0;  // snapshots are numbered in enqueue order from 1
};

// The corner sums and, in second order, the vertex records, which end where the sums' room of
// 15 doubles a vertex would: the sums are dead from their gather to the next node kernel,
// and the records live only between the two gradient kernels that run then. A record's nine
// further doubles (the weights and extremes) so take no room of their own on any mesh of
// more than two cells.
size_t corner_and_vertex_doubles(const DevMesh& d, int second_order) {
  const size_t fs = kNsFs * (size_t)d.nse;
  return second_order ? std::max(fs + 15 * (size_t)d.nv, kNsVert * (size_t)d.nv) : fs;
}

// The per-problem state: a first-order scheme needs neither the second stage's state nor
// the gradients nor the second residual.
int64_t state_bytes(const DevMesh& d, int second_order) {
  const int64_t ne = d.ne;
  const int64_t o1 = kRec * ne + (int64_t)corner_and_vertex_doubles(d, second_order) + kRhs * ne + 5 * ne +
                     6 * (int64_t)ns_partial_blocks(d);
  const int64_t o2 = kRec * ne + kRhs * ne + 15 * ne;
  return 8 * (o1 + (second_order ? o2 : 0));
}

// What admission would add to the mesh for the faster kernels: the node tiles' codes and the
// nodal gradients' pseudo-inverses. The mesh keeps them, whichever problem comes next, so
// they are no problem's charge; they are built while they fit the budget beside the charges,
// and a problem that fits only without them runs on the kernels that do without.
int64_t cache_bytes(const DevMesh& d, const NsParams& P) {
  int64_t n = 0;
  if (!d.node_codes && node_tile_scheme(P)) n += node_codes_bytes(d);
  if (!d.npinv && !d.moving && P.second_order) n += 72 * (int64_t)d.nv;
  return n;
}

}  // namespace

struct subfv_ns_batch {
  NsParams P{};
  cudaStream_t stream = nullptr;
  int cap = 0;
  int64_t budget = 0, used = 0, caches = 0;
  NsScalars* sc = nullptr;  // device [cap]
  unsigned* status = nullptr;  // device [cap]
  std::vector<Slot> slots;
  std::vector<int> order;  // live slots in table order
  // device table and its pinned host staging (double-buffered staging)
  NsTable tab{};
  NsItem* h_items[2] = {nullptr, nullptr};
  int* h_w[2] = {nullptr, nullptr};  // [wv (cap+1) | wc (cap+1) | wt (cap+1) | hdr (4)]
  cudaEvent_t stage_ev[2] = {nullptr, nullptr};
  int stage_cur = 0;
  bool dirty = true;
  // the captured step loop, with the other node kernels and with the tiles
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  int captures = 0;
  Snapshot snap[2];
  std::deque<int> outstanding;  // snapshot indices in enqueue order
  int snap_next = 0;
  // the latest completed snapshot, copied out of the pinned ring
  std::vector<NsScalars> last_sc;
  std::vector<unsigned> last_status;
  bool have_last = false;
  unsigned long long last_seq = 0, snap_count = 0;
  std::vector<int> retiring;    // removed slots whose memory is freed at the next table rewrite
};

namespace {

template <class T>
int dalloc_async(T** p, size_t n, cudaStream_t s) {
  if (pool_alloc((void**)p, std::max<size_t>(n, 1) * sizeof(T), s)) return -1;
  SUBFV_CUDA(cudaMemsetAsync(*p, 0, std::max<size_t>(n, 1) * sizeof(T), s));
  return 0;
}

void slot_free_state(Slot& q, cudaStream_t s) {
  double* bufs[] = {q.U0, q.U1, q.fs, q.rhs1, q.rhs2, q.grad, q.delta, q.partial};  // ngrad lies in fs
  for (double* b : bufs) pool_free(b, s);
  q.U0 = q.U1 = q.fs = q.rhs1 = q.rhs2 = q.ngrad = q.grad = q.delta = q.partial = nullptr;
}

constexpr int kGraphSteps = 8;

// destroys a captured loop once no launch of it runs any more
int graph_drop(subfv_ns_batch* b, int which) {
  if (!b->graph[which]) return 0;
  SUBFV_CUDA(cudaStreamSynchronize(b->stream));
  cudaGraphExecDestroy(b->graph[which]);
  b->graph[which] = nullptr;
  return 0;
}

int graph_for(subfv_ns_batch* b) {
  cudaGraphExec_t& exec = b->graph[b->tab.tiles];
  if (exec) return 0;
  cudaGraph_t g;
  SUBFV_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  for (int i = 0; i < kGraphSteps; ++i) launch_ns_batch_step(b->tab, b->P, b->stream);
  SUBFV_CUDA(cudaStreamEndCapture(b->stream, &g));
  cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    exec = nullptr;
    set_error(std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    return -1;
  }
  ++b->captures;
  return 0;
}

// Rewrite the device table from the live slots (stream-ordered on the batch stream).
int table_upload(subfv_ns_batch* b) {
  for (int i : b->order) {  // a mesh whose vertices moved since the table was written
    Slot& q = b->slots[i];
    DevMesh& d = q.mesh->d;
    if (q.seen_epoch == d.geom_epoch) continue;
    if (b->P.second_order && d.npinv) {
      if (ensure_nodal_pinv(&d, false)) return -1;
      SUBFV_CUDA(cudaEventRecord(q.free_ev, d.stream));
      SUBFV_CUDA(cudaStreamWaitEvent(b->stream, q.free_ev, 0));
    }
    q.seen_epoch = d.geom_epoch;
    b->dirty = true;
  }
  if (!b->dirty) return 0;
  const int k = b->stage_cur;
  SUBFV_CUDA(cudaEventSynchronize(b->stage_ev[k]));  // the staging copy issued two updates ago
  NsItem* it = b->h_items[k];
  int* wv = b->h_w[k];
  int* wc = wv + (b->cap + 1);
  int* wt = wc + (b->cap + 1);
  int* hdr = wt + (b->cap + 1);
  const int n = (int)b->order.size();
  int group = 8, tiles = 1;
  for (int i = 0; i < n; ++i) {
    const DevMesh& d = b->slots[b->order[i]].mesh->d;
    group = std::max(group, ns_node_lanes(d));
    tiles = tiles && b->slots[b->order[i]].tiles;
  }
  // The loop without tiles is captured for one group size; the one with them has none, and
  // each stays for when a mesh beyond the tiles joins or leaves.
  if (n) {
    if (group != b->tab.group && graph_drop(b, 0)) return -1;
    b->tab.group = group;
    b->tab.tiles = tiles;
  }
  const int nbv = b->tab.block_v;  // vertices per work block
  wv[0] = wc[0] = wt[0] = 0;
  for (int i = 0; i < n; ++i) {
    Slot& q = b->slots[b->order[i]];
    NsItem& I = it[i];
    I.m = q.mesh->d;
    I.m.status = b->status + b->order[i];
    I.U0 = q.U0;
    I.U1 = q.U1;
    I.fs = q.fs;
    I.rhs1 = q.rhs1;
    I.rhs2 = q.rhs2;
    I.ngrad = q.ngrad;
    I.grad = q.grad;
    I.delta = q.delta;
    I.partial = q.partial;
    I.sc = b->sc + b->order[i];
    wv[i + 1] = wv[i] + (I.m.nv + nbv - 1) / nbv;
    wc[i + 1] = wc[i] + (I.m.ne + kNsCellBlock - 1) / kNsCellBlock;
    wt[i + 1] = wt[i] + node_tiles(I.m);
  }
  hdr[0] = n;
  if (n) SUBFV_CUDA(cudaMemcpyAsync(b->tab.items, it, n * sizeof(NsItem), cudaMemcpyHostToDevice, b->stream));
  SUBFV_CUDA(cudaMemcpyAsync(b->tab.wv, wv, (n + 1) * sizeof(int), cudaMemcpyHostToDevice, b->stream));
  SUBFV_CUDA(cudaMemcpyAsync(b->tab.wc, wc, (n + 1) * sizeof(int), cudaMemcpyHostToDevice, b->stream));
  SUBFV_CUDA(cudaMemcpyAsync(b->tab.wt, wt, (n + 1) * sizeof(int), cudaMemcpyHostToDevice, b->stream));
  SUBFV_CUDA(cudaMemcpyAsync(b->tab.hdr, hdr, sizeof(int), cudaMemcpyHostToDevice, b->stream));
  SUBFV_CUDA(cudaEventRecord(b->stage_ev[k], b->stream));
  b->stage_cur ^= 1;
  b->dirty = false;
  // slots that left the table: their frees are stream-ordered after the rewrite
  for (int r : b->retiring) {
    Slot& q = b->slots[r];
    slot_free_state(q, b->stream);
    SUBFV_CUDA(cudaEventRecord(q.free_ev, b->stream));
    if (q.owns_mesh && q.mesh) {
      SUBFV_CUDA(cudaStreamWaitEvent(q.mesh->d.stream, q.free_ev, 0));
      subfv_mesh_destroy(q.mesh);
    }
    q.mesh = nullptr;
  }
  b->retiring.clear();
  return 0;
}

void snapshot_take(subfv_ns_batch* b, Snapshot& s) {
  s.pending = 0;
  b->outstanding.pop_front();
  std::memcpy(b->last_sc.data(), s.sc, b->cap * sizeof(NsScalars));
  std::memcpy(b->last_status.data(), s.status, b->cap * sizeof(unsigned));
  b->have_last = true;
  b->last_seq = s.seq;
}

int snapshot_enqueue(subfv_ns_batch* b) {
  const int k = b->snap_next;
  Snapshot& s = b->snap[k];
  if (s.pending) {  // both buffers in flight: retire the older one first
    SUBFV_CUDA(cudaEventSynchronize(s.ev));
    snapshot_take(b, s);
  }
  SUBFV_CUDA(cudaMemcpyAsync(s.sc, b->sc, b->cap * sizeof(NsScalars), cudaMemcpyDeviceToHost, b->stream));
  SUBFV_CUDA(cudaMemcpyAsync(s.status, b->status, b->cap * sizeof(unsigned), cudaMemcpyDeviceToHost, b->stream));
  SUBFV_CUDA(cudaEventRecord(s.ev, b->stream));
  s.pending = 1;
  s.seq = ++b->snap_count;
  b->outstanding.push_back(k);
  b->snap_next ^= 1;
  return 0;
}

}  // namespace

extern "C" {

int subfv_ns_batch_create(const subfv_ns_cfg* cfg, int capacity, int64_t budget_bytes, subfv_ns_batch** out) {
  if (!cfg || !out || capacity < 1 || capacity > (1 << 20) || budget_bytes <= 0 ||
      (cfg->scheme < 1 || cfg->scheme > 8 || cfg->scheme == 7) || (cfg->method < 0 || cfg->method > 6) ||
      cfg->local_time_step != 0 || cfg->n_bc < 0 || cfg->n_bc > 16 || (cfg->precision < 0 || cfg->precision > 2) ||
      cfg->activate_diffusion) {
    set_error("subfv_ns_batch_create: bad argument or unsupported configuration (diffusion is not batched)");
    return -2;
  }
  for (int i = 0; i < cfg->n_bc; ++i)
    if (cfg->bc_type[i] < 1 || cfg->bc_type[i] > 9) {
      set_error("subfv_ns_batch_create: boundary kind not recognized (1-9)");
      return -2;
    }
  auto* b = new subfv_ns_batch();
  b->P = ns_params_from(*cfg);
  b->cap = capacity;
  b->budget = budget_bytes;
  b->slots.resize(capacity);
  b->last_sc.resize(capacity);
  b->last_status.resize(capacity);
  auto fail = [&]() {
    subfv_ns_batch_destroy(b);
    return -1;
  };
  if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) return fail();
  const size_t nw = 3 * (size_t)(capacity + 1) + 4;
  if (cudaMalloc(&b->sc, capacity * sizeof(NsScalars)) != cudaSuccess ||
      cudaMalloc(&b->status, capacity * sizeof(unsigned)) != cudaSuccess ||
      cudaMalloc(&b->tab.items, capacity * sizeof(NsItem)) != cudaSuccess ||
      cudaMalloc(&b->tab.wv, nw * sizeof(int)) != cudaSuccess)
    return fail();
  cudaMemsetAsync(b->sc, 0, capacity * sizeof(NsScalars), b->stream);
  cudaMemsetAsync(b->status, 0, capacity * sizeof(unsigned), b->stream);
  cudaMemsetAsync(b->tab.wv, 0, nw * sizeof(int), b->stream);
  b->tab.wc = b->tab.wv + (capacity + 1);
  b->tab.wt = b->tab.wc + (capacity + 1);
  b->tab.hdr = b->tab.wt + (capacity + 1);
  b->tab.cap = capacity;
  b->tab.block_v = 128;
  b->tab.group = 8;
  b->tab.grid_v = b->tab.grid_c = 148 * 8;
  for (int k = 0; k < 2; ++k) {
    if (cudaHostAlloc((void**)&b->h_items[k], capacity * sizeof(NsItem), cudaHostAllocDefault) != cudaSuccess ||
        cudaHostAlloc((void**)&b->h_w[k], nw * sizeof(int), cudaHostAllocDefault) != cudaSuccess ||
        cudaEventCreateWithFlags(&b->stage_ev[k], cudaEventDisableTiming) != cudaSuccess ||
        cudaHostAlloc((void**)&b->snap[k].sc, capacity * sizeof(NsScalars), cudaHostAllocDefault) != cudaSuccess ||
        cudaHostAlloc((void**)&b->snap[k].status, capacity * sizeof(unsigned), cudaHostAllocDefault) != cudaSuccess ||
        cudaEventCreateWithFlags(&b->snap[k].ev, cudaEventDisableTiming) != cudaSuccess)
      return fail();
    std::memset(b->snap[k].sc, 0, capacity * sizeof(NsScalars));
    std::memset(b->snap[k].status, 0, capacity * sizeof(unsigned));
  }
  for (auto& q : b->slots)
    if (cudaEventCreateWithFlags(&q.free_ev, cudaEventDisableTiming) != cudaSuccess) return fail();
  if (cudaDeviceSynchronize() != cudaSuccess) return fail();
  *out = b;
  return 0;
}

int subfv_ns_batch_destroy(subfv_ns_batch* b) {
  if (!b) return 0;
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (auto& q : b->slots) {
    if (q.live || q.mesh) {
      slot_free_state(q, b->stream);
      if (q.owns_mesh) subfv_mesh_destroy(q.mesh);
    }
    if (q.free_ev) cudaEventDestroy(q.free_ev);
  }
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (cudaGraphExec_t g : b->graph)
    if (g) cudaGraphExecDestroy(g);
  cudaFree(b->sc);
  cudaFree(b->status);
  cudaFree(b->tab.items);
  cudaFree(b->tab.wv);
  for (int k = 0; k < 2; ++k) {
    cudaFreeHost(b->h_items[k]);
    cudaFreeHost(b->h_w[k]);
    if (b->stage_ev[k]) cudaEventDestroy(b->stage_ev[k]);
    cudaFreeHost(b->snap[k].sc);
    cudaFreeHost(b->snap[k].status);
    if (b->snap[k].ev) cudaEventDestroy(b->snap[k].ev);
  }
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return 0;
}

int64_t subfv_ns_batch_state_bytes(const subfv_ns_batch* b, const subfv_mesh* m) {
  return (b && m) ? state_bytes(m->d, b->P.second_order) : -2;
}

int64_t subfv_ns_batch_free_bytes(const subfv_ns_batch* b) { return b ? b->budget - b->used : -2; }

int subfv_ns_batch_add(subfv_ns_batch* b, subfv_mesh* m, int take_mesh, const double* sol, double t0, double tmax,
                       int* slot) {
  if (!b || !m || !sol || !slot) {
    set_error("subfv_ns_batch_add: null argument");
    return -2;
  }
  if (handle_ensure_full_geometry(m->d)) return -1;
  const DevMesh& d = m->d;
  if (ns_node_lanes(d) == 0) {
    set_error("subfv_ns_batch_add: a vertex has more than 32 subfaces or subcells");
    return -2;
  }
  const int64_t need = state_bytes(d, b->P.second_order) + (int64_t)d.bytes;
  int k = -1;
  for (int i = 0; i < b->cap && k < 0; ++i) {
    Slot& q = b->slots[i];
    if (!q.live && !q.mesh && cudaEventQuery(q.free_ev) == cudaSuccess) k = i;
  }
  if (k < 0 || b->used + need > b->budget) {
    set_error("subfv_ns_batch_add: no free slot or HBM budget exhausted");
    return SUBFV_BATCH_FULL;
  }
  Slot& q = b->slots[k];
  int64_t caches = cache_bytes(d, b->P);
  if (b->used + need + b->caches + caches <= b->budget) {
    if (ensure_node_codes(&m->d, b->P) || (b->P.second_order && ensure_nodal_pinv(&m->d, false))) return -1;
  } else {
    caches = 0;
    if (b->P.second_order && d.npinv && ensure_nodal_pinv(&m->d, false)) return -1;
  }
  cudaStream_t s = d.stream;
  const size_t ne = d.ne, nfs = corner_and_vertex_doubles(d, b->P.second_order);
  double* stage = nullptr;
  const bool o2 = b->P.second_order != 0;
  if (dalloc_async(&q.U0, kRec * ne, s) || dalloc_async(&q.fs, nfs, s) ||
      dalloc_async(&q.rhs1, kRhs * ne, s) || dalloc_async(&q.delta, 5 * ne, s) ||
      dalloc_async(&q.partial, 6 * (size_t)ns_partial_blocks(d), s) ||
      (o2 && (dalloc_async(&q.U1, kRec * ne, s) || dalloc_async(&q.rhs2, kRhs * ne, s) ||
              dalloc_async(&q.grad, 15 * ne, s))) ||
      pool_alloc((void**)&stage, 5 * ne * sizeof(double), s)) {
    slot_free_state(q, s);
    return -1;
  }
  if (o2) q.ngrad = q.fs + (nfs - kNsVert * (size_t)d.nv);
  NsScalars h{};
  h.dtred = 1e10;
  h.omega = 1.0;
  h.t = t0;
  h.final_res = -1.0;
  h.tmax = tmax;
  h.done = (t0 < tmax) ? 0 : 1;
  const unsigned zero = 0;
  SUBFV_CUDA(cudaMemcpyAsync(stage, sol, 5 * ne * sizeof(double), cudaMemcpyHostToDevice, s));
  SUBFV_CUDA(cudaMemcpyAsync(b->sc + k, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  SUBFV_CUDA(cudaMemcpyAsync(b->status + k, &zero, sizeof(zero), cudaMemcpyHostToDevice, s));
  launch_ns_pack(d, stage, q.U0);
  pool_free(stage, s);
  cudaEvent_t ready;
  SUBFV_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
  SUBFV_CUDA(cudaEventRecord(ready, s));
  SUBFV_CUDA(cudaStreamWaitEvent(b->stream, ready, 0));
  cudaEventDestroy(ready);  // released once the wait is satisfied
  SUBFV_CUDA(cudaGetLastError());
  q.mesh = m;
  q.owns_mesh = take_mesh ? 1 : 0;
  q.live = 1;
  q.tiles = d.node_codes && node_tile_scheme(b->P);
  q.bytes = need;
  q.caches = caches;
  b->caches += caches;
  q.first_snap = b->snap_count + 1;
  q.t0 = t0;
  q.seen_epoch = d.geom_epoch;
  b->used += need;
  b->order.push_back(k);
  b->dirty = true;
  *slot = k;
  return 0;
}

int subfv_ns_batch_remove(subfv_ns_batch* b, int slot) {
  if (!b || slot < 0 || slot >= b->cap || !b->slots[slot].live) {
    set_error("subfv_ns_batch_remove: bad slot");
    return -2;
  }
  Slot& q = b->slots[slot];
  auto it = std::find(b->order.begin(), b->order.end(), slot);
  if (it != b->order.end()) b->order.erase(it);
  b->used -= q.bytes;
  b->caches -= q.caches;
  q.caches = 0;
  q.bytes = 0;
  q.live = 0;
  b->retiring.push_back(slot);  // freed after the table rewrite that drops it
  b->dirty = true;
  return 0;
}

int subfv_probe_ns_captures(const subfv_ns_batch* b) { return b ? b->captures : -2; }

int subfv_ns_batch_set_launch(subfv_ns_batch* b, int block_v, int grid_v, int grid_c) {
  if (!b || (block_v != 64 && block_v != 128 && block_v != 256) || grid_v < 1 || grid_c < 1) {
    set_error("subfv_ns_batch_set_launch: block_v must be 64, 128 or 256 and the grids positive");
    return -2;
  }
  if (block_v != b->tab.block_v) b->dirty = true;
  if (block_v != b->tab.block_v || grid_v != b->tab.grid_v || grid_c != b->tab.grid_c) {
    b->tab.block_v = block_v;
    b->tab.grid_v = grid_v;
    b->tab.grid_c = grid_c;
    if (graph_drop(b, 0) || graph_drop(b, 1)) return -1;
  }
  return 0;
}

int subfv_ns_batch_set_node_kernel(subfv_ns_batch* b, int lanes) {
  if (!b || (lanes != 0 && lanes != 1 && lanes != 8 && lanes != 16 && lanes != 32)) {
    set_error("subfv_ns_batch_set_node_kernel: lanes must be 0, 1, 8, 16 or 32");
    return -2;
  }
  if (b->P.node_group != lanes) {
    b->P.node_group = lanes;
    if (graph_drop(b, 0) || graph_drop(b, 1)) return -1;
  }
  return 0;
}

int subfv_ns_batch_advance(subfv_ns_batch* b, int n_steps) {
  if (!b || n_steps < 0) {
    set_error("subfv_ns_batch_advance: bad argument");
    return -2;
  }
  if (table_upload(b)) return -1;
  const int chunk = kGraphSteps;
  if (n_steps >= chunk) {
    if (graph_for(b)) return -1;
    for (int i = 0; i + chunk <= n_steps; i += chunk) SUBFV_CUDA(cudaGraphLaunch(b->graph[b->tab.tiles], b->stream));
  }
  for (int i = 0; i < n_steps % chunk; ++i) launch_ns_batch_step(b->tab, b->P, b->stream);
  SUBFV_CUDA(cudaGetLastError());
  return snapshot_enqueue(b);
}

int subfv_ns_batch_time_steps(subfv_ns_batch* b, int n_steps, double* ms) {
  if (!b || n_steps < 1 || !ms) {
    set_error("subfv_ns_batch_time_steps: bad argument");
    return -2;
  }
  if (table_upload(b)) return -1;
  cudaEvent_t e0, e1;
  SUBFV_CUDA(cudaEventCreate(&e0));
  SUBFV_CUDA(cudaEventCreate(&e1));
  SUBFV_CUDA(cudaEventRecord(e0, b->stream));
  if (subfv_ns_batch_advance(b, n_steps)) return -1;
  SUBFV_CUDA(cudaEventRecord(e1, b->stream));
  SUBFV_CUDA(cudaEventSynchronize(e1));
  float f = 0.f;
  SUBFV_CUDA(cudaEventElapsedTime(&f, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = f;
  return 0;
}

int subfv_ns_batch_poll(subfv_ns_batch* b, int wait) {
  if (!b) return -2;
  if (b->outstanding.empty()) {
    if (!wait) return b->have_last ? 0 : 1;
    if (snapshot_enqueue(b)) return -1;
  }
  Snapshot& s = b->snap[b->outstanding.front()];
  if (!wait) {
    cudaError_t e = cudaEventQuery(s.ev);
    if (e == cudaErrorNotReady) return 1;
    SUBFV_CUDA(e);
  } else {
    SUBFV_CUDA(cudaEventSynchronize(s.ev));
  }
  snapshot_take(b, s);
  return 0;
}

int subfv_ns_batch_sync(subfv_ns_batch* b) {
  if (!b) return -2;
  if (snapshot_enqueue(b)) return -1;
  while (!b->outstanding.empty())
    if (subfv_ns_batch_poll(b, 1)) return -1;
  return 0;
}

int subfv_ns_batch_slot_info(const subfv_ns_batch* b, int slot, double* t, int64_t* steps, int* done,
                             unsigned* status) {
  if (!b || slot < 0 || slot >= b->cap) return -2;
  const Slot& q = b->slots[slot];
  if (!q.live || b->last_seq < q.first_snap) {  // not yet seen by a completed snapshot
    if (t) *t = q.t0;
    if (steps) *steps = 0;
    if (done) *done = 0;
    if (status) *status = 0;
    return q.live ? 1 : -2;
  }
  const NsScalars& h = b->last_sc[slot];
  if (t) *t = h.t;
  if (steps) *steps = (int64_t)h.steps;
  if (done) *done = h.done;
  if (status) *status = b->last_status[slot];
  return 0;
}

int subfv_ns_batch_get_sol(subfv_ns_batch* b, int slot, double* sol) {
  if (!b || !sol || slot < 0 || slot >= b->cap || !b->slots[slot].live) {
    set_error("subfv_ns_batch_get_sol: bad slot");
    return -2;
  }
  Slot& q = b->slots[slot];
  const DevMesh& d = q.mesh->d;
  // A problem that a completed snapshot shows done is final: the step kernels no longer
  // write its state, so the copy need not wait for the chunks still queued. Otherwise
  // the copy is ordered after everything enqueued so far on the batch stream.
  if (!(b->last_seq >= q.first_snap && b->last_sc[slot].done)) {
    cudaEvent_t e;
    SUBFV_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    SUBFV_CUDA(cudaEventRecord(e, b->stream));
    SUBFV_CUDA(cudaStreamWaitEvent(d.stream, e, 0));
    cudaEventDestroy(e);
  }
  std::vector<double> rec(kRec * (size_t)d.ne);
  SUBFV_CUDA(cudaMemcpyAsync(rec.data(), q.U0, rec.size() * sizeof(double), cudaMemcpyDeviceToHost, d.stream));
  SUBFV_CUDA(cudaStreamSynchronize(d.stream));
  for (int c = 0; c < d.ne; ++c)
    for (int k = 0; k < 5; ++k) sol[5 * (size_t)c + k] = rec[kRec * (size_t)c + k];
  return 0;
}

int subfv_ns_batch_size(const subfv_ns_batch* b, int* n_live, int64_t* used_bytes) {
  if (!b) return -2;
  if (n_live) *n_live = (int)b->order.size();
  if (used_bytes) *used_bytes = b->used;
  return 0;
}

}  // extern "C"
