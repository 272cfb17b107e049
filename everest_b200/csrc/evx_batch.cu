// Batched queries: many count queries against one resident graph in one
// persistent launch per kind of motif (include/everest_b200.h, evx_batch_*).
//
// The queries are ordered by motif size and by how their last edge is counted;
// each such group forms one device work queue: the root ranges are cut into
// tiles of at most tile_roots roots laid end to end, warps claim tiles with one
// atomicAdd and switch their per-warp query copy when a tile belongs to another
// query, so cheap and expensive queries share the GPU without per-query tails
// or per-query launches.  Each group runs the kernel compiled for exactly that
// size and way (64 mixed queries over 250k-root windows: 20.8 ms, against 23.1
// with one kernel per size).  The launch sequence (query table upload, counter
// reset, the kernels, counts read-back) is captured once into a CUDA graph and
// replayed while the batch keeps the same shape.
//
// The groups' kernels run side by side, the largest motifs first, and a group's
// queries start with the widest time windows: a launch ends with a few warps on
// its heaviest roots, whose SMs the next group's blocks then fill, and the
// heaviest roots start early (the same 64 queries, one size after the other and
// in the given order: 30.0 ms; side by side, widest first: 23.4 ms; 64 requests
// over windows of 1000 roots: 0.61 -> 0.45 ms).  A batch that the caller gave a
// number of blocks per SM runs one launch after the other, one per motif size,
// and so never holds more.
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "evx_internal.cuh"
#include "evx_sides.h"

using namespace evx;

namespace {
constexpr int kSizes = EVX_MAX_MOTIF_EDGES - 1;  // motif sizes

struct CudaApi {
  using Error = cudaError_t;
  using Stream = cudaStream_t;
  using Event = cudaEvent_t;
  static constexpr Error kOk = cudaSuccess;
  static Error create(Stream *s, int priority) {
    return cudaStreamCreateWithPriority(s, cudaStreamNonBlocking, priority);
  }
  static Error priority(Stream s, int *p) { return cudaStreamGetPriority(s, p); }
  static Error destroy(Stream s) { return cudaStreamDestroy(s); }
  static Error synchronize(Stream s) { return cudaStreamSynchronize(s); }
  static Error create_event(Event *e) { return cudaEventCreateWithFlags(e, cudaEventDisableTiming); }
  static Error destroy_event(Event e) { return cudaEventDestroy(e); }
  static Error record(Event e, Stream s) { return cudaEventRecord(e, s); }
  static Error wait(Stream s, Event e) { return cudaStreamWaitEvent(s, e, 0); }
};
SparePool<CudaApi> g_spare;
}  // namespace

struct evx_batch {
  int device = 0;
  int max_q = 0;
  int num_sms = 148;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  const evx_graph *graph = nullptr;
  std::vector<QueryDesc> queries;
  QueryDesc *table_d = nullptr;        // [max_q]
  QueryDesc *table_h = nullptr;        // pinned [max_q]
  unsigned long long *counts_d = nullptr;  // [max_q] counts, kCursors cursor words, [max_q] work meters
  unsigned long long *counts_h = nullptr;  // pinned [max_q] counts, [max_q] meters
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  Sides<CudaApi> sides;  // streams beside it
  // tuning
  int tile_roots = 256, blocks_per_sm = 0, steal_interval = 16, min_split = 2, use_graph = 1;
  unsigned long long limit = 0;  // work limit per query (0 = none)
  // table order -> query index, and the motif-size groups of the table
  // (kGroupWords ints each)
  std::vector<int> order;
  std::vector<int> groups;
  // captured launch and the shape it was captured for
  cudaGraphExec_t exec = nullptr;
  std::vector<int> exec_groups;
  int exec_nq = -1, exec_tile_roots = -1;
  unsigned long long exec_limit = 0;
  const evx_graph *exec_graph = nullptr;
  bool launched = false;
  int last_launches = 0;
  float last_ms = 0.f;
};

namespace {

// one work-queue cursor word per launch: motif sizes x ways of counting the
// last edge (five, with and without strict timestamps, and the kernel that
// holds all)
constexpr int kCursors = kSizes * 11;
// a launch's group of the table: {k, first table position, queries, tiles,
// grid, pair-run walk (0/1), roots per tile, way of counting the last edge}
constexpr int kGroupWords = 8;

void drop_exec(evx_batch *b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  b->exec = nullptr;
  b->exec_nq = -1;
}

int side_streams(const evx_batch *b) { return b->blocks_per_sm > 0 ? 0 : kSides; }

int enqueue(evx_batch *b, int nq) {
  unsigned long long *meter = b->counts_d + b->max_q + kCursors;
  EVX_CUDA(cudaMemcpyAsync(b->table_d, b->table_h, sizeof(QueryDesc) * (size_t)nq, cudaMemcpyHostToDevice,
                           b->stream));
  EVX_CUDA(cudaMemsetAsync(b->counts_d, 0, sizeof(unsigned long long) * (2 * (size_t)b->max_q + kCursors),
                           b->stream));
  int rc = EVX_OK;
  cudaError_t e = b->sides.run(b->stream, (int)(b->groups.size() / kGroupWords), side_streams(b), [&](int gi, cudaStream_t s) {
    const int *gr = &b->groups[(size_t)gi * kGroupWords];
    const int k = gr[0], beg = gr[1], tiles = gr[3], grid = gr[4];
    if (tiles <= 0) return cudaSuccess;
    LaunchArgs la{};
    la.table = b->table_d + beg;
    la.nq = gr[2];
    la.total_tiles = tiles;
    la.tile_roots = gr[6];
    la.cursor = reinterpret_cast<int *>(b->counts_d + b->max_q + gi);
    la.counts = b->counts_d + beg;
    la.limit = b->limit;
    la.meter = meter + beg;
    rc = launch_table(b->graph->g.view(), b->table_h[beg], la, k, gr[7], gr[5] != 0, grid, s);
    const cudaError_t le = cudaGetLastError();
    return rc && le == cudaSuccess ? cudaErrorLaunchFailure : le;
  });
  if (rc) return rc;
  if (e != cudaSuccess) return cuda_fail(e, "batch search launch");
  EVX_CUDA(cudaMemcpyAsync(b->counts_h, b->counts_d, sizeof(unsigned long long) * (size_t)nq,
                           cudaMemcpyDeviceToHost, b->stream));
  if (b->limit)
    EVX_CUDA(cudaMemcpyAsync(b->counts_h + b->max_q, meter, sizeof(unsigned long long) * (size_t)nq,
                             cudaMemcpyDeviceToHost, b->stream));
  return EVX_OK;
}

}  // namespace

extern "C" {

int evx_batch_create(int device, int max_queries, void *stream, evx_batch **out) {
  if (!out) return fail(EVX_ERR_INVALID, "null output pointer");
  if (max_queries < 1 || max_queries > (1 << 20)) return fail(EVX_ERR_INVALID, "max_queries out of range");
  int ndev = 0;
  evx_device_count(&ndev);
  if (ndev == 0) return fail(EVX_ERR_NODEVICE, "no CUDA device");
  if (device < 0 || device >= ndev) return fail(EVX_ERR_INVALID, "bad device index");
  EVX_CUDA(cudaSetDevice(device));
  evx_batch *b = new (std::nothrow) evx_batch();
  if (!b) return fail(EVX_ERR_NOMEM, "host allocation failed");
  b->device = device;
  b->max_q = max_queries;
  cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, device);
  cudaError_t e = cudaSuccess;
  if (stream) {
    b->stream = (cudaStream_t)stream;
  } else {
    e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    b->own_stream = true;
  }
  if (e == cudaSuccess) e = cudaMalloc(&b->table_d, sizeof(QueryDesc) * (size_t)max_queries);
  if (e == cudaSuccess) e = cudaMallocHost(&b->table_h, sizeof(QueryDesc) * (size_t)max_queries);
  if (e == cudaSuccess) e = cudaMalloc(&b->counts_d, sizeof(unsigned long long) * (2 * (size_t)max_queries + kCursors));
  if (e == cudaSuccess) e = cudaMallocHost(&b->counts_h, sizeof(unsigned long long) * 2 * (size_t)max_queries);
  if (e == cudaSuccess) e = cudaEventCreate(&b->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&b->ev1);
  if (e != cudaSuccess) {
    evx_batch_destroy(b);
    return cuda_fail(e, "batch setup");
  }
  b->queries.reserve((size_t)max_queries);
  *out = b;
  return EVX_OK;
}

int evx_batch_destroy(evx_batch *b) {
  if (!b) return EVX_OK;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  drop_exec(b);
  b->sides.drop(g_spare, b->device);
  cudaFree(b->table_d);
  cudaFree(b->counts_d);
  if (b->table_h) cudaFreeHost(b->table_h);
  if (b->counts_h) cudaFreeHost(b->counts_h);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return EVX_OK;
}

int evx_batch_clear(evx_batch *b) {
  if (!b) return fail(EVX_ERR_INVALID, "null batch");
  if (b->launched) return fail(EVX_ERR_STATE, "batch launched: read its result first");
  b->queries.clear();
  b->graph = nullptr;
  return EVX_OK;
}

int evx_batch_set_tuning(evx_batch *b, int tile_roots, int blocks_per_sm, int steal_interval, int min_split,
                         int use_graph, int reserved) {
  (void)reserved;
  if (!b) return fail(EVX_ERR_INVALID, "null batch");
  if (tile_roots < 32 || tile_roots % 32 || tile_roots > (1 << 20))
    return fail(EVX_ERR_INVALID, "tile_roots must be a multiple of 32 in [32, 2^20]");
  if (blocks_per_sm < 0 || steal_interval < 0 || (steal_interval & (steal_interval - 1)) || min_split < 2)
    return fail(EVX_ERR_INVALID, "bad tuning value");
  b->tile_roots = tile_roots;
  b->blocks_per_sm = blocks_per_sm;
  b->steal_interval = steal_interval;
  b->min_split = min_split;
  b->use_graph = use_graph ? 1 : 0;
  drop_exec(b);
  return EVX_OK;
}

int evx_batch_set_limit(evx_batch *b, uint64_t max_work) {
  if (!b) return fail(EVX_ERR_INVALID, "null batch");
  if (b->launched) return fail(EVX_ERR_STATE, "batch launched: read its result first");
  b->limit = max_work;
  return EVX_OK;
}

int evx_batch_add(evx_batch *b, const evx_graph *gh, int k, const int *mu, const int *mv, int delta, int64_t beg,
                  int64_t end, unsigned flags, int *index_out) {
  if (!b || !gh || !mu || !mv) return fail(EVX_ERR_INVALID, "null argument");
  if (b->launched) return fail(EVX_ERR_STATE, "batch launched: read its result first");
  if ((int)b->queries.size() >= b->max_q) return fail(EVX_ERR_INVALID, "batch is full");
  if (b->graph && b->graph != gh) return fail(EVX_ERR_INVALID, "all queries of a batch use one graph");
  if (gh->g.device != b->device) return fail(EVX_ERR_INVALID, "graph and batch on different devices");
  MotifPlan plan;
  int rc = build_plan(k, mu, mv, &plan);
  if (rc) return rc;
  const DeviceGraph &g = gh->g;
  if (delta < 0) return fail(EVX_ERR_INVALID, "delta must be non-negative");
  if ((int64_t)g.max_t + (int64_t)delta > (int64_t)INT_MAX)
    return fail(EVX_ERR_OVERFLOW, "t + delta overflows int32");
  const int64_t E = g.num_edges;
  if (end < 0) end = E - k + 1;
  if (end > E) end = E;
  if (beg < 0) beg = 0;
  if (end < beg) end = beg;
  QueryDesc q;
  std::memset(&q, 0, sizeof(q));
  q.plan = plan;
  q.root_beg = (int)beg;
  q.root_end = (int)end;
  q.delta = delta;
  q.flags = ((flags & EVX_FLAG_STRICT_TS) ? kQStrict : 0) | tail_mode(plan, flags, false);
  q.steal_interval = (flags & EVX_FLAG_NO_STEAL) ? 0 : b->steal_interval;
  q.min_split = b->min_split;
  b->graph = gh;
  b->queries.push_back(q);
  if (index_out) *index_out = (int)b->queries.size() - 1;
  return EVX_OK;
}

int evx_batch_launch(evx_batch *b) {
  if (!b) return fail(EVX_ERR_INVALID, "null batch");
  if (b->launched) return fail(EVX_ERR_STATE, "batch already launched");
  const int nq = (int)b->queries.size();
  if (nq == 0) return fail(EVX_ERR_STATE, "empty batch");
  EVX_CUDA(cudaSetDevice(b->device));
  // table order: the largest motifs first, and of one launch the widest
  // windows; one group (and one launch) per size and way of counting the last
  // edge
  // (a batch with a bound on its blocks runs its launches one after the other,
  // so it has one per size: 64 requests over windows of 1000 roots, 4 blocks
  // per SM, 0.96 ms with one per way and 0.78 with one per size)
  const bool one = !side_streams(b);
  long long size_roots[EVX_MAX_MOTIF_EDGES + 1] = {};
  for (const QueryDesc &q : b->queries) size_roots[q.plan.k] += q.root_end - q.root_beg;
  const auto tail = [&](const QueryDesc &q) {
    return one ? kTailAny : tail_of(q.plan.k, q.flags, size_roots[q.plan.k]);
  };
  b->order.resize(nq);
  for (int i = 0; i < nq; i++) b->order[i] = i;
  std::stable_sort(b->order.begin(), b->order.end(), [&](int x, int y) {
    const QueryDesc &p = b->queries[x], &q = b->queries[y];
    if (p.plan.k != q.plan.k) return p.plan.k > q.plan.k;
    const int tp = tail(p), tq = tail(q);
    return tp != tq ? tp < tq : p.delta > q.delta;
  });
  b->groups.clear();
  int launches = 0;
  for (int pos = 0; pos < nq;) {
    const int k = b->queries[b->order[pos]].plan.k, way = tail(b->queries[b->order[pos]]);
    const int beg = pos;
    long long roots = 0;
    bool ps = false;
    for (; pos < nq && b->queries[b->order[pos]].plan.k == k && tail(b->queries[b->order[pos]]) == way; pos++) {
      const QueryDesc &q = b->queries[b->order[pos]];
      ps = ps || plan_pair_scan(q.plan, q.flags, false);
      roots += std::max(0, q.root_end - q.root_beg);
    }
    int bps = 0;
    int rc = table_occupancy(k, way, ps, &bps);  // also sets the kernel attributes before any capture
    if (rc) return rc;
    if (b->blocks_per_sm > 0) bps = b->blocks_per_sm;
    if (bps < 1) bps = 1;
    const long long warps = (long long)bps * b->num_sms * (kSearchBlock / 32);
    const int tile_roots = tile_roots_for(k, roots, pos - beg, warps, b->tile_roots);
    if (tile_roots == 0) return fail(EVX_ERR_OVERFLOW, "root tiles would overflow int32");
    int tiles = 0;
    for (int i = beg; i < pos; i++) {
      QueryDesc q = b->queries[b->order[i]];
      if (!b->limit) q.flags = bound_rule(q.plan, q.flags);
      q.tile_beg = tiles;
      tiles += (int)tiles_of(q.root_end - q.root_beg, tile_roots);
      b->table_h[i] = q;
    }
    b->groups.insert(b->groups.end(), {k, beg, pos - beg, tiles, bps * b->num_sms, ps ? 1 : 0, tile_roots, way});
    launches += tiles > 0 ? 1 : 0;
  }
  EVX_CUDA(b->sides.ready(g_spare, b->device, b->stream, (int)b->groups.size() / kGroupWords, side_streams(b)));
  EVX_CUDA(cudaEventRecord(b->ev0, b->stream));
  if (b->use_graph) {
    if (!b->exec || b->exec_nq != nq || b->exec_groups != b->groups || b->exec_tile_roots != b->tile_roots ||
        b->exec_graph != b->graph || b->exec_limit != b->limit) {
      drop_exec(b);
      cudaGraph_t graph = nullptr;
      EVX_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
      int rc = enqueue(b, nq);
      cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
      if (rc) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
      }
      if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
      e = cudaGraphInstantiate(&b->exec, graph, 0);
      cudaGraphDestroy(graph);
      if (e != cudaSuccess) { b->exec = nullptr; return cuda_fail(e, "cudaGraphInstantiate"); }
      b->exec_nq = nq; b->exec_groups = b->groups;
      b->exec_tile_roots = b->tile_roots; b->exec_graph = b->graph; b->exec_limit = b->limit;
    }
    EVX_CUDA(cudaGraphLaunch(b->exec, b->stream));
  } else {
    int rc = enqueue(b, nq);
    if (rc) return rc;
  }
  EVX_CUDA(cudaEventRecord(b->ev1, b->stream));
  b->last_launches = launches;
  b->launched = true;
  return EVX_OK;
}

int evx_batch_result(evx_batch *b, uint64_t *counts, int n) {
  if (!b) return fail(EVX_ERR_INVALID, "null batch");
  if (!b->launched) return fail(EVX_ERR_STATE, "result before launch");
  EVX_CUDA(cudaSetDevice(b->device));
  EVX_CUDA(cudaStreamSynchronize(b->stream));
  float ms = 0.f;
  if (cudaEventElapsedTime(&ms, b->ev0, b->ev1) == cudaSuccess) b->last_ms = ms;
  b->launched = false;
  const int nq = (int)b->queries.size();
  if (counts) {
    for (int pos = 0; pos < nq; pos++) {
      const int i = b->order[pos];
      if (i < n)
        counts[i] = (b->limit && b->counts_h[b->max_q + pos] > b->limit) ? UINT64_MAX : b->counts_h[pos];
    }
  }
  return EVX_OK;
}

int evx_batch_query(evx_batch *b, int *done) {
  if (!b || !done) return fail(EVX_ERR_INVALID, "null argument");
  if (!b->launched) return fail(EVX_ERR_STATE, "query before launch");
  cudaError_t e = cudaEventQuery(b->ev1);
  if (e == cudaErrorNotReady) { *done = 0; return EVX_OK; }
  if (e != cudaSuccess) return cuda_fail(e, "cudaEventQuery");
  *done = 1;
  return EVX_OK;
}

int evx_batch_run(evx_batch *b, uint64_t *counts, int n) {
  int rc = evx_batch_launch(b);
  if (rc) return rc;
  return evx_batch_result(b, counts, n);
}

int evx_batch_last_stats(evx_batch *b, int *kernel_launches, float *device_ms) {
  if (!b) return fail(EVX_ERR_INVALID, "null batch");
  if (kernel_launches) *kernel_launches = b->last_launches;
  if (device_ms) *device_ms = b->last_ms;
  return EVX_OK;
}

}  // extern "C"
