// Pair index: for every static edge (u, v) the run of its temporal edges
// {eid, t}, ascending in eid, plus an open-addressing hash table
// (u, v) -> (start, len).  It lets the search count a closing last motif
// edge by range arithmetic (the number of u->v edges with id after the
// previous edge and t <= t(e_0) + delta) instead of scanning a list.
//
// Built on the device from the packed graph.  The in-records are already in
// (target, edge id) order, so one stable radix sort of them by source gives
// (source, target, edge id) order: 21 key bits for 1.1M vertices, where a sort
// of the edges by the pair took 53 of a 64-bit key (7.8M edges: 3 passes of 8
// bytes per edge, 0.28 ms with the key kernel, against 7 passes of 12, 0.69 ms).
// Then the runs' first positions (CUB unique-by-key) and a parallel hash insert
// (atomicCAS on the 64-bit key).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>
#include <cub/iterator/counting_input_iterator.cuh>

#include "evx_internal.cuh"

namespace evx {
namespace {

// Sort input from the in-records: source as the key, edge id as the value.
__global__ void in_keys_kernel(const int4 *__restrict__ in_rec, unsigned *__restrict__ keys,
                               int *__restrict__ vals, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int4 r = in_rec[i];
    keys[i] = (unsigned)r.y;
    vals[i] = r.x;
  }
}

// Sort input by target from the edges, and by source from edges in an order.
__global__ void target_keys_kernel(const int4 *__restrict__ edges, unsigned *__restrict__ keys,
                                   int *__restrict__ vals, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    keys[i] = (unsigned)edges[i].y;
    vals[i] = i;
  }
}
__global__ void source_keys_kernel(const int4 *__restrict__ edges, const int *__restrict__ vals,
                                   unsigned *__restrict__ keys, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    keys[i] = (unsigned)edges[vals[i]].x;
}

// rec[i] = {eid, t} and the pair key of the i-th edge in pair order
__global__ void pair_rec_kernel(const int *__restrict__ eids, const int4 *__restrict__ edges,
                                int2 *__restrict__ rec, unsigned long long *__restrict__ keys, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int e = eids[i];
    const int4 ed = edges[e];
    rec[i] = make_int2(e, ed.z);
    keys[i] = pair_key(ed.x, ed.y);
  }
}

// pair_loc[e] = {position of e in pair_rec, end of its run}.  One thread per
// edge gallops to the end of its run, whatever the run's length (one thread per
// run, writing its entries in turn, took 0.58 ms on 7.8M edges, mostly for the
// few long runs; this takes 0.10 ms).
__global__ void pair_loc_kernel(const int *__restrict__ eids, const unsigned long long *__restrict__ keys,
                                int2 *__restrict__ loc, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned long long k = keys[i];
    int lo = i + 1, hi = n, step = 1;  // the end lies in [lo, hi]
    while (lo < hi) {
      const int q = min(lo + step - 1, hi - 1);
      if (keys[q] != k) { hi = q; break; }
      lo = q + 1;
      step <<= 1;
    }
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (keys[mid] != k) hi = mid; else lo = mid + 1;
    }
    loc[eids[i]] = make_int2(i, lo);
  }
}

// rev[e] for e = (u, v): the entries of the reverse pair's run (v, u) after
// e (edge id greater than e), as {first such position, end of the run};
// {0, 0} when there is no v -> u edge.  later[e]: bit 0, e's own run has a
// later entry; bit 1, the reverse run has one after e.  In edge order: pairs
// that are active at a time then meet in the table's cached slots (0.23 ms on
// 7.8M edges; in pair order, joined with the kernel above, 0.55 ms for both).
__global__ void rev_loc_kernel(const GraphView g, int2 *__restrict__ rev, unsigned char *__restrict__ later, int n) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int4 ed = g.edges[e];
    const int2 f = pair_find(g, ed.y, ed.x);
    int lo = f.x, hi = f.x + f.y;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (g.pair_rec[mid].x > e) hi = mid; else lo = mid + 1;
    }
    rev[e] = f.y > 0 ? make_int2(lo, f.x + f.y) : make_int2(0, 0);
    const int2 own = g.pair_loc[e];
    later[e] = (own.x + 1 < own.y ? 1 : 0) | (lo < f.x + f.y ? 2 : 0);
  }
}

// dir[r] = {v, start} of run r (runs sorted by (u, v)); dir[P] = sentinel;
// dir_off[u] = first run of source u or later, by binary search in the runs'
// keys (counting the runs per source with atomics and a scan took 0.38 ms on
// 7.8M edges, most of it on a few sources' counters; this takes 0.04 ms)
__global__ void pair_dir_kernel(const unsigned long long *__restrict__ ukeys,
                                const int *__restrict__ starts, const int *__restrict__ num_runs,
                                int2 *__restrict__ dir, int *__restrict__ dir_off, int nv, int n_edges) {
  const int P = *num_runs;
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, dt = gridDim.x * blockDim.x;
  for (int r = t0; r <= P; r += dt)
    dir[r] = r == P ? make_int2(0x7fffffff, n_edges) : make_int2((int)(unsigned)(ukeys[r] & 0xffffffffull), starts[r]);
  for (unsigned x = t0; x <= (unsigned)nv; x += dt) {
    const unsigned long long k = pair_key((int)x, 0);
    int lo = 0, hi = P;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (ukeys[mid] < k) lo = mid + 1; else hi = mid;
    }
    dir_off[x] = lo;
  }
}

// Cross-list starts: for e = (u, v), the first position of out(v) and of
// in(u) whose edge comes after e (the two endpoint lists e is not in), so
// a search that extends e from either endpoint starts without a binary
// search.  Taken in list order, where neighbouring threads search the same
// list for neighbouring ids (in edge order, each its own: 0.30 ms on 7.8M edges, against 0.20).
__global__ void cross_pos_kernel(const int4 *__restrict__ node_rng, const int4 *__restrict__ out_rec,
                                 const int4 *__restrict__ in_rec, const int *__restrict__ out_node,
                                 const int *__restrict__ in_node, int *__restrict__ cross_out,
                                 int *__restrict__ cross_in, int n) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    int e = in_rec[p].x, x = in_node[p];
    int lo = node_rng[x].x, hi = node_rng[x].y;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (out_rec[mid].x > e) hi = mid; else lo = mid + 1;
    }
    cross_out[e] = lo;
    e = out_rec[p].x;
    x = out_node[p];
    lo = node_rng[x].z; hi = node_rng[x].w;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (in_rec[mid].x > e) hi = mid; else lo = mid + 1;
    }
    cross_in[e] = lo;
  }
}

// Mark each adjacency record whose edge is followed by another entry of its
// pair run (top bit of the record's fourth word) and whose reverse pair has
// an entry after it (kRevLater).  One byte per edge is gathered, from an array
// that stays in L2 (the two 8-byte locations it was derived from here before
// took 0.27 ms on 7.8M edges; this takes 0.08 ms).
__global__ void mark_runs_kernel(int4 *__restrict__ out_rec, int4 *__restrict__ in_rec,
                                 const unsigned char *__restrict__ later, int n) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int fo = later[out_rec[p].x], fi = later[in_rec[p].x];
    if (fo) out_rec[p].w |= ((fo & 1) ? (int)0x80000000u : 0) | ((fo & 2) ? kRevLater : 0);
    if (fi) in_rec[p].w |= ((fi & 1) ? (int)0x80000000u : 0) | ((fi & 2) ? kRevLater : 0);
  }
}

__global__ void pair_clear_kernel(int4 *__restrict__ tab, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    tab[i] = make_int4(-1, -1, 0, 0);
}

// Insert every run; the probe sequence is bounded by the table size, and the
// longest probe actually used is recorded so lookups can stop there.
__global__ void pair_insert_kernel(const unsigned long long *__restrict__ ukeys,
                                   const int *__restrict__ starts, const int *__restrict__ num_runs,
                                   int4 *__restrict__ tab, unsigned long long mask,
                                   int *__restrict__ max_probe, int *__restrict__ overflow, int n_edges) {
  const int P = *num_runs;
  int longest = 0;  // this thread's longest probe; one atomicMax per warp at the end
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    const unsigned long long key = ukeys[p];
    const int start = starts[p], len = (p + 1 < P ? starts[p + 1] : n_edges) - start;
    unsigned long long h = pair_hash(key) & mask;
    bool done = false;
    for (unsigned long long i = 0; i <= mask; i++) {
      unsigned long long *slot = reinterpret_cast<unsigned long long *>(tab + h);
      const unsigned long long prev = atomicCAS(slot, ~0ull, key);
      if (prev == ~0ull) {
        tab[h].z = start;
        tab[h].w = len;
        longest = max(longest, (int)i + 1);
        done = true;
        break;
      }
      h = (h + 1) & mask;
    }
    if (!done) atomicExch(overflow, 1);
  }
  longest = __reduce_max_sync(0xffffffffu, (unsigned)longest);
  if ((threadIdx.x & 31) == 0 && longest > 0) atomicMax(max_probe, longest);
}

}  // namespace

int build_pair_index(DeviceGraph &g, const ListScratch &lists, bool in_grouped, cudaStream_t s) {
  const int64_t E = g.num_edges;
  if (E <= 0) {
    g.pair_mask = 0;
    g.pair_max_probe = 0;
    EVX_CUDA(dev_alloc((void **)&g.pair_tab, sizeof(int4), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.pair_rec, sizeof(int2), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.pair_loc, sizeof(int2), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.rev_loc, sizeof(int2), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.cross_out, sizeof(int), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.cross_in, sizeof(int), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.pair_dir, sizeof(int2), g.device, s));
    EVX_CUDA(dev_alloc((void **)&g.dir_off, sizeof(int) * (size_t)(g.num_vertices + 1), g.device, s));
    EVX_CUDA(cudaMemsetAsync(g.pair_tab, 0xff, sizeof(int4), s));
    EVX_CUDA(cudaMemsetAsync(g.dir_off, 0, sizeof(int) * (size_t)(g.num_vertices + 1), s));
    {
      const int2 sentinel = make_int2(0x7fffffff, 0);
      EVX_CUDA(cudaMemcpyAsync(g.pair_dir, &sentinel, sizeof(int2), cudaMemcpyHostToDevice, s));
      EVX_CUDA(cudaStreamSynchronize(s));
    }
    g.bytes += sizeof(int4) + 5 * sizeof(int2) + sizeof(int) * (g.num_vertices + 1);
    return EVX_OK;
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g.device);
  const int grid = sms * 8, block = 256;
  const int n = (int)E;
  unsigned *keys = nullptr;                    // [2n] sort keys, double-buffered
  int *vals = nullptr;                         // [2n] edge ids
  unsigned long long *pkeys = nullptr, *ukeys = nullptr;
  int *starts = nullptr, *ctr = nullptr;
  const int *order = nullptr;                  // edge ids in pair order
  unsigned char *later = nullptr;
  void *tmp = nullptr;
  size_t tmp_bytes = 0, t1 = 0, t2 = 0;
  int rc = EVX_OK;
  auto A = [&](void **p, size_t b) {
    if (rc == EVX_OK) {
      cudaError_t e = dev_alloc(p, b, g.device, s);
      if (e != cudaSuccess) rc = cuda_fail(e, "cudaMallocAsync(pair index scratch)");
    }
  };
  const cub::CountingInputIterator<int> positions(0);
  A((void **)&keys, sizeof(unsigned) * 2 * n);
  A((void **)&vals, sizeof(int) * 2 * n);
  A((void **)&pkeys, sizeof(unsigned long long) * n);
  A((void **)&ukeys, sizeof(unsigned long long) * n);
  A((void **)&starts, sizeof(int) * n);
  A((void **)&later, (size_t)n);
  A((void **)&ctr, sizeof(int) * 4);  // [0] runs, [1] max probe, [2] overflow
  if (!rc) {
    cudaError_t e = dev_alloc((void **)&g.pair_rec, sizeof(int2) * (size_t)n, g.device, s);
    if (e == cudaSuccess) e = dev_alloc((void **)&g.pair_loc, sizeof(int2) * (size_t)n, g.device, s);
    if (e != cudaSuccess) rc = cuda_fail(e, "cudaMalloc(pair index)");
  }
  if (rc) goto cleanup;
  {
    // key bits actually used: vertex ids < V
    int vb = 1;
    while ((1ll << vb) < g.num_vertices + 1 && vb < 31) vb++;
    cub::DoubleBuffer<unsigned> dk(keys, keys + n);
    cub::DoubleBuffer<int> dv(vals, vals + n);
    cub::DeviceRadixSort::SortPairs(nullptr, t1, dk, dv, n, 0, vb, s);
    cub::DeviceSelect::UniqueByKey(nullptr, t2, pkeys, positions, ukeys, starts, ctr, n, s);
    tmp_bytes = t1 > t2 ? t1 : t2;
    A(&tmp, tmp_bytes);
    if (rc) goto cleanup;
    if (in_grouped) {
      in_keys_kernel<<<grid, block, 0, s>>>(g.in_rec, keys, vals, n);
    } else {
      // in-lists that are not in (target, edge id) order: from the edges
      target_keys_kernel<<<grid, block, 0, s>>>(g.edges, keys, vals, n);
      cub::DeviceRadixSort::SortPairs(tmp, t1, dk, dv, n, 0, vb, s);
      source_keys_kernel<<<grid, block, 0, s>>>(g.edges, dv.Current(), dk.Current(), n);
    }
    cub::DeviceRadixSort::SortPairs(tmp, t1, dk, dv, n, 0, vb, s);
    order = dv.Current();
    pair_rec_kernel<<<grid, block, 0, s>>>(order, g.edges, g.pair_rec, pkeys, n);
    cub::DeviceSelect::UniqueByKey(tmp, t2, pkeys, positions, ukeys, starts, ctr, n, s);
    pair_loc_kernel<<<grid, block, 0, s>>>(order, pkeys, g.pair_loc, n);
  }
  {
    int runs = 0;
    EVX_CUDA(cudaMemcpyAsync(&runs, ctr, sizeof(int), cudaMemcpyDeviceToHost, s));
    EVX_CUDA(cudaStreamSynchronize(s));
    long long cap = 1;
    while (cap < 2ll * runs + 2) cap <<= 1;
    g.pair_mask = (unsigned long long)(cap - 1);
    cudaError_t e = dev_alloc((void **)&g.pair_tab, sizeof(int4) * (size_t)cap, g.device, s);
    if (e == cudaSuccess) e = dev_alloc((void **)&g.rev_loc, sizeof(int2) * (size_t)n, g.device, s);
    if (e == cudaSuccess) e = dev_alloc((void **)&g.cross_out, sizeof(int) * (size_t)n, g.device, s);
    if (e == cudaSuccess) e = dev_alloc((void **)&g.cross_in, sizeof(int) * (size_t)n, g.device, s);
    if (e != cudaSuccess) { rc = cuda_fail(e, "cudaMalloc(pair index)"); goto cleanup; }
    g.bytes += (int64_t)(sizeof(int4) * cap + 4 * sizeof(int2) * n);
    EVX_CUDA(cudaMemsetAsync(ctr + 1, 0, 2 * sizeof(int), s));
    pair_clear_kernel<<<grid, block, 0, s>>>(g.pair_tab, cap);
    pair_insert_kernel<<<grid, block, 0, s>>>(ukeys, starts, ctr, g.pair_tab, g.pair_mask, ctr + 1, ctr + 2, n);
    // per-node directory of distinct out-neighbours (sorted) -> pair runs
    {
      const int64_t V = g.num_vertices;
      cudaError_t e2 = dev_alloc((void **)&g.pair_dir, sizeof(int2) * ((size_t)runs + 1), g.device, s);
      if (e2 == cudaSuccess) e2 = dev_alloc((void **)&g.dir_off, sizeof(int) * (size_t)(V + 1), g.device, s);
      if (e2 != cudaSuccess) { rc = cuda_fail(e2, "cudaMalloc(pair directory)"); goto cleanup; }
      g.bytes += (int64_t)(sizeof(int2) * ((size_t)runs + 1) + sizeof(int) * (V + 1));
      pair_dir_kernel<<<grid, block, 0, s>>>(ukeys, starts, ctr, g.pair_dir, g.dir_off, (int)V, n);
    }
    int h[2] = {0, 0};
    EVX_CUDA(cudaGetLastError());
    EVX_CUDA(cudaMemcpyAsync(h, ctr + 1, sizeof(h), cudaMemcpyDeviceToHost, s));
    EVX_CUDA(cudaStreamSynchronize(s));
    if (h[1]) { rc = fail(EVX_ERR_CUDA, "pair index insert overflow"); goto cleanup; }
    g.pair_max_probe = h[0];
    rev_loc_kernel<<<grid, block, 0, s>>>(g.view(), g.rev_loc, later, n);
    cross_pos_kernel<<<grid, block, 0, s>>>(g.node_rng, g.out_rec, g.in_rec, lists.out_node, lists.in_node,
                                            g.cross_out, g.cross_in, n);
    mark_runs_kernel<<<grid, block, 0, s>>>(g.out_rec, g.in_rec, later, n);
    EVX_CUDA(cudaGetLastError());
  }
cleanup:
  dev_free(keys, s);
  dev_free(vals, s);
  dev_free(pkeys, s);
  dev_free(ukeys, s);
  dev_free(starts, s);
  dev_free(later, s);
  dev_free(ctr, s);
  dev_free(tmp, s);
  if (rc == EVX_OK) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) rc = cuda_fail(e, "pair index build");
  }
  return rc;
}

}  // namespace evx
