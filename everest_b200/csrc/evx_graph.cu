// Device graph: upload of the host graph arrays and on-device packing into
// the 16-byte record layout the search kernels read.
//
// Host-format inputs are the reference's HostGraphData arrays
// (include/data.h:174-186): Eg (AoS {u,v,t}), outEdgesV / inEdgesV (edge ids
// grouped by endpoint, ascending), outEdgesR / inEdgesR (CSR offsets) and
// Euid.  The upload moves exactly those bytes (24 E + 8 (V+1), as
// calcTotalBytes, src/core/gpu/data.cu:22-24) and expands them on the device
// into the layout described in evx_internal.cuh (16-byte adjacency records
// carrying each edge's position in its other list, per-node int4 ranges).
#include <climits>

#include "evx_internal.cuh"

namespace evx {
namespace {

// positions: outpos[out_v[p]] = p, inpos[in_v[p]] = p (-1 before)
__global__ void scatter_pos_kernel(const int *__restrict__ out_v, const int *__restrict__ in_v,
                                   int *__restrict__ outpos, int *__restrict__ inpos, int n) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    outpos[out_v[p]] = p;
    inpos[in_v[p]] = p;
  }
}

// The packed edges.  *lost is set when a list does not hold every edge (each
// has E entries, so one is then named twice): the arrays that the lists fill
// edge by edge would keep gaps, which a search would take for list positions.
__global__ void pack_edges_kernel(const int *__restrict__ eg, const int *__restrict__ euid_in,
                                  const int *__restrict__ outpos, const int *__restrict__ inpos,
                                  int4 *__restrict__ edges, int *__restrict__ euid, int *lost, int n) {
  bool bad = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int at = outpos[i];
    const int *e = eg + 3ll * i;
    edges[i] = make_int4(e[0], e[1], e[2], at);
    euid[i] = euid_in ? euid_in[i] : i;
    bad |= at < 0 || inpos[i] < 0;
  }
  if (bad) *lost = 1;
}

// Neighbour signatures: one bit per neighbour (sig_bit) in the node's word.
// Neighbouring threads of a list belong to the same node, so a warp joins their
// bits first: one atomic per node in the warp (one per edge took 0.46 ms on 7.8M
// edges).
__device__ __forceinline__ void join_sig(unsigned long long *sig, int node, int bit) {
  const unsigned same = __match_any_sync(__activemask(), node);
  const unsigned long long b = 1ull << bit;
  const unsigned lo = __reduce_or_sync(same, (unsigned)b), hi = __reduce_or_sync(same, (unsigned)(b >> 32));
  if ((threadIdx.x & 31) == __ffs(same) - 1) atomicOr(sig + node, ((unsigned long long)hi << 32) | lo);
}

// The adjacency records, each list position's node, and the signatures; stray
// is set when the in-lists are not grouped by target with ascending ids.
__global__ void pack_rec_kernel(const int *__restrict__ out_v, const int *__restrict__ in_v,
                                const int4 *__restrict__ edges, const int *__restrict__ inpos,
                                const int4 *__restrict__ node_rng, int4 *__restrict__ out_rec,
                                int4 *__restrict__ in_rec, unsigned long long *__restrict__ sig_out,
                                unsigned long long *__restrict__ sig_in, ListScratch lists, int n) {
  bool bad = false;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int eo = out_v[p], ei = in_v[p];
    const int4 a = edges[eo], b = edges[ei];
    out_rec[p] = make_int4(eo, a.y, a.z, inpos[eo]);
    in_rec[p] = make_int4(ei, b.x, b.z, b.w);
    lists.out_node[p] = a.x;
    lists.in_node[p] = b.y;
    const int4 rg = node_rng[b.y];
    bad |= p < rg.z || p >= rg.w || (p > rg.z && in_v[p - 1] >= ei);
    join_sig(sig_out, a.x, sig_bit(a.y));
    join_sig(sig_in, b.y, sig_bit(b.x));
  }
  if (bad) *lists.stray = 1;
}

__global__ void pack_nodes_kernel(const int *__restrict__ out_r, const int *__restrict__ in_r,
                                  int4 *__restrict__ node_rng, int nv) {
  for (unsigned x = blockIdx.x * blockDim.x + threadIdx.x; x < (unsigned)nv; x += gridDim.x * blockDim.x) {
    node_rng[x] = make_int4(out_r[x], out_r[x + 1], in_r[x], in_r[x + 1]);
  }
}

// Input checks: edge ids in [0, E), vertex ids in [0, V), timestamps sorted,
// CSR offsets monotone from 0 to E.  Bits of *err name the failed check.  The
// list positions start at -1 here too (two fills of their own took 5 us of a
// small graph's load).
__global__ void validate_kernel(const int *__restrict__ eg, const int *__restrict__ out_v,
                                const int *__restrict__ in_v, const int *__restrict__ out_r,
                                const int *__restrict__ in_r, int *__restrict__ outpos, int *__restrict__ inpos,
                                int E, int V, int *err) {
  const int n = max(E, V + 1);
  int bad = 0;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)n; i += gridDim.x * blockDim.x) {
    if (i < (unsigned)E) {
      const int *e = eg + 3ll * i;
      outpos[i] = inpos[i] = -1;
      if ((unsigned)out_v[i] >= (unsigned)E || (unsigned)in_v[i] >= (unsigned)E) bad |= 1;
      if ((unsigned)e[0] >= (unsigned)V || (unsigned)e[1] >= (unsigned)V) bad |= 2;
      if (i > 0 && e[2] < e[-1]) bad |= 4;
    }
    if (i < (unsigned)V && (out_r[i + 1] < out_r[i] || in_r[i + 1] < in_r[i])) bad |= 8;
    if (i == 0 && (out_r[0] != 0 || in_r[0] != 0 || out_r[V] != E || in_r[V] != E)) bad |= 16;
  }
  if (bad) atomicOr(err, bad);
}

// min / max timestamp (for the t + delta overflow check)
__global__ void t_range_kernel(const int4 *__restrict__ edges, int n, int *out) {
  int lo = INT_MAX, hi = INT_MIN;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int t = edges[i].z;
    lo = min(lo, t);
    hi = max(hi, t);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_down_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_down_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(out, lo);
    atomicMax(out + 1, hi);
  }
}

__global__ void t_range_init_kernel(int *out) {
  out[0] = INT_MAX;
  out[1] = INT_MIN;
}

}  // namespace

int pack_graph(DeviceGraph &g, const int *eg_d, const int *out_v_d, const int *in_v_d,
               const int *out_r_d, const int *in_r_d, const int *euid_d, const ListScratch &lists, cudaStream_t s) {
  const int64_t E = g.num_edges, V = g.num_vertices;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g.device);
  const int grid = sms * 8, block = 256;
  EVX_CUDA(cudaMemsetAsync(g.sig_out, 0, sizeof(unsigned long long) * (size_t)(V > 0 ? V : 1), s));
  EVX_CUDA(cudaMemsetAsync(g.sig_in, 0, sizeof(unsigned long long) * (size_t)(V > 0 ? V : 1), s));
  if (V > 0) pack_nodes_kernel<<<grid, block, 0, s>>>(out_r_d, in_r_d, g.node_rng, (int)V);
  if (E > 0) {
    scatter_pos_kernel<<<grid, block, 0, s>>>(out_v_d, in_v_d, lists.outpos, g.inpos, (int)E);
    pack_edges_kernel<<<grid, block, 0, s>>>(eg_d, euid_d, lists.outpos, g.inpos, g.edges, g.euid, lists.lost, (int)E);
    pack_rec_kernel<<<grid, block, 0, s>>>(out_v_d, in_v_d, g.edges, g.inpos, g.node_rng, g.out_rec,
                                           g.in_rec, g.sig_out, g.sig_in, lists, (int)E);
  }
  EVX_CUDA(cudaGetLastError());
  return EVX_OK;
}

int validate_graph(const DeviceGraph &g, const int *eg_d, const int *out_v_d, const int *in_v_d,
                   const int *out_r_d, const int *in_r_d, const ListScratch &lists, cudaStream_t s) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g.device);
  validate_kernel<<<sms * 8, 256, 0, s>>>(eg_d, out_v_d, in_v_d, out_r_d, in_r_d, lists.outpos, g.inpos,
                                          (int)g.num_edges, (int)g.num_vertices, lists.err);
  int h = 0;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, lists.err, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "graph validation");
  if (h & 1) return fail(EVX_ERR_INVALID, "edge id out of range in out/in lists");
  if (h & 2) return fail(EVX_ERR_INVALID, "vertex id out of range in Eg");
  if (h & 4) return fail(EVX_ERR_INVALID, "edges are not sorted by timestamp");
  if (h & 8) return fail(EVX_ERR_INVALID, "CSR offsets are not monotone");
  if (h & 16) return fail(EVX_ERR_INVALID, "CSR offsets must start at 0 and end at num_edges");
  return EVX_OK;
}

int graph_t_range(DeviceGraph &g, int *scratch_d, bool *in_grouped, cudaStream_t s) {
  int h[4] = {0, 0, 0, 0};
  t_range_init_kernel<<<1, 1, 0, s>>>(scratch_d);
  if (g.num_edges > 0) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g.device);
    t_range_kernel<<<sms * 4, 256, 0, s>>>(g.edges, (int)g.num_edges, scratch_d);
  }
  EVX_CUDA(cudaGetLastError());
  EVX_CUDA(cudaMemcpyAsync(h, scratch_d, sizeof(h), cudaMemcpyDeviceToHost, s));
  EVX_CUDA(cudaStreamSynchronize(s));
  if (h[3]) return fail(EVX_ERR_INVALID, "the out/in lists do not hold every edge once");
  *in_grouped = h[2] == 0;
  g.min_t = g.num_edges ? h[0] : 0;
  g.max_t = g.num_edges ? h[1] : 0;
  return EVX_OK;
}

}  // namespace evx
