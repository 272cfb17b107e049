// Choice and launch of the search kernels (evx_search.cu has the kernels, one
// object per motif size).
#include <cstring>

#include "evx_internal.cuh"

namespace evx {
namespace {

// Single-query launch description from the worker's SearchArgs.
QueryDesc single_query(const MotifPlan &plan, const SearchArgs &args) {
  QueryDesc q;
  memset(&q, 0, sizeof(q));
  q.plan = plan;
  q.root_beg = args.root_beg;
  q.root_end = args.root_end;
  q.delta = args.delta;
  q.flags = (args.strict_ts ? kQStrict : 0) | args.tail_flags;
  q.steal_interval = args.steal_interval;
  q.min_split = args.min_split;
  q.tile_beg = 0;
  return q;
}

// f<K>(args...) for the motif size k
#define EVX_SIZES(f, ...)                                                   \
  switch (k) {                                                              \
    case 2: return f<2>(__VA_ARGS__);                                       \
    case 3: return f<3>(__VA_ARGS__);                                       \
    case 4: return f<4>(__VA_ARGS__);                                       \
    case 5: return f<5>(__VA_ARGS__);                                       \
    case 6: return f<6>(__VA_ARGS__);                                       \
    case 7: return f<7>(__VA_ARGS__);                                       \
    case 8: return f<8>(__VA_ARGS__);                                       \
    default: return fail(EVX_ERR_INVALID, "motif edge count out of range"); \
  }
static_assert(EVX_MAX_MOTIF_EDGES == 8, "one case per motif size");

int launch(int k, const SearchKernel &x, const GraphView &g, const QueryDesc &q0, const LaunchArgs &la,
           const EnumArgs &ea, int grid, cudaStream_t s) {
  EVX_SIZES(launch_size, x, g, q0, la, ea, grid, s)
}

int occupancy(int k, const SearchKernel &x, int *blocks_per_sm) {
  EVX_SIZES(occupancy_size, x, blocks_per_sm)
}

}  // namespace

// Whether a query walks a pair run at some level: an edge between two nodes
// mapped before it that is scanned (every level before the last; the last
// one only when enumerating: a counted closing last edge takes range
// arithmetic instead).
bool plan_pair_scan(const MotifPlan &plan, int qflags, bool enumerate) {
  if (!(qflags & kQPairScan)) return false;
  for (int l = 0; l <= plan.k - 2; l++) {
    if (plan_kind(plan.info[l]) != 2) continue;
    if (l < plan.k - 2 || enumerate) return true;
  }
  return false;
}

int launch_search(const GraphView &g, const MotifPlan &plan, const SearchArgs &args, int grid, int block,
                  cudaStream_t stream) {
  (void)block;
  const int k = plan.k;
  const bool enumerate = args.enumerate != 0;
  const QueryDesc q0 = single_query(plan, args);
  LaunchArgs la{};
  la.table = nullptr;
  la.nq = 1;
  const int n = args.root_end - args.root_beg;
  la.tile_roots = tile_roots_for(k, n, 1, (long long)grid * (kSearchBlock / 32), n);
  if (la.tile_roots == 0) return fail(EVX_ERR_OVERFLOW, "root tiles would overflow int32");
  la.total_tiles = (int)tiles_of(n, la.tile_roots);
  la.cursor = args.cursor;
  la.counts = args.count;
  la.limit = args.limit;
  la.meter = args.meter;
  EnumArgs ea;
  ea.rows = args.rows;
  ea.cap = args.cap;
  ea.exact_total = args.exact_total;
  ea.stop = args.stop;
  ea.count = args.count;
  la.state = args.state;
  la.out = args.out;
  la.cons = args.cons;
  const SearchKernel x{enumerate, plan_pair_scan(plan, q0.flags, enumerate), cons_any(args.cons),
                       tail_of(k, q0.flags, n)};
  return launch(k, x, g, q0, la, ea, grid, stream);
}

int launch_table(const GraphView &g, const QueryDesc &q0, const LaunchArgs &la, int k, int tail, bool ps, int grid,
                 cudaStream_t stream) {
  EnumArgs ea;
  memset(&ea, 0, sizeof(ea));
  return launch(k, SearchKernel{false, ps, false, tail}, g, q0, la, ea, grid, stream);
}

int search_occupancy(int k, int qflags, long long roots, bool enumerate, bool ps, bool cs, int block,
                     int *blocks_per_sm) {
  (void)block;
  return occupancy(k, SearchKernel{enumerate, ps, cs, tail_of(k, qflags, roots)}, blocks_per_sm);
}

int table_occupancy(int k, int tail, bool ps, int *blocks_per_sm) {
  return occupancy(k, SearchKernel{false, ps, false, tail}, blocks_per_sm);
}

// A launch of fewer roots than warps ends with its heaviest roots, each alone on
// its warp, where the kernels with every way, at more registers and fewer blocks
// per SM, go faster: requests over windows of 1000 roots of 63M edges, per way
// and with every way, five edges with a pair-table last edge 8918 / 7987 ms (23
// requests), a new node 6086 / 4964 (113), a fixed pair 1471 / 1361 (442); four
// edges with a new node 282 / 244 (320), but a fixed pair 123 / 151 (42).  Over
// 20k roots of 7.8M edges both are even, over all of 1.3M edges one way takes 10
// to 25 % less.
int tail_of(int k, int qflags, long long roots) {
  const int t = qflags & kTailFlags, way = t & ~kQStrict;
  const bool one =
      way == kQInlineLast || way == kQSamePair || way == kQRevPair || way == kQPairHash || way == kQNewArith;
  const bool few = roots < kFewRoots && (k == 5 || (k == 4 && way == kQNewArith));
  return k >= 3 && k <= 5 && one && !few ? t : kTailAny;
}

}  // namespace evx
