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
  const SearchKernel x{enumerate, plan_pair_scan(plan, q0.flags, enumerate), cons_any(args.cons), q0.flags & kTailFlags};
  return launch(k, x, g, q0, la, ea, grid, stream);
}

int launch_table(const GraphView &g, const QueryDesc &q0, const LaunchArgs &la, int k, int tail, bool ps, int grid,
                 cudaStream_t stream) {
  EnumArgs ea;
  memset(&ea, 0, sizeof(ea));
  return launch(k, SearchKernel{false, ps, false, tail}, g, q0, la, ea, grid, stream);
}

int search_occupancy(int k, int qflags, bool enumerate, bool ps, bool cs, int block, int *blocks_per_sm) {
  (void)block;
  return occupancy(k, SearchKernel{enumerate, ps, cs, qflags & kTailFlags}, blocks_per_sm);
}

int table_occupancy(int k, int tail, bool ps, int *blocks_per_sm) {
  return occupancy(k, SearchKernel{false, ps, false, tail}, blocks_per_sm);
}

int tail_of(int k, int qflags) {
  const int t = qflags & kTailFlags, way = t & ~kQStrict;
  const bool one =
      way == kQInlineLast || way == kQSamePair || way == kQRevPair || way == kQPairHash || way == kQNewArith;
  return k >= 3 && k <= 5 && one ? t : kTailAny;
}

}  // namespace evx
