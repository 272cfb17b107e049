// Side streams of a batch (everest_b200/csrc/evx_sides.h) against a runtime
// that fails at any one of its calls.  Prints "ok" or the first broken rule.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>
#include <vector>

#include "evx_sides.h"

#define CHECK(c) \
  do { if (!(c)) { std::printf("line %d: %s (n %d, call %d)\n", __LINE__, #c, g_n, g_fail); std::exit(1); } } while (0)

static int g_n, g_fail, g_calls;

struct Fake {
  using Error = int;
  using Stream = int;
  using Event = int;
  static constexpr Error kOk = 0;
  static inline int next = 1;
  static inline std::map<int, int> work, done;   // per stream: launches made, launches known to have ended
  static inline std::map<int, std::pair<int, int>> at;  // event -> stream, launches it covers
  static inline std::set<int> streams, events, forked;
  static int call() { return ++g_calls == g_fail ? 7 : 0; }
  static inline std::map<int, int> prio;
  static Error create(Stream *s, int p) {
    if (int e = call()) return e;
    *s = next++;
    streams.insert(*s);
    prio[*s] = p;
    return 0;
  }
  static Error priority(Stream, int *p) { if (int e = call()) return e; *p = own_priority; return 0; }
  static inline int own_priority = 0;
  static Error destroy(Stream s) { CHECK(streams.erase(s) == 1); return call(); }
  static Error synchronize(Stream s) { if (int e = call()) return e; done[s] = work[s]; return 0; }
  static Error create_event(Event *v) { if (int e = call()) return e; *v = next++; events.insert(*v); return 0; }
  static Error destroy_event(Event v) { CHECK(events.erase(v) == 1); return call(); }
  static Error record(Event v, Stream s) { if (int e = call()) return e; at[v] = {s, work[s]}; return 0; }
  static Error wait(Stream s, Event v) {
    if (int e = call()) return e;
    CHECK(at.count(v));
    if (at[v].first == kOwn) forked.insert(s);
    if (s == kOwn) done[at[v].first] = at[v].second;
    return 0;
  }
  static constexpr int kOwn = -1;
};

int main() {
  for (int round = 0; round < 30; round++) {
    g_n = 1 + round % 15;
    const int sides = round < 15 ? evx::kSides : 0;
    int last = 0;
    for (g_fail = 0; g_fail <= last; g_fail++) {
      evx::SparePool<Fake> pool;
      evx::Sides<Fake> s;
      Fake::own_priority = -(g_n % 3);
      bool failed = false;
      g_calls = 0;
      for (int pass = 0; pass < 2; pass++) {
        Fake::forked.clear();
        if (s.ready(pool, 0, Fake::kOwn, g_n, sides)) { failed = true; continue; }
        for (int x : Fake::streams) CHECK(Fake::work[x] == Fake::done[x]);  // nothing is taken busy
        int ran = 0;
        const int e = s.run(Fake::kOwn, g_n, sides, [&](int i, int st) {
          CHECK(i == ran);
          ran++;
          CHECK(i == 0 || !sides ? st == Fake::kOwn : Fake::forked.count(st) == 1);
          CHECK(st == Fake::kOwn || Fake::prio[st] == Fake::own_priority);
          Fake::work[st]++;
          return Fake::call();
        });
        CHECK(e || ran == g_n);
        if (e) failed = true;
        for (int x : Fake::streams) CHECK(Fake::work[x] == Fake::done[x] || s.astray);
      }
      CHECK(!failed == (g_fail == 0 || g_calls < g_fail));  // every failure is reported
      s.drop(pool, 0);
      if (g_fail == 0) last = g_calls;
      CHECK(Fake::events.empty());
      // what the pool hands out is idle
      const int mark = Fake::next;
      for (int i = 0; i < evx::kSides; i++) {
        int x = 0;
        if (pool.take(0, Fake::own_priority, &x)) continue;
        CHECK(x >= mark || Fake::work[x] == Fake::done[x]);
        Fake::destroy(x);
      }
      CHECK(Fake::streams.empty());
    }
  }
  // a device's idle streams are bounded, and keep their device and priority
  evx::SparePool<Fake> pool;
  g_fail = 0;
  std::vector<int> got;
  for (int i = 0; i < 100; i++) { int x; Fake::create(&x, -1); got.push_back(x); }
  for (int x : got) pool.give(1, -1, x);
  CHECK((int)Fake::streams.size() == evx::SparePool<Fake>::kSpare);
  int x;
  CHECK(pool.take(0, -1, &x) == 0 && x > got.back());
  CHECK(pool.take(1, 0, &x) == 0 && x > got.back());
  CHECK(pool.take(1, -1, &x) == 0 && x <= got.back());
  std::printf("ok\n");
}
