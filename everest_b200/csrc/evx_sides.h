// Streams beside a batch's own.  Plain C++ over an Api type that names the
// runtime's streams, events and calls, so that host tests can run it against a
// runtime that fails.
#ifndef EVX_SIDES_H_
#define EVX_SIDES_H_

#include <mutex>

namespace evx {

// Streams beside the batch's own (64 mixed queries over 250k-root windows, eight
// launches: 24.6 ms with one, 20.1 with six).
constexpr int kSides = 6;

// Idle streams that destroyed batches gave back, of every priority: creating one
// takes up to 0.5 ms.  At most kSpare of a device are kept.
template <class Api>
class SparePool {
 public:
  static constexpr int kSpare = 4 * kSides, kMost = 256;

  typename Api::Error take(int device, int priority, typename Api::Stream *s) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      for (int i = 0; i < n_; i++) {
        if (spare_[i].device != device || spare_[i].priority != priority) continue;
        *s = spare_[i].stream;
        spare_[i] = spare_[--n_];
        return Api::kOk;
      }
    }
    return Api::create(s, priority);
  }

  // (s is idle)
  void give(int device, int priority, typename Api::Stream s) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      int kept = 0;
      for (int i = 0; i < n_; i++) kept += spare_[i].device == device;
      if (kept < kSpare && n_ < kMost) {
        spare_[n_++] = {device, priority, s};
        return;
      }
    }
    Api::destroy(s);
  }

 private:
  struct Spare {
    int device, priority;
    typename Api::Stream stream;
  };
  std::mutex mu_;
  Spare spare_[kMost] = {};
  int n_ = 0;
};

// A batch's side streams, of its own stream's priority, taken when first needed
// and its alone until dropped.
template <class Api>
struct Sides {
  using Error = typename Api::Error;
  using Stream = typename Api::Stream;
  using Event = typename Api::Event;
  Stream side[kSides] = {};
  Event fork = {}, join[kSides] = {};
  int priority = 0;
  bool astray = false;  // a side stream may have work that the batch's stream has not joined

  // Make run() of n launches on `sides` streams possible (before a capture begins).
  Error ready(SparePool<Api> &pool, int device, Stream own, int n, int sides) {
    Error e = settle();
    if (!sides) return e;
    if (e == Api::kOk && n > 1 && !fork) e = Api::priority(own, &priority);
    if (e == Api::kOk && n > 1 && !fork) e = Api::create_event(&fork);
    for (int i = 0; e == Api::kOk && i < sides && i + 1 < n; i++) {
      if (!side[i]) e = pool.take(device, priority, &side[i]);
      if (e == Api::kOk && !join[i]) e = Api::create_event(&join[i]);
    }
    return e;
  }

  // launch(i, stream) for i in [0, n): the first on `own`, the others beside it
  // on `sides` streams and joined to it (none: all on `own`, one after the
  // other).  What was forked is joined on an error too, the first
  // error is returned, and a stream whose join failed is waited for before it
  // is used again or given away.
  template <class F>
  Error run(Stream own, int n, int sides, F launch) {
    Error e = n > 1 && sides ? Api::record(fork, own) : Api::kOk;
    int forked = 0;
    for (int i = 0; e == Api::kOk && i < n; i++) {
      if (i > forked && forked < sides) {
        e = Api::wait(side[forked], fork);
        if (e != Api::kOk) break;
        forked++;
      }
      e = launch(i, i && sides ? side[(i - 1) % sides] : own);
    }
    for (int i = 0; i < forked; i++) {
      Error j = Api::record(join[i], side[i]);
      if (j == Api::kOk) j = Api::wait(own, join[i]);
      if (j == Api::kOk) continue;
      astray = true;
      if (e == Api::kOk) e = j;
    }
    return e;
  }

  Error settle() {
    Error e = Api::kOk;
    for (int i = 0; astray && i < kSides; i++) {
      const Error x = side[i] ? Api::synchronize(side[i]) : Api::kOk;
      if (x != Api::kOk) e = x;
    }
    if (e == Api::kOk) astray = false;
    return e;
  }

  // Give the streams back (the batch's own has been waited for).
  void drop(SparePool<Api> &pool, int device) {
    settle();
    for (int i = 0; i < kSides; i++) {
      if (join[i]) Api::destroy_event(join[i]);
      if (side[i] && astray) Api::destroy(side[i]);
      else if (side[i]) pool.give(device, priority, side[i]);
    }
    if (fork) Api::destroy_event(fork);
    *this = Sides();
  }
};

}  // namespace evx

#endif  // EVX_SIDES_H_
