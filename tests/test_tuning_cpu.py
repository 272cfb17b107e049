"""The tuning that a worker starts with can be asked for again: set_tuning()
without arguments, and the tuner's restore after its trials, leave the interval
to the rule (-1), as in a new worker."""
import types

from everest_b200 import autotune, capi


def test_defaults_are_a_new_workers(monkeypatch):
    seen = []
    fake = types.SimpleNamespace(evx_worker_set_tuning=lambda h, *a: seen.append(a) or 0)
    monkeypatch.setattr(capi, "lib", lambda: fake)
    w = types.SimpleNamespace(_h=None)
    capi.Worker.set_tuning(w)
    w.set_tuning = lambda **kw: capi.Worker.set_tuning(w, **kw)
    assert autotune.Autotuner.apply(w, autotune.DEFAULT) == 0
    assert [x[1:] for x in seen] == [(0, 32, -1, 2)] * 2  # blocks per SM, roots per fetch, interval, split


def test_candidates_differ_whatever_the_rules_say():
    # the interval (4 or 16) and the window bound (on or off) that a query's
    # default resolves to: no two other candidates are the same search, and one
    # at most is the default's
    on, off = capi.FLAG_ROOT_BOUND, capi.FLAG_NO_ROOT_BOUND
    for interval in (4, 16):
        for bound in (on, off):
            seen = []
            for c in autotune.CANDIDATES:
                flags = c["flags"] if c["flags"] & (on | off) else c["flags"] | bound
                seen.append((c["blocks_per_sm"], interval if c["steal_interval"] < 0 else c["steal_interval"],
                             c["min_split"], flags))
            assert len(set(seen)) >= len(seen) - 1
            assert len(set(seen[1:])) == len(seen) - 1
