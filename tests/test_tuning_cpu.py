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
