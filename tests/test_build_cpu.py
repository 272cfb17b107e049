"""The build's compiler commands are the same on every machine: what a kernel
compiles to (its registers, its spills) must not depend on the number of CPUs."""
import os

from everest_b200 import build


def test_commands_do_not_depend_on_the_cpu_count(monkeypatch):
    seen = []
    for cpus in (2, 64):
        cmds = []
        monkeypatch.setattr(os, "cpu_count", lambda: cpus)
        monkeypatch.setattr(build, "_run", lambda cmd, verbose: cmds.append(cmd))
        build.build(force=True)
        seen.append(sorted(cmds))
    assert seen[0] == seen[1]
    flags = [f for cmd in seen[0] for f in cmd]
    # (0 parts means one per CPU, and the parts change the code)
    assert not [f for f in flags if "split-compile" in f]
    assert sum("-DEVX_K=" in f for f in flags) == 7
