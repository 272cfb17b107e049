"""The streams beside a batch's own, on the host: whichever call of the runtime
fails, what was forked is joined or waited for before it is used again, and no
stream goes back to the pool with work that nothing waited for."""
import os
import subprocess

from everest_b200 import build


def test_any_call_may_fail(tmp_path):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "sides_host.cc")
    exe = str(tmp_path / "sides")
    subprocess.run([build._cxx(), "-std=c++17", "-pthread", "-I", build.CSRC, "-o", exe, src], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert (r.returncode, r.stdout.strip()) == (0, "ok"), r.stdout
