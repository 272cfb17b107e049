"""The bench line holds what its own run measured: no figure of an earlier
profile is read into it."""
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_profile_is_read():
    with open(os.path.join(ROOT, "bench.py")) as f:
        text = f.read()
    assert "profiles" not in text and "traffic_bytes_per_step" not in text
