"""bench.py reads the query kernel's limiter and DRAM traffic from the committed
profile summary: what it finds there is what the summary says."""
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402


def _profile():
    with open(os.path.join(ROOT, "profiles", "k_query_uneven_batch_k16.txt")) as f:
        return f.read()


def test_limiter_is_read_from_the_profile():
    limiter = bench.profiled_limiter(16)
    assert limiter is not None
    assert 0 < limiter["alu_pipe_active_pct"] <= 100
    assert 0 < limiter["issue_active_pct"] <= 100
    assert limiter["warp_instructions_per_query"] > 0
    assert limiter["source"] == os.path.join("profiles", "k_query_uneven_batch_k16.txt")


def test_traffic_is_the_profiles_read_and_write():
    text = _profile()
    parts = [int(re.search(rf"dram__bytes_{way}\.sum\s+([0-9,]+) B", text).group(1).replace(",", ""))
             for way in ("read", "write")]
    assert bench.profiled_traffic(16) == sum(parts)


def test_profile_is_of_one_kernel():
    """One capture, one set of figures: no column of a replaced kernel."""
    assert "before" not in _profile().split("reading")[0]


def test_no_profile_no_claim():
    assert bench.profiled_limiter(17) is None and bench.profiled_traffic(17) is None
