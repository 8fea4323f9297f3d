"""Memory ordering of the waits in the tensor-core contraction kernel (green-mbpt_b200/csrc/split.cu), read from the
source: where one lane of a warp waits on an mbarrier for all of it, a __syncwarp must follow before the other lanes
touch what the barrier guards.  A shuffle of the outcome, which also brings the lanes together, orders no memory."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ONE_LANE = re.compile(r"if \((?:lane|threadIdx\.x % 32) == 0\)\s*ok = mbar_wait\(")


def test_single_lane_waits_are_followed_by_syncwarp():
    with open(os.path.join(ROOT, "green-mbpt_b200", "csrc", "split.cu")) as f:
        src = f.read()
    found = list(ONE_LANE.finditer(src))
    assert found, "the pattern no longer matches the kernel's waits"
    for m in found:
        rest = src[src.index(";", m.end()) + 1:]
        assert rest.lstrip().startswith("__syncwarp();"), src[m.start():m.end() + 200]
