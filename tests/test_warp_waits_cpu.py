"""Memory ordering of the waits in the tensor-core contraction kernel (green-mbpt_b200/csrc/split.cu), read from the
source: lanes that touch what an mbarrier guards wait for it themselves.  Where one lane waits for its whole warp, a
__syncwarp must follow; a shuffle of the outcome, which also brings the lanes together, orders no memory."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ONE_LANE = re.compile(r"if \((?:lane|threadIdx\.x % 32) == 0\)\s*ok = mbar_wait\(")


def test_no_outcome_of_a_wait_is_handed_over_by_a_shuffle():
    with open(os.path.join(ROOT, "green-mbpt_b200", "csrc", "split.cu")) as f:
        src = f.read()
    assert src.count("mbar_wait(&tabe_bar") == src.count("mbar_wait(&tabf_bar") == src.count("mbar_wait(&accf_bar") == 1
    for m in ONE_LANE.finditer(src):
        rest = src[src.index(";", m.end()) + 1:]
        assert rest.lstrip().startswith("__syncwarp();"), src[m.start():m.end() + 200]
    assert not re.search(r"__shfl_sync\(0xffffffffu, ok", src)
