"""A ring slot goes back to the thread that refills it by one lane's arrival for its whole warp. That arrival releases the lane's own
reads and writes; what the other 31 lanes did is ordered before it by a __syncwarp (a vote such as __all_sync orders
no memory accesses). The order cannot be seen to fail on a device on demand, so it is read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qwen38-3090-cuda-server_b200", "csrc")
# barriers that hand over what a whole warp read or wrote with ordinary accesses or tensor-memory loads and stores
HANDED_OVER = ("wempty_a", "afull_a", "afull_l", "dempty_a", "dempty_l", "mailfull_a", "bready_a", "tmemrdy_a")


def _arrivals(name):
    """(line number, barrier, the code in front of the arrival: comments out, the lane test and fellow arrivals skipped)."""
    with open(os.path.join(CSRC, name)) as f:
        lines = [re.sub(r"//.*", "", line).strip() for line in f]
    for i, line in enumerate(lines):
        m = re.match(r"(?:if \(\w+\) |if \(lane == 0\) )?mbar_arrive(?:_cluster)?\((\w+)", line)
        if not m or m.group(1) not in HANDED_OVER:
            continue
        if line.startswith("if (lane == 0)"):
            inside, j = True, i - 1
        else:
            j = i - 1
            while re.match(r"(if \(\w+\) )?mbar_arrive", lines[j]):
                j -= 1
            inside = lines[j] == "if (lane == 0) {"
            j -= 1
        assert inside, f"{name}:{i + 1}: not one lane's arrival"
        while not lines[j]:
            j -= 1
        yield i + 1, m.group(1), lines[j]


@pytest.mark.parametrize("name,count", [("prefill.cu", 3), ("skinny.cu", 8)])
def test_one_lane_arrives_behind_a_syncwarp(name, count):
    seen = list(_arrivals(name))
    assert len(seen) >= count
    for line, bar, before in seen:
        assert before == "__syncwarp();", f"{name}:{line}: {bar} is handed over behind `{before}`"
