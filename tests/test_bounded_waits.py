"""The bounded waits of the warp-specialised kernels, by their source: what a
role that gave up must still do."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parents[1] / "eemd4cuda_b200" / "csrc" / "surrogate.cu").read_text()
KERNELS = ["k_conv_ws", "k_wgrad_ws"]


def body(name):
    i = SOURCE.index(" %s(const" % name)
    j = SOURCE.index("\n}\n", i)
    return SOURCE[i:j]


@pytest.mark.parametrize("name", KERNELS)
def test_last_waits_do_not_take_the_callers_limit(name):
    """A wait whose outcome nothing looks at is there for what it waits for
    (copies into shared memory, MMAs on tensor memory about to be freed)."""
    unread = re.findall(r"(?:^|[;{})])\s*(wait_parity\([^;]*\));", body(name), flags=re.M)
    assert len(unread) == 2
    assert all(w.endswith("DRAIN_SPINS)") for w in unread), unread


@pytest.mark.parametrize("name", KERNELS)
def test_a_warps_lanes_agree_on_giving_up(name):
    """What a vote decides is the same in every lane of a warp only if no lane
    adds a read of the shared flag after it."""
    votes = re.findall(r"=\s*(__all_sync\(.*?\));", body(name), flags=re.S)
    assert votes
    for v in votes:
        depth = 0
        for i, ch in enumerate(v):
            depth += (ch == "(") - (ch == ")")
            if depth == 0 and i >= len("__all_sync"):
                assert v[i + 1:].strip() == "", v
                break
