"""A slot of the refinement queue is taken only for a patch that will be written.

`k_refine` trusts the queue's counter: it indexes the points with every counted slot's entry. A
kernel whose bounded wait for the products runs out leaves without a patch, so it must not have
taken a slot by then, or `k_refine` would index with whatever an earlier pass (or nothing) left there.
"""

import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parents[1] / "autorift.jl_b200" / "csrc" / "ar_track.cu"


def kernel(name):
    text = SRC.read_text()
    start = re.search(r"__global__ void __launch_bounds__\([^)]*\) " + name + r"\(const \w+ A\) \{", text).end()
    end = text.find("__global__", start)
    body = text[start:end if end > 0 else None]
    return re.sub(r"//[^\n]*", "", body)


@pytest.mark.parametrize("name", ["k_corr_tc", "k_corr_bf"])
def test_slot_is_taken_after_the_last_wait_that_can_run_out(name):
    body = kernel(name)
    give_up = body.index("failed = true;")
    assert body.count("failed = true;") == 1
    slot = body.index("atomicAdd(A.sub_count")
    assert body.count("atomicAdd(A.sub_count") == 1
    assert slot > give_up
    # From the slot on nothing is waited for before its patch is written.
    written = body.index("A.sub_point[slot] = k;")
    assert slot < written and "mbar_wait" not in body[slot:written]
