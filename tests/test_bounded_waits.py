"""A warp of the tcgen05 kernels gives up a wait as a whole.  Waits on an mbarrier are bounded, and a lane that stops after one
while others of its warp go on leaves them waiting in the warp's next collective instruction (a vote, a shuffle, a
tensor-memory load) for good.  So outside the branch of one lane no lane leaves a loop by a wait, or by the CTA's `failed`, of
its own: the sources are read for such statements, which no launch that meets its bounds would show."""
import os
import re

import pytest

from helpers import ROOT

CSRC = os.path.join(ROOT, "aarambh-ai_b200", "csrc")
KERNELS = ["gemm_bf16_tc.cu", "gemm_w4a16_tc.cu", "gemm_i8_tc.cu", "gemm_q4km_tc.cu", "gemv_w4a16_tc.cu", "attention_prompt_tc.cu"]
ONE_LANE = re.compile(r"\b(lane|threadIdx\.x) == 0\b")
VOTE = re.compile(r"\b(warp_wait|__any_sync|__all_sync)\(")


def statements(text):
    """(headers of the enclosing blocks, statement) in order; a header is what stands before a block's brace."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
    blocks, start, depth = [], 0, 0
    for i, c in enumerate(text):
        depth += (c == "(") - (c == ")")
        if depth or c not in "{};":
            continue
        part = text[start:i].strip()
        start = i + 1
        yield list(blocks), part
        if c == "{":
            blocks.append(part)
        elif c == "}" and blocks:
            blocks.pop()


def lanes_that_leave_alone(text):
    for blocks, part in statements(text):
        if any(ONE_LANE.search(b) for b in blocks + [part]):
            continue
        leaves = re.search(r"\bbreak\b", part) and re.search(r"(?<!\w)bar_wait\(", part)
        asks = re.match(r"(for|while|if)\b", part) and re.search(r"\*failed\b", part) and not VOTE.search(part)
        if leaves or asks:
            yield part


@pytest.mark.parametrize("name", KERNELS)
def test_warps_decide_together(name):
    with open(os.path.join(CSRC, name)) as f:
        assert list(lanes_that_leave_alone(f.read())) == []


def test_the_reader_sees_them():
    text = """if (warp == 1) { for (int i = 0; i < n && !*failed; ++i) { if (!bar_wait(&b[i], 0, failed)) break; vote(); } }
              else if (lane == 0) { for (int i = 0; i < n && !*failed; ++i) { if (!bar_wait(&b[i], 0, failed)) break; } }
              else { bool ok = true; for (int i = 0; i < n && ok; ++i) { ok = warp_wait(&b[i], 0, failed); if (!ok) break; } }
              if (!*failed) { store(); }"""
    assert list(lanes_that_leave_alone(text)) == ["for (int i = 0; i < n && !*failed; ++i)", "if (!bar_wait(&b[i], 0, failed)) break", "if (!*failed)"]
