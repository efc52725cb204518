"""Tensor memory of a pair of CTAs (cta_group::2) is allocated and given back by both together, and PTX asks that the other CTA is running
whenever one of them does: a cluster barrier has to stand ahead of the allocation and behind the deallocation, in the source of
every kernel that multiplies by pairs."""
import glob
import os

import pytest

from helpers import ROOT

FILES = [f for f in sorted(glob.glob(os.path.join(ROOT, "aarambh-ai_b200", "csrc", "*.cu"))) if "tcgen05.alloc.cta_group::2" in open(f).read()]


def kernels(text):
    """Bodies of the __global__ functions."""
    at = text.find("__global__")
    while at >= 0:
        start = text.index("{", text.index(")", text.index("(", text.index("kernel", at))))
        depth, i = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield text[start:i]
        at = text.find("__global__", i)


def test_there_are_such_kernels():
    assert [os.path.basename(f) for f in FILES] == ["gemm_bf16_tc.cu"]


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_the_other_cta_is_there(path):
    seen = 0
    for body in kernels(open(path).read()):
        if "tcgen05.alloc.cta_group::2" not in body:
            continue
        seen += 1
        assert "cluster_sync_all();" in body[:body.index("tcgen05.alloc.cta_group::2")]
        assert "cluster_sync_all();" in body[body.rindex("tcgen05.dealloc.cta_group::2"):]
        # arrivals of the other CTA's MMAs are waited for before either leaves
        assert "(u / STAGES) & 1" in body
    assert seen
