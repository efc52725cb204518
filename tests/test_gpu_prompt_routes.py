"""Prompt attention is taken by the kernel that is estimated to be the faster one.  The tests of prompts run once more in processes of their
own with every prompt that it serves sent to the tcgen05 kernel, and with none, so that both are tested at every size."""
import os
import subprocess
import sys

import pytest

from helpers import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("route", ["tc", "other"])
def test_prompts_by_one_kernel(route):
    # values that are not finite: the warp-level kernels multiply hidden ones of a tile too, as they always have
    skip = [] if route == "tc" else ["-k", "not not_finite"]
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", "tests/test_gpu_prompt_attention.py", "tests/test_gpu_prompt_rows.py",
           "tests/test_gpu_tovelix.py::test_window_attention"] + skip
    r = subprocess.run(cmd, cwd=ROOT, env=dict(os.environ, AB2_PROMPT_ATTN=route), capture_output=True, text=True, timeout=400)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
