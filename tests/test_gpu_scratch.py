"""Calls whose scratch memory is refused go on without it: the K split is left out, Q4_K_M linears and prompts over INT8 caches or
rings that wrap take the kernels that need none.  The library reads the limit once, so the tests that cover these calls run
in a process of their own."""
import os
import subprocess
import sys

import pytest

from helpers import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [0, 300000])  # bytes: none, and enough for a Q4_K_M linear's activations but not for its parts
def test_refused_scratch(most):
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", "tests/test_gpu_linear_tiles.py", "tests/test_gpu_prompt_attention.py",
           "tests/test_gpu_tovelix.py::test_window_attention", "-k", "q4km or tensor_core_tiles or 16_byte or test_window or (test_prompt_attention and not finite)"]
    r = subprocess.run(cmd, cwd=ROOT, env=dict(os.environ, AB2_SCRATCH_MAX_BYTES=str(most)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
