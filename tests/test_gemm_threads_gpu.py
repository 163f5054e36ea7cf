"""The GEMM called from a thread that has done no CUDA work before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def test_a_gemm_may_be_the_first_work_of_a_thread():
    """Autograd runs a backward pass on its own thread, whose first CUDA call can be the GEMM's tensor-map encoder.  In a
    process of its own: where the thread has no context the call ends the process."""
    code = """
import threading, torch
from autoparallel_b200.ops import cuda_impl, library
cuda_impl.ensure_loaded()
a = torch.randn(999, 2048, device="cuda", dtype=torch.bfloat16)
w = torch.randn(1408, 2048, device="cuda", dtype=torch.bfloat16)
ref, out = cuda_impl._mm_nd(a, w, True, torch.bfloat16), []
torch.cuda.synchronize()
t = threading.Thread(target=lambda: out.append(cuda_impl._mm_nd(a, w, True, torch.bfloat16)))
t.start(), t.join()
torch.cuda.synchronize()
assert torch.equal(out[0], ref)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-2000:]
