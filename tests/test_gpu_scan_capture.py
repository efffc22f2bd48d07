"""The first scan of a process under a stream capture, in each capture mode, and (relaxed) on a stream beside the one that
is captured: a process of its own for each."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes, sys
import numpy as np, torch
import vkscanlinepr_gb300 as sr
mode, beside, n = sys.argv[1], sys.argv[2] == "beside", 300001
sr.lib()
x = torch.randint(0, 40, (n,), dtype=torch.int32, device="cuda")
o, y = torch.zeros(n + 1, dtype=torch.int32, device="cuda"), torch.zeros_like(x)
other = torch.cuda.Stream()
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, capture_error_mode=mode):
    st = other.cuda_stream if beside else torch.cuda.current_stream().cuda_stream
    sr.exclusive_scan_i32(x.data_ptr(), o.data_ptr(), n, ctypes.c_void_p(st))
    y.copy_(x)
want = np.concatenate([[0], np.cumsum(x.cpu().numpy().astype(np.int64))]).astype(np.int32)
other.synchronize()
for _ in range(2):
    if not beside:
        o.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(o.cpu().numpy(), want) and torch.equal(x, y)
sr.scan_status()
"""


@pytest.mark.parametrize("mode,where", [("global", "captured"), ("thread_local", "captured"), ("relaxed", "captured"),
                                        ("relaxed", "beside")])
def test_first_scan(gpu, mode, where):
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE, mode, where], cwd=repo, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-1500:]
