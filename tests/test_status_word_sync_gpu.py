"""The status word of a process that has made no asynchronous call: every call is a synchronous one, good
calls leave the stream alone, a wait that runs out in the native or the tensor-core kernels is reported
by the call it happened in, and the next call is good again.  A fresh process for each method, since one
asynchronous call changes the route for the rest of a process.  The same then after an asynchronous call."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import torch
import blaze_gb300 as G

method, before = sys.argv[1], sys.argv[2] == "async"
m, n, k = 300, 280, 512
A = torch.rand(m, k, device="cuda", dtype=torch.float64)
B = torch.rand(k, n, device="cuda", dtype=torch.float64)
C = torch.empty(m, n, device="cuda", dtype=torch.float64)
torch.cuda.synchronize()


def call(**kw):
    C.zero_()
    torch.cuda.synchronize()
    G.dgemm_ex(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, C, n, G.opts(method=method, **kw))
    assert G.lib().gb300_synchronize() == G.OK
    assert torch.allclose(C, A @ B, rtol=1e-12)


if before:
    call(synchronous=False)
call()
for _ in range(2):
    G.lib().gb300_debug_inject_stall(1, 2_000_000)  # 2 ms: the kernel's own waits run out
    try:
        G.dgemm_ex(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, C, n, G.opts(method=method))
        sys.exit("the stalled call was not reported")
    except G.Gb300Error as e:
        assert e.status == G.ERR_DEVICE_TIMEOUT, e
    call()
    call()
print("status ok")
"""


@pytest.mark.parametrize("before", ["sync", "async"])
@pytest.mark.parametrize("method", ["native", "split", "bf16x3"])
def test_fresh_process(method, before):
    tol = "1e-12" if method != "bf16x3" else "1e-3"
    r = subprocess.run([sys.executable, "-c", CHILD.replace("rtol=1e-12", "rtol=" + tol), method, before], cwd=ROOT,
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "status ok" in r.stdout, r.stdout + r.stderr
