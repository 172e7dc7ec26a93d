"""The first tensor-core product of a process loads its device code, which takes about a millisecond (eleven
while the code came compressed)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys, time
import torch
import blaze_gb300 as G
n = 512
dt, call = (torch.float64, G.dgemm_ex) if sys.argv[1] == "d" else (torch.float32, G.sgemm_ex)
A = torch.rand(n, n, device="cuda", dtype=dt)
C = torch.empty_like(A)
torch.cuda.synchronize()
for method in ("native", "split"):  # the native call sets the library up
    t = time.perf_counter()
    call(G.RowMajor, G.NoTrans, G.NoTrans, n, n, n, 1.0, A, n, A, n, 0.0, C, n, G.opts(method=method))
    ms = 1e3 * (time.perf_counter() - t)
print(ms)
"""


@pytest.mark.parametrize("dtype", ["d", "s"])
def test_first_split_product(dtype):
    ms = []
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", CHILD, dtype], cwd=ROOT, capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr
        ms.append(float(r.stdout))
    assert min(ms) < 5.0, ms
