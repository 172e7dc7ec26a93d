"""After autotuning, a mixed batch of ten thousand products takes no longer than with the default shapes (in
a child process: the tuning state is the process's)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import math, random, sys
import torch
import blaze_gb300 as G

esz = int(sys.argv[1])
r = random.Random(5)
sizes = [tuple(round(math.exp(r.uniform(math.log(4), math.log(256)))) for _ in range(3)) for _ in range(10000)]
dt = torch.float64 if esz == 8 else torch.float32
ab = torch.rand(sum(m * k + k * n for m, n, k in sizes), device="cuda", dtype=dt) * 2 - 1
c = torch.empty(sum(m * n for m, n, k in sizes), device="cuda", dtype=dt)
specs, off, coff = [], 0, 0
for m, n, k in sizes:
    specs.append(dict(order=G.RowMajor, transA=G.NoTrans, transB=G.NoTrans, m=m, n=n, k=k, alpha=1.0, beta=0.0,
                      A=ab.data_ptr() + off * esz, lda=k, B=ab.data_ptr() + (off + m * k) * esz, ldb=n,
                      C=c.data_ptr() + coff * esz, ldc=n))
    off += m * k + k * n
    coff += m * n
probs = G.problems(specs)
default = G.GroupedPlan(probs, elem_bytes=esz)
G.grouped_autotune(esz, 1)
tuned = G.GroupedPlan(probs, elem_bytes=esz)
s = torch.cuda.Stream()


def ms(plan):
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(s)
    for _ in range(3):
        plan.run(stream=s.cuda_stream)
    e1.record(s)
    e1.synchronize()
    return e0.elapsed_time(e1) / 3


torch.cuda.synchronize()
t = [(ms(default), ms(tuned)) for _ in range(8)][1:]
print("default %.4f tuned %.4f" % (min(a for a, _ in t), min(b for _, b in t)))
"""


@pytest.mark.parametrize("esz", [8, 4])
def test_autotuned_shapes_are_not_slower(esz):
    r = subprocess.run([sys.executable, "-c", CHILD, str(esz)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    w = r.stdout.split()
    default, tuned = float(w[1]), float(w[3])
    # the tuner keeps the default unless another choice is 1 % faster on a batch of this distribution
    assert tuned <= 1.03 * default, (default, tuned)
