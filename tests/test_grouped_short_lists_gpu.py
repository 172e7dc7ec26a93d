"""Short grouped lists take smaller tiles than long ones, and their tiles are dealt out over the SMs: a
product has the same result bits alone, in a short list and in a long one, and lists around every change
of the kernel's ticket rule (fewer tiles than warps, between one and three a warp, more) are complete."""
import os
import subprocess
import sys

import numpy as np
import pytest

import blaze_gb300 as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _batch(sizes, dt, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    e = 8 if dt == torch.float64 else 4
    ab = torch.rand(sum(m * k + k * n for m, n, k in sizes), generator=g, device="cuda", dtype=dt) - 0.5
    c = torch.full((sum(m * n for m, n, _ in sizes),), float("nan"), device="cuda", dtype=dt)
    specs, off, coff = [], 0, 0
    for m, n, k in sizes:
        specs.append(dict(order=G.RowMajor, transA=G.NoTrans, transB=G.NoTrans, m=m, n=n, k=k, alpha=1.0, beta=0.0,
                          A=ab.data_ptr() + off * e, lda=k, B=ab.data_ptr() + (off + m * k) * e, ldb=n,
                          C=c.data_ptr() + coff * e, ldc=n))
        off += m * k + k * n
        coff += m * n
    torch.cuda.synchronize()
    plan = G.GroupedPlan(G.problems(specs), elem_bytes=e)
    plan.run()
    G.synchronize()
    return ab, c, plan


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (9, 17, 33), (64, 64, 64), (61, 130, 47), (257, 31, 200)])
def test_same_bits_alone_and_in_lists_of_every_length(m, n, k, dt):
    for count in (1, 3, 28, 150, 400, 1500, 6000):
        if count * m * n * k > 2e9:
            continue
        ab, c, plan = _batch([(m, n, k)] * count, dt, 7)
        per = m * k + k * n
        # every product against float64, the first one bit for bit against itself in the other lists
        A = ab.view(count, per)[:, :m * k].reshape(count, m, k).double()
        B = ab.view(count, per)[:, m * k:].reshape(count, k, n).double()
        got = c.view(count, m, n).double()
        err = float((got - A @ B).norm())
        u = 2.0 ** (-53 if dt == torch.float64 else -24)
        assert err <= k * u * float(A.norm()) * float(B.norm()), count
        # the same operands again, alone: the bits of product 0 and of the last one
        for q in (0, count - 1):
            x = torch.full((m * n,), float("nan"), device="cuda", dtype=dt)
            e = ab.element_size()
            one = G.GroupedPlan(G.problems([dict(order=G.RowMajor, transA=G.NoTrans, transB=G.NoTrans, m=m, n=n, k=k,
                                                 alpha=1.0, beta=0.0, A=ab.data_ptr() + q * per * e, lda=k,
                                                 B=ab.data_ptr() + (q * per + m * k) * e, ldb=n, C=x.data_ptr(),
                                                 ldc=n)]), elem_bytes=e)
            torch.cuda.synchronize()
            one.run()
            G.synchronize()
            assert torch.equal(x, c.view(count, m * n)[q]), (count, q)


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
def test_uneven_lists_around_the_ticket_rule(dt):
    rng = np.random.default_rng(3)
    for count in (7, 60, 120, 240, 300, 450, 600, 1000, 1900, 3700):
        sizes = [tuple(int(v) for v in rng.integers(1, 70, 3)) for _ in range(count)]
        ab, c, _ = _batch(sizes, dt, count)
        off = coff = 0
        worst = 0.0
        u = 2.0 ** (-53 if dt == torch.float64 else -24)
        h, hc = ab.cpu().numpy().astype(np.float64), c.cpu().numpy().astype(np.float64)
        for m, n, k in sizes:
            A, B = h[off:off + m * k].reshape(m, k), h[off + m * k:off + m * k + k * n].reshape(k, n)
            err = np.linalg.norm(hc[coff:coff + m * n].reshape(m, n) - A @ B)
            worst = max(worst, err / (2 * k * u * np.linalg.norm(A) * np.linalg.norm(B)))
            off += m * k + k * n
            coff += m * n
        assert worst <= 1.0, (count, worst)


TILES = """
import sys
import blaze_gb300 as G
esz = int(sys.argv[1])
prob = dict(order=G.RowMajor, transA=G.NoTrans, transB=G.NoTrans, m=64, n=64, k=64, alpha=1.0, beta=0.0, A=256, lda=64,
            B=256, ldb=64, C=256, ldc=64)
tiles = [G.GroupedPlan(G.problems([prob] * n), elem_bytes=esz).info()[0] // n for n in (20, 2000)]  # never run
assert tiles[0] > tiles[1], tiles
"""


@pytest.mark.parametrize("esz", [8, 4])
def test_short_lists_take_smaller_tiles(esz):
    # in a fresh process: a loaded tuning table keeps its shapes, and the table is the process's
    r = subprocess.run([sys.executable, "-c", TILES, str(esz)], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
