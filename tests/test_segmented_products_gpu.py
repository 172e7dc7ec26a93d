"""Products whose k is split into segments (at most half the chip's CTA pairs would have a tile): the
reconstruction adds up the segments' residues.  The results are exact on integer operands for every
remainder of the four columns a thread takes, and a product in two segments takes no longer than one of
half as many outputs more, whose tiles need no segments."""
import pytest

import blaze_gb300 as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("m,n,k", [(64, 61, 20000), (300, 262, 9000), (513, 515, 8192), (1135, 1557, 1766), (1, 3, 60000)])
@pytest.mark.parametrize("beta", [0.0, 1.0])
def test_integer_products_are_exact(m, n, k, beta, dt):
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)
    A = torch.randint(-8, 9, (m, k), generator=g, device="cuda").to(dt)
    B = torch.randint(-8, 9, (n, k), generator=g, device="cuda").to(dt)
    C = torch.randint(-99, 99, (m, n), generator=g, device="cuda").to(dt)
    ref = A.double() @ B.double().T + beta * C.double()  # below 2^24: exact in every form
    torch.cuda.synchronize()
    call = G.dgemm_ex if dt == torch.float64 else G.sgemm_ex
    o = call(G.RowMajor, G.NoTrans, G.Trans, m, n, k, 1.0, A, k, B, k, beta, C, n, G.opts(method="split"))
    assert o.method_used == G.METHOD_SPLIT_CRT
    assert torch.equal(C.double(), ref)


def test_two_segments_cost_no_more_than_a_larger_product():
    def best(m, n, k):
        A, B = torch.rand(m, k, device="cuda", dtype=torch.float64), torch.rand(k, n, device="cuda", dtype=torch.float64)
        C = torch.empty(m, n, device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        ts = []
        for _ in range(60):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            G.dgemm_ex(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, C, n,
                       G.opts(method="split", residency=G.PTR_DEVICE))
            e1.record()
            e1.synchronize()
            ts.append(e0.elapsed_time(e1))
        return min(ts)

    # 5 x 7 pair tiles in two segments; 6 x 8 pair tiles in one
    two, one = best(1135, 1557, 1766), best(1400, 1800, 1766)
    assert two < 1.2 * one, (two, one)  # 1.4 while each column added up its own bytes
