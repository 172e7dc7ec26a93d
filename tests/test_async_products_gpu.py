"""Products queued on the caller's stream without a wait between them: each one's planes, exponents,
counters and level planes are the previous one's, whose kernels (dependent launches) and second stream
may still be at work.  Different operands with different row exponents in every product, shapes on
either side of the two-part rule (152 pair tiles of 256 x 256), double, float and the digit form; the
results are those of the same calls made one at a time.  The same for products replayed from a captured
graph with new operands."""
import pytest

import blaze_gb300 as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(3000, 3500, 300), (403, 517, 389), (256, 8200, 200), (3900, 2700, 1100), (130, 70, 2000), (3000, 3500, 300)]


def _operands(i, m, n, k, dt):
    g = torch.Generator(device="cuda")
    g.manual_seed(100 + i)
    A = torch.rand(m, k, generator=g, device="cuda", dtype=dt) - 0.5
    B = torch.rand(k, n, generator=g, device="cuda", dtype=dt) - 0.5
    # row and column exponents that differ from product to product
    A *= torch.pow(2.0, torch.randint(-20, 20, (m, 1), generator=g, device="cuda").to(dt))
    B *= torch.pow(2.0, torch.randint(-20, 20, (1, n), generator=g, device="cuda").to(dt))
    return A, B


def _call(A, B, C, **kw):
    (m, k), n = A.shape, B.shape[1]
    (G.dgemm_ex if A.dtype == torch.float64 else G.sgemm_ex)(
        G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, C, n, G.opts(residency=G.PTR_DEVICE, **kw))


def _check(A, B, C):
    u = 2.0 ** (-53 if A.dtype == torch.float64 else -24)
    err = float((C.double() - A.double() @ B.double()).norm())
    assert err <= 2 * A.shape[1] * u * float(A.double().norm()) * float(B.double().norm())


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("kw", [dict(method="split"), dict(method="auto"), dict(method="split", slices=8)])
def test_queued_products(dt, kw):
    prods = [_operands(i, *s, dt) for i, s in enumerate(SHAPES)]
    ref = [torch.empty(A.shape[0], B.shape[1], device="cuda", dtype=dt) for A, B in prods]
    torch.cuda.synchronize()
    for (A, B), C in zip(prods, ref):
        _call(A, B, C, **kw)
        _check(A, B, C)
    out = [torch.full_like(c, float("nan")) for c in ref]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        for (A, B), C in zip(prods, out):
            _call(A, B, C, synchronous=False, stream=s.cuda_stream, **kw)
    s.synchronize()
    for c, r in zip(out, ref):
        assert torch.equal(c, r)


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
def test_captured_products(dt):
    # the largest first, so that the buffers do not grow under the capture
    shapes = [SHAPES[3], SHAPES[0], SHAPES[1]]
    bufs = [_operands(0, *s, dt) for s in shapes]
    outs = [torch.zeros(m, n, device="cuda", dtype=dt) for m, n, _ in shapes]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    kw = dict(method="split", synchronous=False, stream=s.cuda_stream)
    for (A, B), C in zip(bufs, outs):
        _call(A, B, C, **kw)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        for (A, B), C in zip(bufs, outs):
            _call(A, B, C, **kw)
    for rep in range(1, 4):
        for (A, B), (m, n, k) in zip(bufs, shapes):
            a, b = _operands(10 * rep + m % 7, m, n, k, dt)
            A.copy_(a)
            B.copy_(b)
        for C in outs:
            C.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for (A, B), C in zip(bufs, outs):
            ref = torch.empty_like(C)
            _call(A, B, ref, method="split")
            _check(A, B, ref)
            assert torch.equal(C, ref)
