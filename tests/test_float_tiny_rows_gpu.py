"""Float products of values below 2^-86, where a zero and a subnormal number are no longer told apart by
the statistics' first pass: the same product scaled by powers of two has the same plan, the same bits up
to the scale, and takes about as long."""
import pytest

import blaze_gb300 as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _operands(m, n, k, zeros):
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)
    A = torch.rand(m, k, generator=g, device="cuda") - 0.5
    B = torch.rand(k, n, generator=g, device="cuda") - 0.5
    if zeros:
        A[torch.rand(m, k, generator=g, device="cuda") < 0.4] = 0.0
        A[m // 2] = 0.0
    # no values below 2^-30, so that 2^-90 leaves no subnormal ones
    return A.where(A.abs() > 2.0 ** -25, A * 0), B.where(B.abs() > 2.0 ** -25, B * 0)


def _product(A, B, reps=1):
    m, k = A.shape
    n = B.shape[1]
    C = torch.empty(m, n, device="cuda")
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s = torch.cuda.current_stream()
        e0.record(s)
        o = G.sgemm_ex(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, C, n,
                       G.opts(method="split", residency=G.PTR_DEVICE))
        e1.record(s)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return C, o, best


@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("m,n,k", [(40, 50, 64), (130, 70, 517), (33, 300, 2600)])
def test_scaled_operands_have_the_same_plan_and_result(m, n, k, zeros):
    A, B = _operands(m, n, k, zeros)
    C0, o0, _ = _product(A, B)
    C1, o1, _ = _product(A * 2.0 ** -90, B)
    C2, o2, _ = _product(A * 2.0 ** 40, B * 2.0 ** -90)
    assert o1.error_bound == o0.error_bound and o2.error_bound == o0.error_bound
    assert o1.slices_used == o0.slices_used == o2.slices_used
    assert torch.equal(C1, C0 * 2.0 ** -90) and torch.equal(C2, C0 * 2.0 ** -50)


def test_tiny_values_cost_about_the_same():
    A, B = _operands(2048, 2048, 2048, True)
    plain, tiny = _product(A, B, 20)[2], _product(A * 2.0 ** -90, B * 2.0 ** -90, 20)[2]
    assert tiny < 1.5 * plain, (tiny, plain)
