"""A solve keeps the method that it began with while another thread changes the default: a leaf product
that is written into its own right-hand sides is never handed to the native kernel, which reads as it
writes."""
import threading

import pytest

import blaze_gb300 as G

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [141, 142])
def test_solve_while_the_default_method_changes(side):
    ka, other = 2048, 320
    g = torch.Generator(device="cuda")
    g.manual_seed(side)
    A = (torch.rand(ka, ka, generator=g, device="cuda", dtype=torch.float64) - 0.5) / ka
    A.diagonal().add_(1.0)
    T = torch.tril(A)
    m, n = (ka, other) if side == 141 else (other, ka)
    X = torch.rand(m, n, generator=g, device="cuda", dtype=torch.float64) - 0.5
    B = T @ X if side == 141 else X @ T
    prev = G.lib().gb300_set_default_method(G.METHOD_AUTO)
    stop = threading.Event()

    def flip():
        L, i = G.lib(), 0
        while not stop.is_set():
            L.gb300_set_default_method(G.METHOD_NATIVE if i & 1 else G.METHOD_AUTO)
            i += 1

    th = threading.Thread(target=flip)
    th.start()
    try:
        worst = 0.0
        for _ in range(150):
            Y = B.clone()
            torch.cuda.synchronize()
            G.cblas_trsm(G.RowMajor, side, 122, G.NoTrans, 131, m, n, 1.0, A, ka, Y, n)
            worst = max(worst, float((Y - X).abs().max()))
    finally:
        stop.set()
        th.join()
        G.lib().gb300_set_default_method(prev)
    # a well-conditioned triangle (diagonal near 1, off-diagonal rows of norm 0.01): a few k 2^-53
    assert worst < 1e-11, worst
