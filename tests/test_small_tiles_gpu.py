"""The native kernel's small square tiles: the edges of the 8, 16 and 32 wide tiles and of the 32-deep
k chunks, split k, every storage order and transposition, bases aligned for one element only and odd
leading dimensions, against the CPU restatement of Blaze's kernel.  The tolerance is the classical
bound of a dot product summed in any order, k u |A||B| for each side, elementwise."""
import numpy as np
import pytest

import blaze_gb300 as G
import oracle as O
from helpers import stored_dims

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (8, 8, 32), (9, 7, 33), (16, 17, 31), (5, 200, 64), (65, 1, 129), (96, 80, 112), (33, 31, 2000),
         (250, 130, 65), (160, 304, 97)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("order", [O.ROW_MAJOR, O.COL_MAJOR])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_small_tiles(m, n, k, order, dtype):
    torch = pytest.importorskip("torch")
    u = 2.0 ** -53 if dtype == np.float64 else 2.0 ** -24
    gemm = G.dgemm_ex if dtype == np.float64 else G.sgemm_ex
    for i, (ta, tb) in enumerate([(a, b) for a in (O.NO_TRANS, O.TRANS) for b in (O.NO_TRANS, O.TRANS)]):
        ra, ca = stored_dims(order, ta, m, k)
        rb, cb = stored_dims(order, tb, k, n)
        rc, cc = stored_dims(order, O.NO_TRANS, m, n)
        lda, ldb, ldc = ca + i, cb + 1, cc + (3 if i % 2 else 0)
        alpha, beta = (1.0, 0.0) if i == 0 else (-1.5, 0.5)
        A = O.uniform(1 + ra * lda, 10 + i, dtype=dtype)
        B = O.uniform(1 + rb * ldb, 20 + i, dtype=dtype)
        C = O.uniform(rc * ldc, 30 + i, dtype=dtype)
        if beta == 0.0:
            C[:] = np.nan  # C is not read
        dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C))
        gemm(order, ta, tb, m, n, k, alpha, dA[1:], lda, dB[1:], ldb, beta, dC, ldc, G.opts(method="native"))
        opA = O.logical(order, ta, m, k, np.ascontiguousarray(A[1:]), lda).astype(np.float64)
        opB = O.logical(order, tb, k, n, np.ascontiguousarray(B[1:]), ldb).astype(np.float64)
        C0 = O.logical(order, O.NO_TRANS, m, n, C, ldc).astype(np.float64)
        ref = alpha * (opA @ opB) + (beta * C0 if beta else 0.0)
        got = O.logical(order, O.NO_TRANS, m, n, dC.cpu().numpy(), ldc).astype(np.float64)
        mag = abs(alpha) * (np.abs(opA) @ np.abs(opB)) + (abs(beta) * np.abs(C0) if beta else 0.0)
        assert np.all(np.abs(got - ref) <= 2 * (k + 4) * u * mag), (ta, tb, float(np.max(np.abs(got - ref))))
        if ldc > cc:  # the gap between C's rows keeps its values
            gap = dC.cpu().numpy().reshape(rc, ldc)[:, cc:]
            assert np.array_equal(gap, C.reshape(rc, ldc)[:, cc:], equal_nan=True)
