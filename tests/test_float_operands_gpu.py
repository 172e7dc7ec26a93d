"""Float products whose statistics and slicing read the float operands themselves: rows and columns at
the ends of the float range (zero, subnormal, tiny, huge, one large value among ones), Inf and NaN,
every transposition, leading dimensions of every parity, bases aligned for one element only, C read and
not read.  A 17-bit rounding of both operands meets the float target k 2^-24 on these sizes, which
bounds an entry's error by k 2^-16 of its row's and column's largest values; 2^-14 is checked."""
import numpy as np
import pytest

import blaze_gb300 as G
import oracle as O
from helpers import stored_dims

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [O.ROW_MAJOR, O.COL_MAJOR])
@pytest.mark.parametrize("ta", [O.NO_TRANS, O.TRANS])
@pytest.mark.parametrize("tb", [O.NO_TRANS, O.TRANS])
@pytest.mark.parametrize("m,n,k,pad", [(64, 96, 300, 0), (67, 93, 301, 1), (256, 260, 1030, 2), (33, 40, 64, 4)])
def test_extreme_rows(m, n, k, pad, ta, tb, order):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(7)
    A = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    B = rng.uniform(-1, 1, (k, n)).astype(np.float32)
    A[0] = 0.0
    A[1] = (A[1] * 2.0 ** 20).round() * np.float32(2.0 ** -149)  # subnormal
    A[2] *= np.float32(2.0 ** -110)                              # normal, below the fast range
    A[3] *= np.float32(2.0 ** 100)
    A[4, 7] = np.float32(2.0 ** 90)
    A[5] *= np.float32(2.0 ** -84)                               # at the edge of the fast range
    A[5, ::3] = 0.0
    B[:, 0] = 0.0
    B[:, 1] *= np.float32(2.0 ** -120)
    B[:, 2] *= np.float32(2.0 ** 20)
    beta = 0.0 if ta == tb else 0.5

    def store(L, trans):
        X = L.T if trans == O.TRANS else L
        X = X if order == O.ROW_MAJOR else X.T
        buf = np.full((X.shape[0], X.shape[1] + pad), np.nan, dtype=np.float32)  # the gaps are not read
        buf[:, :X.shape[1]] = X
        return np.concatenate([np.full(1, np.nan, np.float32), buf.ravel()]), X.shape[1] + pad

    bufA, lda = store(A, ta)
    bufB, ldb = store(B, tb)
    rc, cc = stored_dims(order, O.NO_TRANS, m, n)
    C = np.full((rc, cc + pad), 0.25 if beta else np.nan, dtype=np.float32)
    dA, dB, dC = torch.from_numpy(bufA).cuda(), torch.from_numpy(bufB).cuda(), torch.from_numpy(C).cuda()
    o = G.sgemm_ex(order, ta, tb, m, n, k, 1.0, dA[1:], lda, dB[1:], ldb, beta, dC, cc + pad, G.opts(method="split"))
    assert o.method_used == G.METHOD_SPLIT_CRT
    got = dC.cpu().numpy()[:, :cc].astype(np.float64)
    got = got if order == O.ROW_MAJOR else got.T
    ref = A.astype(np.float64) @ B.astype(np.float64) + beta * 0.25
    scale = k * np.outer(np.abs(A).max(axis=1).astype(np.float64), np.abs(B).max(axis=0).astype(np.float64))
    tol = scale * 2.0 ** -14 + np.abs(ref) * 2.0 ** -23 + 2.0 ** -148
    fine = np.abs(ref) < 3e38
    assert np.all(np.abs(got - ref)[fine] <= tol[fine]), float(np.max((np.abs(got - ref) / tol)[fine]))
    assert np.all(got[0] == beta * 0.25) and np.all(got[:, 0] == beta * 0.25)
    if beta == 0.0:
        assert np.count_nonzero(got[1, 2:]) == 0 or np.all(np.abs(got[1, 2:]) < 1e-30)


def test_nonfinite_rows_and_columns():
    torch = pytest.importorskip("torch")
    m, n, k = 130, 260, 300
    A = torch.rand(m, k, device="cuda") - 0.5
    B = torch.rand(k, n, device="cuda") - 0.5
    A[5, 7] = float("inf")
    B[11, 3] = float("nan")
    C = torch.zeros(m, n, device="cuda")
    torch.cuda.synchronize()
    G.sgemm_ex(O.ROW_MAJOR, O.NO_TRANS, O.NO_TRANS, m, n, k, 1.0, A, k, B, n, 0.0, C, n, G.opts(method="split"))
    c = C.cpu().numpy()
    assert np.isnan(c[5]).all() and np.isnan(c[:, 3]).all()
    mask = np.ones((m, n), bool)
    mask[5, :] = False
    mask[:, 3] = False
    assert np.isfinite(c[mask]).all()
