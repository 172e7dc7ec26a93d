"""The plan's norms and scale factors are FP64 sums over the rows: on operands of signed powers of two,
whose squares and row sums are exact in FP32, the reported bound of the residue form
    2^(-beta-1) (rA + rB) + 2^(-2 beta-2) rA rB + 2^-52,   rX = sqrt(k) ||2^e|| / ||X||,
is that of the same sums in numpy to a few roundings (FP32 sums over the rows are off by 1e-8)."""
import math

import numpy as np
import pytest
import torch

import blaze_gb300 as G

pytestmark = pytest.mark.gpu


def _operand(g, rows, k):
    """rows x k, row i with c_i entries +-2^(e_i - 1) and zeros; (X, r) with r = sqrt(k s / n)."""
    e = -g.integers(0, 21, rows)
    c = g.integers(1, k + 1, rows)
    X = np.where(np.arange(k)[None, :] < c[:, None], np.where(g.random((rows, k)) < 0.5, -1.0, 1.0), 0.0)
    X = g.permuted(X, axis=1) * (2.0 ** (e - 1.0))[:, None]
    s, n = math.fsum(4.0 ** e), math.fsum(4.0 ** e * (c / 4.0))
    return X, math.sqrt(k * s / n)


@pytest.mark.parametrize("m,n,k", [(300, 280, 64), (1000, 37, 1300), (33, 2500, 700), (3000, 3100, 520)])
@pytest.mark.parametrize("order", [G.RowMajor, G.ColMajor])
def test_reported_bound_has_fp64_sums(m, n, k, order):
    g = np.random.default_rng(m + n + k)
    A, rA = _operand(g, m, k)
    B, rB = _operand(g, n, k)
    B = B.T
    if order == G.ColMajor:
        a, b, lda, ldb, ldc = A.T.copy(), B.T.copy(), m, k, m
    else:
        a, b, lda, ldb, ldc = A, B.copy(), k, n, n
    # device operands: products of host operands are planned block by block
    a, b = torch.from_numpy(np.ascontiguousarray(a)).cuda(), torch.from_numpy(np.ascontiguousarray(b)).cuda()
    C = torch.empty(m * n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    o = G.dgemm_ex(order, G.NoTrans, G.NoTrans, m, n, k, 1.0, a, lda, b, ldb, 0.0, C, ldc, G.opts(method="split_crt"))
    rel = min(abs((2.0 ** (-t - 1) * (rA + rB) + 2.0 ** (-2 * t - 2) * rA * rB + 2.0 ** -52) / o.error_bound - 1.0)
              for t in range(1, 56))
    # four square roots, quotients and sums of a few thousand terms: some 2^-53 each
    assert rel <= 1e-13, rel
