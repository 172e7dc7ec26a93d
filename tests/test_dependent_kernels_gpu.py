"""Kernels that start under the one ahead of them read its results only after it has finished: products
of one shape follow one another with other row and column exponents and other plans each time, so that
an exponent or a plan of the product before would show.  Every entry is rounded to at least 40 bits
(float: 17) of its row's or column's largest value, which bounds the error by k 2^-39 (k 2^-16) of
their product; 2^-36 (2^-14) is checked."""
import numpy as np
import pytest

import blaze_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,slices", [("split_crt", 0), ("split", 6), ("float", 0)])
@pytest.mark.parametrize("m,n,k", [(2048, 512, 256), (300, 200, 130), (4100, 1500, 520)])
def test_products_in_a_row(m, n, k, method, slices):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    dtype = np.float32 if method == "float" else np.float64
    spread = 15 if method == "float" else 200
    ops = []
    for i in range(4):
        A = rng.uniform(-1, 1, (m, k)) * 2.0 ** rng.integers(-spread, spread + 1, (m, 1))
        B = rng.uniform(-1, 1, (k, n)) * 2.0 ** rng.integers(-spread, spread + 1, (1, n))
        if i == 2:
            A[0, 0] = np.inf  # no stale flag in the next one
        ops.append((A.astype(dtype), B.astype(dtype)))
    dev = [(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()) for a, b in ops]
    out = [torch.empty(m, n, dtype=torch.float32 if method == "float" else torch.float64, device="cuda") for _ in ops]
    torch.cuda.synchronize()
    o = G.opts(method="split" if method == "float" else method, slices=slices)
    gemm = G.sgemm_ex if method == "float" else G.dgemm_ex
    for (a, b), c in zip(dev, out):
        gemm(O.ROW_MAJOR, O.NO_TRANS, O.NO_TRANS, m, n, k, 1.0, a, k, b, n, 0.0, c, n, o)
    for i, ((A, B), c) in enumerate(zip(ops, out)):
        rows = slice(1, None) if i == 2 else slice(None)
        A, B = A[rows].astype(np.float64), B.astype(np.float64)
        scale = k * np.outer(np.abs(A).max(axis=1), np.abs(B).max(axis=0))
        err = np.abs(c.cpu().numpy()[rows] - A @ B) / scale
        assert err.max() <= (2.0 ** -14 if method == "float" else 2.0 ** -36), (i, float(err.max()))
