"""Grouped products at the sizes where their tiles can go wrong: one row or column, the edges of the
tile sizes and of the staged k chunks, every transposition, with and without C read.  Each output
against a 64-bit product within the classical bound of a dot product in any order, k u |A||B|."""
import numpy as np
import pytest

import blaze_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

SIDES = [1, 2, 5, 8, 15, 16, 17, 31, 32, 33, 49, 65]
DEPTHS = [1, 3, 15, 16, 17, 32, 33, 70]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_grouped_tile_edges(dtype):
    torch = pytest.importorskip("torch")
    u = 2.0 ** -53 if dtype == np.float64 else 2.0 ** -24
    shapes = [(m, n, DEPTHS[(i * 5 + j * 3) % len(DEPTHS)]) for i, m in enumerate(SIDES) for j, n in enumerate(SIDES)]
    shapes += [(m, 20, k) for m in (7, 40) for k in DEPTHS]
    A = O.uniform(sum((m + 3) * (k + 3) for m, n, k in shapes), 1, dtype=dtype)
    B = O.uniform(sum((k + 3) * (n + 3) for m, n, k in shapes), 2, dtype=dtype)
    C = O.uniform(sum((m + 3) * (n + 3) for m, n, k in shapes), 3, dtype=dtype)
    dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C))
    torch.cuda.synchronize()
    specs, refs, oa, ob, oc, e = [], [], 0, 0, 0, dA.element_size()
    for q, (m, n, k) in enumerate(shapes):
        ta, tb = q % 2, (q // 2) % 2
        ra, ca, rb, cb = (k, m) if ta else (m, k), None, (n, k) if tb else (k, n), None
        (ra, ca), (rb, cb) = ra, rb
        pad = q % 4  # leading dimensions of every parity
        alpha, beta = ((1.0, 0.0), (-1.5, 0.5))[q % 3 == 2]
        specs.append(dict(order=O.ROW_MAJOR, transA=O.TRANS if ta else O.NO_TRANS, transB=O.TRANS if tb else O.NO_TRANS,
                          m=m, n=n, k=k, alpha=alpha, beta=beta, A=dA.data_ptr() + oa * e, lda=ca + pad,
                          B=dB.data_ptr() + ob * e, ldb=cb + pad, C=dC.data_ptr() + oc * e, ldc=n + pad))
        a = A[oa:oa + ra * (ca + pad)].reshape(ra, ca + pad)[:, :ca].astype(np.float64)
        b = B[ob:ob + rb * (cb + pad)].reshape(rb, cb + pad)[:, :cb].astype(np.float64)
        a, b = (a.T if ta else a), (b.T if tb else b)
        c = C[oc:oc + m * (n + pad)].reshape(m, n + pad)
        refs.append((oc, m, n, pad, alpha * (a @ b) + beta * c[:, :n].astype(np.float64),
                     2 * (k + 4) * u * (abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(c[:, :n].astype(np.float64))),
                     c[:, n:].copy()))
        oa += (m + 3) * (k + 3); ob += (k + 3) * (n + 3); oc += (m + 3) * (n + 3)
    (G.dgemm_grouped if dtype == np.float64 else G.sgemm_grouped)(G.problems(specs))
    out = dC.cpu().numpy()
    for sp, (oc, m, n, pad, ref, tol, gap) in zip(specs, refs):
        got = out[oc:oc + m * (n + pad)].reshape(m, n + pad)
        assert np.all(np.abs(got[:, :n].astype(np.float64) - ref) <= tol), (m, n, sp["k"], sp["transA"], sp["transB"])
        assert np.array_equal(got[:, n:], gap)
