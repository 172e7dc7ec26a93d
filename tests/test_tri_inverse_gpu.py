"""The inverses of a triangular solve's diagonal blocks, built from 16 x 16 blocks by doubling: sizes
at the edges of the base blocks, of every level and of the 512-row leaf, both triangles, transposed,
conjugated, unit.  Well-conditioned triangles, so each solve's residual stays within a few times the
classical n u |A||X| (u = 2^-53 or 2^-24), in the Frobenius norm."""
import numpy as np
import pytest

import blaze_gb300 as G
import oracle as O

pytestmark = pytest.mark.gpu

NO_TRANS, TRANS, CONJ = 111, 112, 113


@pytest.mark.parametrize("dtype", ["d", "s", "z"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 63, 65, 129, 257, 511, 513, 700])
def test_solve_sizes(n, dtype):
    torch = pytest.importorskip("torch")
    t = {"d": np.float64, "s": np.float32, "z": np.complex128}[dtype]
    u = 2.0 ** -24 if dtype == "s" else 2.0 ** -53
    nr = 9
    w = 2 if dtype == "z" else 1
    for lower in (True, False):
        for ta, unit in ((NO_TRANS, False), (TRANS, True), (CONJ if dtype == "z" else NO_TRANS, False)):
            A = O.uniform(n * n * w, 3).view(t if w == 2 else np.float64).reshape(n, n).astype(t) / n
            A[np.diag_indices(n)] = 1 + A[np.diag_indices(n)] * (n / 2)
            B = O.uniform(n * nr * w, 4).view(t if w == 2 else np.float64).reshape(n, nr).astype(t)
            full = A.copy()
            full[np.triu_indices(n, 1) if lower else np.tril_indices(n, -1)] = np.nan  # not read
            if unit:
                full[np.diag_indices(n)] = np.nan
            dA, dB = torch.from_numpy(full).cuda(), torch.from_numpy(B).cuda()
            torch.cuda.synchronize()
            G.cblas_trsm(101, 141, 122 if lower else 121, ta, 132 if unit else 131, n, nr, 1.0, dA, n, dB, nr, dtype=dtype)
            X = dB.cpu().numpy()
            T = np.tril(A) if lower else np.triu(A)
            if unit:
                T[np.diag_indices(n)] = 1
            T = T if ta == NO_TRANS else T.T if ta == TRANS else T.conj().T
            wide = np.complex128 if dtype == "z" else np.float64
            res = np.linalg.norm(T.astype(wide) @ X.astype(wide) - B)
            assert res <= 8 * (n + 8) * u * np.linalg.norm(T) * np.linalg.norm(X), (lower, ta, unit, res)
