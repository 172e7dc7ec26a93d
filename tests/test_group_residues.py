"""The tensor-core epilogue's residues (residue2 in split_gemm.cu), evaluated exactly: for an FP32
integer x, q = rint(x inv) with inv = 1 / p rounded to FP32 and r = x - p q.  Next to every half
multiple of p, where the estimate comes closest to the wrong multiple, |r| <= (p + 1) / 2 for
|x| <= 2^24 (a drain group's sum) and |r| <= p / 2 for |x| < 2^23 (a sum of residues), and what the
epilogue stores, r + p, stays inside the range the reconstruction's reduction takes."""
import importlib.util
import os
import struct

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _gen():
    spec = importlib.util.spec_from_file_location("crt_tables_gen", os.path.join(ROOT, "blaze_gb300", "csrc", "crt_tables.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def _residues(x, p):
    """r of every integer in x, the quotient rounded once to the nearest integer, ties to even."""
    inv = struct.unpack("<f", struct.pack("<f", 1.0 / p))[0]
    m, e = np.frexp(np.float64(inv))
    mant, shift = int(m * (1 << 24)), 24 - int(e)
    num = x * mant
    half = np.int64(1) << (shift - 1)
    fl = num >> shift
    rem = num - (fl << shift)
    q = fl + ((rem > half) | ((rem == half) & (fl % 2 == 1))).astype(np.int64)
    assert np.all(np.abs(q) < 1 << 22)  # the 1.5 * 2^23 form of rint
    return x - p * q


@pytest.mark.parametrize("p", _gen().MODULI)
@pytest.mark.parametrize("limit,slack", [(1 << 24, 1), ((1 << 23) - 1, 0)])
def test_residue_magnitude(p, limit, slack):
    k = np.arange(-(limit // p) - 1, limit // p + 1, dtype=np.int64)
    x = np.unique(np.concatenate([k * p + o for o in (p // 2 - 1, p // 2, p // 2 + 1, p // 2 + 2)]))
    x = np.concatenate([x[np.abs(x) <= limit], [-limit, limit, 0]])
    r = _residues(x, p)
    assert np.all((r - x) % p == 0)
    assert np.all(np.abs(r) <= (p + slack) // 2)
    assert np.all(np.abs(p * ((x - r) // p)) < 1 << 25)  # p q is exact inside the multiply-add


@pytest.mark.parametrize("n", list(range(2, 16)))
def test_stored_residues_reduce(n):
    """x = c_p A + c_q B for the largest stored residues, and its 32-bit Barrett reduction."""
    for s in _gen().table(n)["sups"]:
        cp, cq = s["p"] + (s["p"] + 1) // 2, (s["q"] + (s["q"] + 1) // 2) if s["ib"] >= 0 else 0
        x = cp * s["A"] + cq * s["B"]
        assert x < 1 << 26
        for v in (x, x - x % s["Ps"], x - x % s["Ps"] - 1):
            u = v - ((v * s["Psinv32"]) >> 32) * s["Ps"]
            assert 0 <= u < 2 * s["Ps"]
