"""The tensor-core epilogue's residues (residue2 in split_gemm.cu), evaluated exactly: for an FP32
integer x, q = rint(x inv) with inv = 1 / p rounded to FP32 and r = x - p q.  Next to every half
multiple of p, where the estimate comes closest to the wrong multiple, |r| <= (p + 1) / 2 for
|x| <= 2^24 (a drain group's sum) and |r| <= p / 2 for |x| < 2^23 (a sum of residues).  The
reconstruction gives back every integer of the plan's range from the bytes r + 128 that the epilogue
stores."""
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


def _replay(t, residues, gen):
    """The reconstruction of one output from its stored bytes r + 128 (crt_cols): x = b_p A + b_q B + K,
    W - round(estimate) P modulo 2^(32 limbs)."""
    from fractions import Fraction
    f32 = np.float32
    fq = f32(0)
    W = 0
    for s in t["sups"]:
        x = residues[s["ia"]] * s["A"] + s["K"] + (residues[s["ib"]] * s["B"] if s["ib"] >= 0 else 0)
        assert 0 <= x < 1 << 26
        # x rounded to FP32, then one rounding of x finv + fq: a double holds the product's 48 bits, and
        # the sum's error stays far below half an FP32 unit except at ties, which do not matter here
        fq = f32(float(f32(x)) * float(f32(1.0 / s["Ps"])) + float(fq))
        W += x * (t["P"] // s["Ps"])
        assert all(x * ((t["P"] // s["Ps"] >> 32 * l) & 0xFFFFFFFF) < 1 << 58 for l in range(4))
    assert 0 <= fq < 1 << 14
    assert abs(Fraction(float(fq)) - Fraction(W, t["P"])) < Fraction(1, 100)  # the half integers are 0.029 away
    q = int(round(Fraction(float(fq))))
    mod = 1 << (32 * t["limbs"])
    w = (W + q * t["negP"]) % mod
    return w - mod if w >= mod // 2 else w


@pytest.mark.parametrize("n", list(range(2, 16)))
def test_reconstruction_from_stored_bytes(n):
    import random
    gen = _gen()
    t = gen.table(n)
    lim = t["P"] * 1000 // 2125  # |T| < P / 2.125
    rng = random.Random(n)
    cases = [0, 1, -1, lim - 1, 1 - lim] + [rng.randrange(1 - lim, lim) for _ in range(400)]
    for T in cases:
        res = []
        for p in gen.MODULI[:n]:
            r = T % p
            r = r - p if r > p // 2 else r  # symmetric
            assert 0 <= r + 128 <= (256 if p == 257 else 255) or p == 256
            res.append((r + 128) % 256 if p != 257 else r + 128)
        assert _replay(t, res, gen) == T, (n, T)
