"""The reconstruction's conversion of a two's-complement integer to a double (words_to_double in
split_gemm.cu), compiled from the source with host forms of its intrinsics, against Python's
integers: rounding to nearest even for both signs at every length the residue plans use, with the
runs of ones whose rounding carries into the next power of two."""
import ctypes as ct
import functools
import importlib.util
import math
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "blaze_gb300", "csrc")

HOST = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
using std::max;
using std::min;
#define __device__
#define __noinline__
#define __forceinline__ inline
constexpr int kNonFinite = 0x7fff;
static double __longlong_as_double(long long x) { double d; std::memcpy(&d, &x, 8); return d; }
static uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, int s) { s &= 31; return s ? (hi << s) | (lo >> (32 - s)) : hi; }
static int __clz(int x) { return x ? __builtin_clz(unsigned(x)) : 32; }
static double __hiloint2double(int hi, int lo) {
    return __longlong_as_double((long long)((uint64_t(uint32_t(hi)) << 32) | uint32_t(lo)));
}
"""


@functools.lru_cache(maxsize=1)
def _tables():
    spec = importlib.util.spec_from_file_location("crt_tables_gen", os.path.join(CSRC, "crt_tables.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return {n: (mod.table(n)["limbs"], mod.table(n)["bits"]) for n in range(2, 16)}


@pytest.fixture(scope="module")
def convert(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    with open(os.path.join(CSRC, "split_gemm.cu")) as f:
        src = f.read()
    body = src[src.index("template <int LB>\n__device__ __noinline__ double words_to_double_any"):
               src.index("// Residue (CRT) reconstruction of four consecutive outputs")]
    cases = "".join(f"case {n}: return words_to_double<{lb}, {bits}>(w, ei, fj, scale);\n"
                    for n, (lb, bits) in _tables().items())
    d = tmp_path_factory.mktemp("wtd")
    (d / "w.cpp").write_text(HOST + body + 'extern "C" double conv(int n, const uint32_t* p, int ei, int fj, int scale) {\n'
                             "    const uint32_t w[4] = {p[0], p[1], p[2], p[3]};\n    switch (n) {\n" + cases +
                             "    }\n    return -1.0;\n}\n")
    so = str(d / "w.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-o", so, str(d / "w.cpp")], check=True)
    lib = ct.CDLL(so)
    lib.conv.restype = ct.c_double
    lib.conv.argtypes = [ct.c_int, ct.POINTER(ct.c_uint32), ct.c_int, ct.c_int, ct.c_int]

    def call(n, W, ei=0, fj=0, scale=0):
        limbs = _tables()[n][0]
        u = W % (1 << (32 * limbs))
        return lib.conv(n, (ct.c_uint32 * 4)(*[(u >> (32 * i)) & 0xffffffff for i in range(4)]), ei, fj, scale)

    return call


def _integers(bits, seed):
    """Magnitudes of up to bits - 1 bits: runs of ones, ties, powers of two and their neighbours."""
    r = random.Random(seed)
    out = {0, 1, 2, 3}
    for p in range(1, bits):
        for low in (0, 1, p - 55, p - 54, p - 53, p - 52, p // 2):
            if 0 <= low < p:
                out |= {(1 << p) - (1 << low), (1 << p) - (1 << low) - 1, (1 << p) - (1 << low) + 1}
        out.add((1 << (p - 1)) + (r.getrandbits(p - 1) if p > 1 else 0))
        if p > 54:  # halfway between two doubles, the lower one odd or even
            m = (1 << 52) | r.getrandbits(52)
            out |= {((m << 1) | 1) << (p - 54), (((m | 1) << 1) | 1) << (p - 54), ((1 << 54) - 1) << (p - 54)}
    return [x for x in out if 0 <= x < 1 << (bits - 1)]


def _ldexp(x, e):
    try:
        return math.ldexp(x, e)
    except OverflowError:
        return math.copysign(math.inf, x)


@pytest.mark.parametrize("n", list(range(2, 16)))
def test_rounds_to_nearest_even(convert, n):
    for x in _integers(_tables()[n][1], n):
        for W in (x, -x):
            for ei, fj, scale in ((0, 0, 0), (7, -30, 60)):
                assert convert(n, W, ei, fj, scale) == _ldexp(float(W), ei + fj - scale), (n, W, ei, fj, scale)


@pytest.mark.parametrize("n", [2, 5, 9, 13, 15])
def test_ends_of_the_exponent_range(convert, n):
    for x in _integers(_tables()[n][1], 100 + n)[::7]:
        if not x:
            continue
        top = x.bit_length()
        for W in (x, -x):
            for e in (1022 - top, 1023 - top, 1024 - top, 1025 - top, -1020 - top, -1021 - top, -1022 - top, -1040 - top, -1080 - top):
                assert convert(n, W, e, 0, 0) == _ldexp(float(W), e), (n, W, e)


def test_rows_or_columns_with_inf_or_nan_give_nan(convert):
    for ei, fj in ((0x7fff, 0), (0, 0x7fff), (0x7fff, -1073), (-1073, 0x7fff), (0x7fff, 0x7fff)):
        assert math.isnan(convert(12, 5 << 70, ei, fj, 100)) and math.isnan(convert(12, 0, ei, fj, 100))


@pytest.mark.gpu
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_products_just_below_a_power_of_two(single, sign):
    # row i of A is s_i (1, -2^-(27 + i % 3), 0 ...), column j of B is t_j (1, 2^-(27 + j % 3), 0 ...):
    # the exact s_i t_j (1 - 2^-54 or closer) rounds to the power of two s_i t_j
    import numpy as np

    import blaze_gb300 as G

    m, n, k = 130, 140, 300
    dt = np.float32 if single else np.float64
    i, j = np.arange(m), np.arange(n)
    s, t = 2.0 ** (i % 21 - 10), 2.0 ** (j % 17 - 8)
    A, B, C = np.zeros((m, k), dt), np.zeros((k, n), dt), np.zeros((m, n), dt)
    A[:, 0], A[:, 1] = sign * s, -sign * s * 2.0 ** -(27.0 + i % 3)
    B[0], B[1] = t, t * 2.0 ** -(27.0 + j % 3)
    (G.sgemm_ex if single else G.dgemm_ex)(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, C, n,
                                           G.opts(method="split", target_error=1e-14))
    assert np.array_equal(C, (sign * np.outer(s, t)).astype(dt))
