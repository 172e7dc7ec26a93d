"""The residue reconstruction of four outputs (crt_cols in split_gemm.cu), compiled from the source with
host forms of its intrinsics: for every modulus count N = 2..15 it returns every integer T with
|T| < P / 2.125 (the range that the plan guarantees) rounded to nearest even, from the residue bytes the
tensor-core kernel stores (r + 128, 16 bits for 257), at both ends of that range, next to multiples of
P / P_s, with residues one past the symmetric range where the store allows them, and with k in segments."""
import ctypes as ct
import importlib.util
import os
import random
import shutil
import subprocess
from fractions import Fraction

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
#define __host__
#define __noinline__
#define __forceinline__ inline
#define fmaf std::fmaf
constexpr int kNonFinite = 0x7fff;
constexpr uint32_t MAGIC_BITS = 0x4B400000u;
constexpr float MAGIC = 12582912.0f;
struct uint2 { uint32_t x, y; };
static double __longlong_as_double(long long x) { double d; std::memcpy(&d, &x, 8); return d; }
static uint32_t __float_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, int s) { s &= 31; return s ? (hi << s) | (lo >> (32 - s)) : hi; }
static int __clz(int x) { return x ? __builtin_clz(unsigned(x)) : 32; }
static double __hiloint2double(int hi, int lo) {
    return __longlong_as_double((long long)((uint64_t(uint32_t(hi)) << 32) | uint32_t(lo)));
}
static float __uint2float_rn(uint32_t x) { return float(x); }
static uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
    const uint64_t v = (uint64_t(b) << 32) | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= uint32_t((v >> (8 * ((s >> (4 * i)) & 7))) & 0xff) << (8 * i);
    return r;
}
static uint32_t dp2a(uint32_t a, uint32_t b, uint32_t c, int sh) {
    return c + (a & 0xffff) * ((b >> sh) & 0xff) + (a >> 16) * ((b >> (sh + 8)) & 0xff);
}
static uint32_t __dp2a_lo(uint32_t a, uint32_t b, uint32_t c) { return dp2a(a, b, c, 0); }
static uint32_t __dp2a_hi(uint32_t a, uint32_t b, uint32_t c) { return dp2a(a, b, c, 16); }
"""


def _gen():
    spec = importlib.util.spec_from_file_location("crt_tables_gen", os.path.join(CSRC, "crt_tables.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.fixture(scope="module")
def cols(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    with open(os.path.join(CSRC, "split_gemm.cu")) as f:
        src = f.read()

    def part(start, end):
        return src[src.index(start):src.index(end, src.index(start))]

    body = (part("__device__ __forceinline__ uint32_t mod_small(", "// A modulus' constants") +
            part("__host__ __device__ __forceinline__ int64_t crt_plane(", "// With k in segments") +
            part("// With k in segments: ", "// The double W 2^(x)") +
            part("template <int LB>\n__device__ __noinline__ double words_to_double_any", "// Residue (CRT) reconstruction of four") +
            part("template <int N>\n__device__ __forceinline__ void crt_cols(", "template <typename TC>\nstruct CrtCombine"))
    cases = "".join(f"case {n}: crt_cols<{n}>(crt_load<{n}>(res, S, 0, 0), res, S, 0, nseg, levels, scale, 0, fj, v); break;\n"
                    for n in range(2, 16))
    d = tmp_path_factory.mktemp("crt")
    (d / "c.cpp").write_text(HOST + '#include "crt_tables.h"\nusing namespace gb;\n' + body +
                             'extern "C" void cols(int n, const uint8_t* res, int64_t S, int nseg, int levels, int scale, double* out) {\n'
                             "    const int fj[4] = {0, 0, 0, 0};\n    double v[4] = {0, 0, 0, 0};\n    switch (n) {\n" + cases +
                             "    }\n    std::memcpy(out, v, sizeof(v));\n}\n")
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-shared", "-fPIC", "-o", str(d / "c.so"),
                    str(d / "c.cpp")], check=True)
    lib = ct.CDLL(str(d / "c.so"))
    lib.cols.argtypes = [ct.c_int, ct.c_char_p, ct.c_int64, ct.c_int, ct.c_int, ct.c_int, ct.c_void_p]

    def call(n, residues, nseg=1):
        """residues[segment][modulus][column], integers congruent to r, stored as the kernel stores them."""
        S = 16  # elements a plane: 4 columns used
        buf = bytearray(nseg * (n + 1) * S)
        for g in range(nseg):
            base = g * (n + 1) * S
            for t in range(n):
                for c in range(4):
                    b = residues[g][t][c] + 128
                    if t == 0:
                        buf[base + 2 * c:base + 2 * c + 2] = int(b).to_bytes(2, "little")
                    else:
                        buf[base + (t + 1) * S + c] = b & 0xff
        out = (ct.c_double * 4)()
        lib.cols(n, bytes(buf), S, nseg, n, 0, out)
        return list(out)

    return call


def _sym(x, p):
    r = x % p
    return r - p if r > p // 2 else r


@pytest.mark.parametrize("n", list(range(2, 16)))
def test_every_integer_of_the_range(cols, n):
    g = _gen()
    mods = g.MODULI[:n]
    P = g.table(n)["P"]
    lim = int(Fraction(P) * 1000 / 2125)
    r = random.Random(n)
    ts = [0, 1, -1, lim, -lim, lim - 1, 1 - lim, lim // 2, -(lim // 3)]
    for s in g.table(n)["sups"]:  # next to the multiples that the quotient estimate tells apart
        q = P // s["Ps"]
        ts += [min(lim, k * q) for k in (1, 2, s["Ps"] // 3)] + [max(-lim, -k * q + 1) for k in (1, 5, s["Ps"] // 3)]
    for p in range(1, lim.bit_length()):
        ts += [(1 << p) - 1, 1 - (1 << p), (1 << p) - (1 << (p // 2))]
    ts += [r.randrange(-lim, lim + 1) for _ in range(400)]
    ts = [t for t in ts if abs(t) <= lim]
    ts += [0] * (-len(ts) % 4)
    for i in range(0, len(ts), 4):
        four = ts[i:i + 4]
        got = cols(n, [[[_sym(t, p) for t in four] for p in mods]])
        assert got == [float(t) for t in four], (n, four)


@pytest.mark.parametrize("n", [3, 8, 12, 15])
def test_single_group_residues_one_past_the_symmetric_range(cols, n):
    g = _gen()
    mods = g.MODULI[:n]
    lim = int(Fraction(g.table(n)["P"]) * 1000 / 2125)
    r = random.Random(50 + n)
    for _ in range(100):
        four = [r.randrange(-lim, lim + 1) for _ in range(4)]
        res = []
        for t, p in enumerate(mods):
            row = [_sym(x, p) for x in four]
            if t not in (0, 2):  # 257 and 255 are reduced again before they are stored
                row = [v - p if v == p // 2 and p % 2 else v + p if v == -(p // 2) else v for v in row]
            res.append(row)
        assert cols(n, [res]) == [float(t) for t in four]


@pytest.mark.parametrize("nseg", [2, 3, 38, 76, 254, 255, 256, 700])
@pytest.mark.parametrize("n", [2, 5, 12, 13, 15])
def test_segments(cols, n, nseg):
    g = _gen()
    mods = g.MODULI[:n]
    lim = int(Fraction(g.table(n)["P"]) * 1000 / 2125)
    r = random.Random(n * 100 + nseg)
    for _ in range(20):
        four = [r.randrange(-lim, lim + 1) for _ in range(4)]
        parts = [[r.randrange(-lim, lim + 1) // nseg for _ in range(4)] for _ in range(nseg - 1)]
        parts.append([t - sum(p[c] for p in parts) for c, t in enumerate(four)])
        res = [[[_sym(x, p) for x in part] for p in mods] for part in parts]
        assert cols(n, res, nseg) == [float(t) for t in four]
