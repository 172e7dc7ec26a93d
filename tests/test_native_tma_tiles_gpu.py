"""The native kernel's 16384-output tiles (128 x 128, 256 x 64, 64 x 256; operands through TMA), which
native_plan picks where they fill the chip or split a long k: every tile width, with and without a split,
every transposition, both types, ragged sizes, against float64 products; and the allocation-free entry
point with a product that does use its scratch.  That the plan picks these tiles for these sizes (on 152
SMs) is checked on the host, with the plan compiled from the source."""
import os
import shutil
import subprocess

import pytest

import blaze_gb300 as G

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMS = 152

# element bytes, m, n, k, tile columns, k splits (row-major logical sizes)
SHAPES = [
    (8, 253, 55, 40001, 64, 152), (8, 115, 113, 40001, 128, 152), (8, 55, 253, 40001, 256, 152),
    (8, 38900, 59, 131, 64, 1), (8, 371, 19259, 67, 128, 1), (8, 59, 38900, 131, 256, 1),
    (4, 229, 43, 40001, 64, 78), (4, 69, 161, 40001, 128, 76), (4, 43, 229, 40001, 256, 78),
    (4, 38900, 59, 131, 64, 1), (4, 1021, 1531, 203, 128, 1), (4, 59, 38900, 131, 256, 1),
]
# allocation-free products whose split sums fill most of the 16 MiB scratch, and their tiles (0: the large ones)
NOALLOC = [(240, 224, 12000, 16, 38), (464, 48, 20000, 16, 76), (48, 464, 20000, 16, 76), (114, 114, 40000, 0, 152)]

HOST = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
struct NativePlan { int tile = 0, splits = 1; };
"""
MAIN = r"""
int main(int argc, char** argv) {
    for (int i = 1; i + 3 < argc; i += 4) {
        const long e = atol(argv[i]), m = atol(argv[i + 1]), n = atol(argv[i + 2]), k = atol(argv[i + 3]);
        const NativePlan p = native_plan(m, n, k, int(e), 152, false);
        std::printf("%d %d %d %d\n", p.tile, native_tile_n(m, n), p.splits, native_choose_splits(m, n, k, int(e), 152));
    }
}
"""


@pytest.fixture(scope="module")
def host_plan(tmp_path_factory):
    """Plans of (element bytes, m, n, k): (small tile or 0, large tiles' columns, splits, large tiles' splits)."""
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    with open(os.path.join(ROOT, "blaze_gb300", "csrc", "native_gemm.cu")) as f:
        src = f.read()
    line = lambda start: src[src.index(start):src.index("\n", src.index(start)) + 1]  # noqa: E731
    plan = src[src.index("int native_choose_splits("):src.index("template <typename T>\ncudaError_t native_gemm(const Gemm& g, const NativePlan& plan")]
    d = tmp_path_factory.mktemp("plan")
    (d / "p.cpp").write_text(HOST + line("constexpr int PANEL_BYTES") + line("int native_tile_n(") + plan + MAIN)
    subprocess.run([gxx, "-std=c++17", "-o", str(d / "p"), str(d / "p.cpp")], check=True)

    def run(cases):
        out = subprocess.run([str(d / "p"), *[str(x) for c in cases for x in c[:4]]], check=True, capture_output=True, text=True)
        return [tuple(int(x) for x in l.split()) for l in out.stdout.splitlines()]

    return run


def test_the_plan_picks_these_tiles(host_plan):
    cases = SHAPES + [(8, *c) for c in NOALLOC]
    tiles = [(0, c[4], c[5]) for c in SHAPES] + [(c[3], None, c[4]) for c in NOALLOC]
    got = [p[:3] for p in host_plan(cases)]
    assert [(a, b if w[1] else None, c) for (a, b, c), w in zip(got, tiles)] == tiles


def test_small_tiles_sum_no_longer_chains(host_plan):
    # a plan in small tiles splits k at least as far as the large tiles do for the same product
    cases = [(e, m, n, k) for e in (8, 4) for m in (1, 60, 100, 512, 1024, 4096) for n in (1, 48, 64, 200, 512, 4096)
             for k in (100, 600, 1600, 6000, 8192, 20003, 100000)]
    for case, (tile, _, splits, large) in zip(cases, host_plan(cases)):
        assert splits >= large, (case, tile, splits, large)


def _stored(torch, x, trans, pad):
    """x (or its transpose) in row-major storage with `pad` extra NaN elements a row."""
    x = x.T if trans else x
    buf = torch.full((x.shape[0], x.shape[1] + pad), float("nan"), dtype=x.dtype, device="cuda")
    buf[:, :x.shape[1]] = x
    return buf


@pytest.mark.gpu
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
@pytest.mark.parametrize("elem,m,n,k,bn,splits", SHAPES)
def test_every_tile_width_and_transposition(elem, m, n, k, bn, splits, ta, tb):
    torch = pytest.importorskip("torch")
    assert G.device_info()[0] == SMS
    dt = torch.float64 if elem == 8 else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)
    A = torch.rand(m, k, generator=g, device="cuda", dtype=dt) * 2 - 1
    B = torch.rand(k, n, generator=g, device="cuda", dtype=dt) * 2 - 1
    C0 = torch.rand(m, n, generator=g, device="cuda", dtype=dt)
    alpha, beta, pad = (1.0, 0.0, 0) if ta == tb else (-0.75, 0.5, 3)
    a, b, c = _stored(torch, A, ta, pad), _stored(torch, B, tb, pad), _stored(torch, C0, False, pad)
    torch.cuda.synchronize()
    call = G.dgemm_ex if elem == 8 else G.sgemm_ex
    o = call(G.RowMajor, G.Trans if ta else G.NoTrans, G.Trans if tb else G.NoTrans, m, n, k, alpha, a, a.shape[1], b,
             b.shape[1], beta, c, c.shape[1], G.opts(method="native"))
    assert o.method_used == G.METHOD_NATIVE
    ref = alpha * (A.double() @ B.double()) + beta * C0.double()
    # the worst-case bound of a chain of k multiply-adds and the update, normwise
    u = 2.0 ** (-53 if elem == 8 else -24)
    err = float((c[:, :n].double() - ref).norm())
    bound = (k + 4) * u * (abs(alpha) * float(A.double().norm()) * float(B.double().norm()) + float(C0.double().norm()))
    assert err <= bound, (err, bound)
    assert pad == 0 or bool(c[:, n:].isnan().all())


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,tile,splits", NOALLOC)
def test_noalloc_products_that_use_the_scratch(m, n, k, tile, splits):
    torch = pytest.importorskip("torch")
    assert G.device_info()[0] == SMS
    assert splits * m * n * 8 <= (16 << 20) - 256
    g = torch.Generator(device="cuda")
    for seed in range(2):  # another product's sums are in the scratch the second time
        g.manual_seed(seed)
        A = torch.rand(m, k, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        B = torch.rand(k, n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        c1 = torch.zeros(m, n, device="cuda", dtype=torch.float64)
        c2 = torch.zeros(m, n, device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        st = G.lib().gb300_dgemm_native_noalloc(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A.data_ptr(), k,
                                                B.data_ptr(), n, 0.0, c1.data_ptr(), n, None)
        assert st == G.OK, G.last_error()
        G.dgemm_ex(G.RowMajor, G.NoTrans, G.NoTrans, m, n, k, 1.0, A, k, B, n, 0.0, c2, n, G.opts(method="native"))
        assert torch.equal(c1, c2)  # the same plan
        err = float((c1 - A @ B).norm())
        assert err <= 2 * k * 2.0 ** -53 * float(A.norm()) * float(B.norm())


def test_float_products_of_full_large_tiles_stay_in_them(host_plan):
    # sizes that a 32-wide tile's rate of 40 multiply-adds a clock gave to the small tiles, which took longer
    cases = [(4, 1024, 256, 2048), (4, 512, 512, 2048), (4, 1024, 512, 1024), (4, 1024, 1024, 512)]
    assert [p[0] for p in host_plan(cases)] == [0] * len(cases)
    # and sizes whose small tiles are faster
    cases = [(4, 512, 512, 512), (4, 768, 768, 768), (4, 300, 300, 2000), (4, 2000, 100, 1500), (4, 256, 256, 256)]
    assert all(p[0] != 0 for p in host_plan(cases))
