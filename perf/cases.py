"""Workloads whose speed is tracked: what a program that uses this library has it do, through the
public entry points, from the smallest products to the largest.

    listed()            the cases with names
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the operands and plans a program holds before the call
    run(state)          one pass
    work(case)          the bytes and operations a pass cannot do without
    exact(case, seed)   the same results from plain torch in 64 bits

Operands are device-resident unless the case says host.  Every product is C = alpha A B + beta C
with uniform [-1, 1] entries, as the repository's own benchmark and Blaze's tests draw them.
"""
import math
import random

import numpy as np
import torch

import blaze_gb300 as G

UPPER, LOWER, NON_UNIT, UNIT, LEFT, RIGHT = 121, 122, 131, 132, 141, 142


def listed():
    return [
        # one small product of two DynamicMatrix<double> of a few dozen rows: latency is everything
        dict(name="dgemm_small", kind="dgemm", m=96, n=80, k=112, order="R", ta=False, tb=False, beta=0.0, pad=0),
        # ragged sizes and odd leading dimensions, B transposed (a row-major times a column-major
        # matrix), some hundred rows
        dict(name="dgemm_ragged", kind="dgemm", m=403, n=517, k=389, order="R", ta=False, tb=True, beta=0.0, pad=0),
        # the 1024^3 product of the plain configuration
        dict(name="dgemm_1024", kind="dgemm", m=1024, n=1024, k=1024, order="R", ta=False, tb=False, beta=0.0, pad=0),
        # the 8192^3 product of the headline configuration
        dict(name="dgemm_8192", kind="dgemm", m=8192, n=8192, k=8192, order="R", ta=False, tb=False, beta=0.0, pad=0),
        # a tall, skinny product with short k and column-major operands (the rectangular configuration)
        dict(name="dgemm_tall", kind="dgemm", m=65536, n=256, k=256, order="C", ta=False, tb=False, beta=0.0, pad=0),
        # the call Blaze itself makes: operands in pageable host memory
        dict(name="dgemm_host", kind="dgemm_host", m=3000, n=2000, k=2500, order="R", ta=False, tb=False),
        # DynamicMatrix<float>
        dict(name="sgemm_2048", kind="sgemm", m=2048, n=2048, k=2048, order="R", ta=False, tb=False, beta=0.0, pad=0),
        # DynamicMatrix<complex<double>>
        dict(name="zgemm_1024", kind="zgemm", m=1024, n=1024, k=1024, order="R", ta=False, tb=False, beta=0.0, pad=0),
        # a triangular solve with as many right-hand sides as rows
        dict(name="dtrsm_2048", kind="dtrsm", m=2048, n=2048, order="R", side="L", lower=True, ta=False, unit=False),
        # ten thousand uneven StaticMatrix / HybridMatrix products in one plan, double and float
        dict(name="grouped_f64", kind="grouped", count=10000, dtype="d", shapes=7),
        dict(name="grouped_f32", kind="grouped", count=10000, dtype="s", shapes=7),
        # matrix x vector
        dict(name="dgemv_8192", kind="dgemv", m=8192, n=8192, order="R", ta=False),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["dgemm", "dgemm", "dgemm", "tall", "dgemm_host", "sgemm", "zgemm", "dtrsm", "grouped", "dgemv"])
    order, ta, tb = rng.choice("RC"), rng.random() < 0.3, rng.random() < 0.4
    if kind == "tall":
        return dict(kind="dgemm", m=_logint(rng, 16384, 65536), n=_logint(rng, 64, 512), k=_logint(rng, 64, 512),
                    order=order, ta=ta, tb=tb, beta=0.0, pad=rng.choice([0, 2]))
    if kind in ("dgemm", "sgemm", "zgemm"):
        lo, hi = {"dgemm": (48, 8192), "sgemm": (64, 4096), "zgemm": (64, 2048)}[kind]
        mid = math.sqrt(lo * hi)
        s = _logint(rng, lo, hi)  # a size, and three dimensions around it
        lo1, hi1 = max(lo, int(s / 2 if s > mid else s / 1.5)), min(hi, int(s * 1.5))
        return dict(kind=kind, m=_logint(rng, lo1, hi1), n=_logint(rng, lo1, hi1), k=_logint(rng, lo1, hi1), order=order,
                    ta=ta, tb=tb, beta=rng.choice([0.0, 0.0, 1.0]), pad=rng.choice([0, 0, 1, 8]))
    if kind == "dgemm_host":
        return dict(kind=kind, m=_logint(rng, 256, 4096), n=_logint(rng, 256, 4096), k=_logint(rng, 256, 4096),
                    order=order, ta=ta, tb=tb)
    if kind == "dtrsm":
        return dict(kind=kind, m=_logint(rng, 256, 4096), n=_logint(rng, 256, 4096), order=order, side=rng.choice("LR"),
                    lower=rng.random() < 0.5, ta=ta, unit=rng.random() < 0.3)
    if kind == "grouped":
        return dict(kind=kind, count=_logint(rng, 500, 10000), dtype=rng.choice("ds"), shapes=rng.randrange(1, 1 << 30))
    return dict(kind="dgemv", m=_logint(rng, 1024, 16384), n=_logint(rng, 1024, 16384), order=order, ta=ta)


DTYPE = {"dgemm": torch.float64, "sgemm": torch.float32, "zgemm": torch.complex128}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, rows, cols, dtype=torch.float64, pad=0):
    """rows x cols uniform [-1, 1] entries in row-major storage with `pad` extra elements a row."""
    real = torch.float32 if dtype == torch.float32 else torch.float64
    w = 2 if dtype.is_complex else 1
    x = torch.rand(rows, (cols + pad) * w, generator=g, device="cuda", dtype=real).mul_(2).sub_(1)
    return torch.view_as_complex(x.view(rows, cols + pad, 2)) if dtype.is_complex else x


def _stored(rows, cols, order, trans):
    """Row-major shape of the buffer that holds op(X) = rows x cols."""
    return (rows, cols) if (order == "R") != trans else (cols, rows)


def _operands(case, seed):
    g = _generator(seed)
    dt = DTYPE.get(case["kind"], torch.float64)
    m, n, k, order, pad = case["m"], case["n"], case["k"], case["order"], case.get("pad", 0)
    a = _uniform(g, *_stored(m, k, order, case["ta"]), dt, pad)
    b = _uniform(g, *_stored(k, n, order, case["tb"]), dt, pad)
    c = _uniform(g, *_stored(m, n, order, False), dt, pad)
    return a, b, c


def _problem_sizes(case):
    """The (m, n, k) of a batch: log-uniform integers in [4, 256]."""
    r = random.Random(case["shapes"])
    return [tuple(_logint(r, 4, 256) for _ in range(3)) for _ in range(case["count"])]


def _batch(case, seed):
    sizes = _problem_sizes(case)
    total = sum(m * k + k * n for m, n, k in sizes)
    dt = torch.float64 if case["dtype"] == "d" else torch.float32
    ab = _uniform(_generator(seed), 1, total, dt).view(-1)
    return sizes, ab, dt


def _triangle(case, seed):
    """A well-conditioned triangular matrix (off-diagonal u / size, diagonal 1 + u / 2) and B."""
    g = _generator(seed)
    m, n, order = case["m"], case["n"], case["order"]
    ka = m if case["side"] == "L" else n
    a = _uniform(g, ka, ka) / ka
    d = torch.diagonal(a)
    d.mul_(ka / 2).add_(1)
    b = _uniform(g, *_stored(m, n, order, False))
    return a, b


def prepare(case, seed):
    kind = case["kind"]
    order = G.RowMajor if case.get("order", "R") == "R" else G.ColMajor
    tr = lambda t: G.Trans if t else G.NoTrans  # noqa: E731
    s = dict(case=case, kind=kind, order=order)
    if kind in DTYPE or kind == "dgemm_host":
        a, b, c = _operands(case, seed)
        if kind == "dgemm_host":
            a, b, c = a.cpu().numpy(), b.cpu().numpy(), np.zeros(tuple(c.shape))
        s.update(a=a, b=b, c0=c, c=c, ta=tr(case["ta"]), tb=tr(case["tb"]), lda=a.shape[1], ldb=b.shape[1], ldc=c.shape[1])
        if case.get("beta"):
            s["c"] = c.clone()
    elif kind == "dtrsm":
        a, b = _triangle(case, seed)
        s.update(a=a, b=b, x=b.clone(), ta=tr(case["ta"]))
    elif kind == "grouped":
        sizes, ab, dt = _batch(case, seed)
        c = torch.empty(sum(m * n for m, n, _ in sizes), dtype=dt, device="cuda")
        specs, off, coff, e = [], 0, 0, ab.element_size()
        for m, n, k in sizes:
            specs.append(dict(order=G.RowMajor, transA=G.NoTrans, transB=G.NoTrans, m=m, n=n, k=k, alpha=1.0, beta=0.0,
                              A=ab.data_ptr() + off * e, lda=k, B=ab.data_ptr() + (off + m * k) * e, ldb=n,
                              C=c.data_ptr() + coff * e, ldc=n))
            off += m * k + k * n
            coff += m * n
        s.update(ab=ab, c=c, plan=G.GroupedPlan(G.problems(specs), elem_bytes=e))
    else:  # dgemv
        g = _generator(seed)
        m, n = case["m"], case["n"]
        a = _uniform(g, *_stored(m, n, case["order"], False))
        s.update(a=a, x=_uniform(g, 1, m if case["ta"] else n), y=torch.empty(n if case["ta"] else m, dtype=torch.float64, device="cuda"),
                 ta=tr(case["ta"]))
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind in DTYPE or kind == "dgemm_host":
        beta = case.get("beta", 0.0)
        if beta:  # the matrix that the product is added to is the program's own and new in each pass
            s["c"].copy_(s["c0"])
            torch.cuda.current_stream().synchronize()
        call = {"sgemm": G.cblas_sgemm, "zgemm": G.cblas_zgemm}.get(kind, G.cblas_dgemm)
        call(s["order"], s["ta"], s["tb"], case["m"], case["n"], case["k"], 1.0, s["a"], s["lda"], s["b"], s["ldb"], beta,
             s["c"], s["ldc"])
        rows, cols = _stored(case["m"], case["n"], case["order"], False)
        return s["c"][:rows, :cols]
    if kind == "dtrsm":
        # the solve overwrites its right-hand sides: a program that keeps them copies them first
        s["x"].copy_(s["b"])
        torch.cuda.current_stream().synchronize()
        G.cblas_trsm(s["order"], LEFT if case["side"] == "L" else RIGHT, LOWER if case["lower"] else UPPER, s["ta"],
                     UNIT if case["unit"] else NON_UNIT, case["m"], case["n"], 1.0, s["a"], s["a"].shape[1], s["x"],
                     s["x"].shape[1])
        return s["x"]
    if kind == "grouped":
        s["plan"].run()
        return s["c"]
    G.cblas_gemv(s["order"], s["ta"], case["m"], case["n"], 1.0, s["a"], s["a"].shape[1], s["x"], 1, 0.0, s["y"], 1)
    return s["y"]


def work(case):
    kind = case["kind"]
    if kind in DTYPE or kind == "dgemm_host":
        m, n, k = case["m"], case["n"], case["k"]
        e = {"sgemm": 4, "zgemm": 16}.get(kind, 8)
        c = 2 if case.get("beta") else 1
        return {"bytes": e * (m * k + k * n + c * m * n), "flops": (8 if kind == "zgemm" else 2) * m * n * k}
    if kind == "dtrsm":
        m, n = case["m"], case["n"]
        ka = m if case["side"] == "L" else n
        return {"bytes": 8 * (ka * (ka + 1) // 2 + 2 * m * n), "flops": ka * m * n}
    if kind == "grouped":
        sizes = _problem_sizes(case)
        e = 8 if case["dtype"] == "d" else 4
        return {"bytes": e * sum(m * k + k * n + m * n for m, n, k in sizes), "flops": 2 * sum(m * n * k for m, n, k in sizes)}
    return {"bytes": 8 * (case["m"] * case["n"] + case["m"] + case["n"]), "flops": 2 * case["m"] * case["n"]}


def exact(case, seed):
    kind = case["kind"]
    if kind in DTYPE or kind == "dgemm_host":
        a, b, c = _operands(case, seed)
        m, n, k = case["m"], case["n"], case["k"]
        flip = case["order"] == "C"
        wide = lambda x: x if x.is_complex() else x.double()  # noqa: E731
        ra, ca = _stored(m, k, case["order"], case["ta"])
        rb, cb = _stored(k, n, case["order"], case["tb"])
        a, b = wide(a)[:, :ca], wide(b)[:, :cb]
        a = a.T if case["ta"] != flip else a  # m x k
        b = b.T if case["tb"] != flip else b  # k x n
        r = a @ b
        if case.get("beta"):
            r = r + case["beta"] * (wide(c)[:, :m].T if flip else wide(c)[:, :n])
        r = r.T if flip else r
        return r.cpu().numpy() if kind == "dgemm_host" else r
    if kind == "dtrsm":
        a, b = _triangle(case, seed)
        flip = case["order"] == "C"
        a, b = (a.T, b.T) if flip else (a, b)
        t = torch.tril(a) if case["lower"] else torch.triu(a)
        if case["unit"]:
            t = t - torch.diag(torch.diagonal(t)) + torch.eye(t.shape[0], dtype=t.dtype, device=t.device)
        t, upper = (t.T, case["lower"]) if case["ta"] else (t, not case["lower"])
        x = torch.linalg.solve_triangular(t, b, upper=upper, left=case["side"] == "L")
        return x.T if flip else x
    if kind == "grouped":
        sizes, ab, _ = _batch(case, seed)
        ab, out, off = ab.double(), [], 0
        for m, n, k in sizes:
            out.append((ab[off:off + m * k].view(m, k) @ ab[off + m * k:off + m * k + k * n].view(k, n)).view(-1))
            off += m * k + k * n
        return torch.cat(out)
    g = _generator(seed)
    a = _uniform(g, *_stored(case["m"], case["n"], case["order"], False))
    x = _uniform(g, 1, case["m"] if case["ta"] else case["n"]).view(-1)
    a = a.T if case["order"] == "C" else a
    return a.T @ x if case["ta"] else a @ x
