"""What a user of this framework has it do, as cases that can be timed: the posit32 Rgemm on
device and host buffers, factor-and-solve, batched plans and served solves, each through
the public Python entry points, over the sizes of the benchmark configurations.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw(rng)`` gives
more of the same ranges, ``prepare(case, seed)`` makes what a program holds before the
call, ``run(state)`` is one pass, ``work(case)`` what a pass cannot do without.  Every
output is a posit32 bit pattern (int32 / uint32) or an integer, so it has to be the same
bits whatever the implementation: ``exact`` has nothing to add.
"""
import math
import random

import numpy as np
import torch

import posit_gpu_b200 as pg

ALPHA_MINUS_ONE = pg.P32_MINUS_ONE
HALF = 0x38000000  # 0.5 as posit32


def listed():
    return [
        # the smallest device call: latency and launches (a block of a small factorization)
        {"name": "gemm_tiny", "kind": "gemm", "ta": "N", "tb": "N", "m": 48, "n": 48, "k": 32, "pad": 0,
         "alpha": pg.P32_ONE, "beta": 0, "dist": "uniform"},
        # the drop-in call on host buffers (RgemmG), plain 512^3, alpha 1, beta 0.5
        {"name": "rgemm_host_512", "kind": "host_gemm", "ta": "N", "tb": "N", "m": 512, "n": 512, "k": 512},
        # dot-then-combine order, ragged sizes and padded leading dimensions
        {"name": "gemm_tn_ragged", "kind": "gemm", "ta": "T", "tb": "N", "m": 2049, "n": 1537, "k": 3001, "pad": 5,
         "alpha": ALPHA_MINUS_ONE, "beta": pg.P32_ONE, "dist": "uniform"},
        # magnitudes 10^U(-20, 20): long regimes everywhere
        {"name": "gemm_nt_wide", "kind": "gemm", "ta": "N", "tb": "T", "m": 2048, "n": 2048, "k": 2048, "pad": 0,
         "alpha": ALPHA_MINUS_ONE, "beta": pg.P32_ONE, "dist": "wide"},
        # the headline GEMM
        {"name": "gemm_nn_8192", "kind": "gemm", "ta": "N", "tb": "N", "m": 8192, "n": 8192, "k": 8192, "pad": 0,
         "alpha": ALPHA_MINUS_ONE, "beta": pg.P32_ONE, "dist": "uniform"},
        # the trailing update of a blocked LU of order 8192 at panel width 64
        {"name": "gemm_trailing_64", "kind": "gemm", "ta": "N", "tb": "N", "m": 8128, "n": 8128, "k": 64, "pad": 0,
         "alpha": ALPHA_MINUS_ONE, "beta": pg.P32_ONE, "dist": "uniform"},
        # device-resident factor-and-solve, one right-hand side, small and large
        {"name": "lu_1024", "kind": "lu", "n": 1024, "nrhs": 1, "trans": "N"},
        {"name": "lu_4096", "kind": "lu", "n": 4096, "nrhs": 1, "trans": "N"},
        {"name": "chol_4096", "kind": "chol", "uplo": "L", "n": 4096, "nrhs": 1},
        # a burst of served solves, three in ten on a cached factor
        {"name": "served_40", "kind": "served", "count": 40, "n_lo": 32, "n_hi": 2048},
        # one persistent launch over many uneven problems
        {"name": "batch_solve_2000", "kind": "batch_solve", "count": 2000, "n_lo": 8, "n_hi": 512},
        {"name": "batch_gemm_5000", "kind": "batch_gemm", "count": 5000, "lo": 4, "hi": 512},
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["gemm", "gemm", "gemm", "host_gemm", "lu", "lu", "chol", "chol", "served", "batch_solve",
                       "batch_gemm"])
    if kind == "gemm":
        dist = "wide" if rng.random() < 0.25 else "uniform"
        most = 2 ** 31 if dist == "wide" else 2 ** 36
        while True:
            m, n, k = (_logu(rng, 4, 8192) for _ in range(3))
            if m * n * k <= most:
                break
        alpha, beta = rng.choice([(pg.P32_ONE, 0), (ALPHA_MINUS_ONE, pg.P32_ONE), (pg.P32_ONE, HALF)])
        return {"kind": kind, "ta": rng.choice("NT"), "tb": rng.choice("NT"), "m": m, "n": n, "k": k,
                "pad": rng.choice([0, 0, 1, 7]), "alpha": alpha, "beta": beta, "dist": dist}
    if kind == "host_gemm":
        return {"kind": kind, "ta": rng.choice("NT"), "tb": rng.choice("NT"), "m": _logu(rng, 32, 1024),
                "n": _logu(rng, 32, 1024), "k": _logu(rng, 32, 1024)}
    if kind == "lu":
        trans = rng.choice(["N", "N", "N", "T"])
        return {"kind": kind, "n": _logu(rng, 64, 1024 if trans == "T" else 4096), "nrhs": rng.randint(1, 16),
                "trans": trans}
    if kind == "chol":
        uplo = rng.choice(["L", "L", "U"])
        return {"kind": kind, "uplo": uplo, "n": _logu(rng, 64, 1024 if uplo == "U" else 4096),
                "nrhs": rng.randint(1, 16)}
    if kind == "served":
        return {"kind": kind, "count": rng.randint(8, 40), "n_lo": 32, "n_hi": _logu(rng, 256, 2048)}
    if kind == "batch_solve":
        return {"kind": kind, "count": _logu(rng, 200, 2000), "n_lo": 8, "n_hi": _logu(rng, 64, 512)}
    return {"kind": "batch_gemm", "count": _logu(rng, 500, 5000), "lo": 4, "hi": _logu(rng, 64, 512)}


# --------------------------------------------------------------------------------------
# Inputs: entries uniform in [-1, 1] (or magnitudes 10^U(-20, 20)) in FP64, converted to
# posit32 on the device; Cholesky matrices are M M^T / n + I
# --------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _fp64(g, numel, dist="uniform"):
    u = torch.rand(numel, dtype=torch.float64, device="cuda", generator=g)
    if dist == "uniform":
        return u * 2.0 - 1.0
    sign = torch.rand(numel, dtype=torch.float64, device="cuda", generator=g)
    mag = torch.pow(10.0, u * 40.0 - 20.0)
    return torch.where(sign < 0.5, -mag, mag)


def _system(g, kind, n, nrhs):
    """(matrix, right-hand sides) as flat column-major patterns; b = A x, x uniform."""
    M = _fp64(g, n * n).view(n, n)
    if kind == "chol":
        M = torch.addmm(torch.eye(n, dtype=torch.float64, device="cuda"), M, M.t(), alpha=1.0 / n)
        M = torch.tril(M) + torch.tril(M, -1).t()  # exactly symmetric
    A = pg.from_double_dev(M.t().contiguous().view(-1))  # column-major
    x = _fp64(g, n * nrhs).view(nrhs, n)
    B = pg.from_double_dev((x @ M.t()).contiguous().view(-1))
    return A, B


def _sizes(case, seed):
    rng = random.Random(17)  # the mix of sizes belongs to the case, the values to the seed
    return [_logu(rng, case["n_lo"], case["n_hi"]) for _ in range(case["count"])]


def _prepare_gemm(c, seed):
    g = _gen(seed)
    ra, ca = (c["m"], c["k"]) if c["ta"] == "N" else (c["k"], c["m"])
    rb, cb = (c["k"], c["n"]) if c["tb"] == "N" else (c["n"], c["k"])
    lda, ldb, ldc = ra + c["pad"], rb + c["pad"], c["m"] + c["pad"]
    A = pg.from_double_dev(_fp64(g, lda * ca, c["dist"]))
    B = pg.from_double_dev(_fp64(g, ldb * cb, c["dist"]))
    C0 = pg.from_double_dev(_fp64(g, ldc * c["n"], c["dist"]))
    return {"c": c, "A": A, "lda": lda, "B": B, "ldb": ldb, "C0": C0, "C": C0.clone(), "ldc": ldc}


def _run_gemm(s):
    c = s["c"]
    if c["beta"] != 0:  # the call updates C in place: start from the same C each pass
        s["C"].copy_(s["C0"])
    pg.Rgemm_dev(c["ta"], c["tb"], c["m"], c["n"], c["k"], c["alpha"], s["A"], s["lda"], s["B"], s["ldb"], c["beta"],
                 s["C"], s["ldc"])
    return s["C"]


def _prepare_host_gemm(c, seed):
    g = _gen(seed)
    m, n, k = c["m"], c["n"], c["k"]
    host = [pg.from_double_dev(_fp64(g, numel)).cpu().numpy().view(np.uint32) for numel in (m * k, k * n, m * n)]
    return {"c": c, "A": host[0], "B": host[1], "C": host[2], "lda": m if c["ta"] == "N" else k,
            "ldb": k if c["tb"] == "N" else n}


def _run_host_gemm(s):
    c = s["c"]
    pg.Rgemm(c["ta"], c["tb"], c["m"], c["n"], c["k"], pg.P32_ONE, s["A"], s["lda"], s["B"], s["ldb"], HALF, s["C"],
             c["m"])
    return s["C"]


def _prepare_factor(c, seed):
    n = c["n"]
    A, B = _system(_gen(seed), c["kind"], n, c["nrhs"])
    return {"c": c, "A": A, "B": B, "F": torch.empty_like(A), "X": torch.empty_like(B),
            "ipiv": torch.zeros(n, dtype=torch.int32, device="cuda"),
            "info": torch.zeros(1, dtype=torch.int32, device="cuda")}


def _run_factor(s):
    c, n = s["c"], s["c"]["n"]
    s["F"].copy_(s["A"])  # the factorization is in place; the matrix is kept for residuals
    s["X"].copy_(s["B"])
    if c["kind"] == "lu":
        pg.Rgetrf_dev(n, n, s["F"], n, s["ipiv"], s["info"])
        pg.Rgetrs_dev(c["trans"], n, c["nrhs"], s["F"], n, s["ipiv"], s["X"], n)
        return {"factor": s["F"], "ipiv": s["ipiv"], "info": s["info"], "x": s["X"]}
    pg.Rpotrf_dev(c["uplo"], n, s["F"], n, s["info"])
    pg.Rpotrs_dev(c["uplo"], n, c["nrhs"], s["F"], n, s["X"], n)
    return {"factor": s["F"], "info": s["info"], "x": s["X"]}


def _pinned(t):
    return t.cpu().pin_memory()


def _prepare_served(c, seed):
    """Fresh matrices, and every third or so request on a factor that the server already
    holds (its matrix was solved with before)."""
    g, rng = _gen(seed), random.Random(23)
    srv = pg.Server()
    reqs, warm = [], []
    for i, n in enumerate(_sizes(c, seed)):
        kind, nrhs = ("lu", "chol")[i % 2], rng.randint(1, 16)
        A, B = _system(g, kind, n, nrhs)
        A, B = _pinned(A), _pinned(B)
        X = torch.empty_like(B).pin_memory()
        code = pg.SOLVE_LU if kind == "lu" else pg.SOLVE_CHOLESKY
        if i % 10 in (2, 5, 9):
            warm.append(srv.submit(code, n, nrhs, A, B, X, matrix_id=i))
            reqs.append((code, n, nrhs, None, B, X, i))
        else:
            reqs.append((code, n, nrhs, A, B, X, -1))
    for t in warm:
        srv.wait(t)
    return {"srv": srv, "reqs": reqs}


def _run_served(s):
    srv = s["srv"]
    tickets = [srv.submit(code, n, nrhs, A, B, X, matrix_id=mid) for code, n, nrhs, A, B, X, mid in s["reqs"]]
    res = [srv.wait(t) for t in tickets]
    return {"x": [q[5] for q in s["reqs"]], "status": np.array([r["status"] for r in res], np.int32),
            "info": np.array([r["info"] for r in res], np.int32)}


def _prepare_batch_solve(c, seed):
    g = _gen(seed)
    sizes = _sizes(c, seed)
    A0 = torch.empty(sum(n * n for n in sizes), dtype=torch.int32, device="cuda")
    B0 = torch.empty(sum(sizes), dtype=torch.int32, device="cuda")
    A, B = torch.empty_like(A0), torch.empty_like(B0)
    ipiv = torch.zeros(sum(sizes), dtype=torch.int32, device="cuda")
    info = torch.zeros(len(sizes), dtype=torch.int32, device="cuda")
    probs, oa, ob = [], 0, 0
    for i, n in enumerate(sizes):
        kind = ("lu", "chol")[i % 2]
        a, b = _system(g, kind, n, 1)
        A0[oa:oa + n * n].copy_(a)
        B0[ob:ob + n].copy_(b)
        probs.append((pg.BATCH_LU if kind == "lu" else pg.BATCH_CHOLESKY, A[oa:oa + n * n], B[ob:ob + n],
                      ipiv[ob:ob + n], info[i:i + 1]))
        oa, ob = oa + n * n, ob + n
    return {"plan": pg.BatchPlan(probs), "A0": A0, "B0": B0, "A": A, "B": B, "ipiv": ipiv, "info": info}


def _run_batch_solve(s):
    s["A"].copy_(s["A0"])
    s["B"].copy_(s["B0"])
    s["plan"].launch()
    return {"factors": s["A"], "x": s["B"], "ipiv": s["ipiv"], "info": s["info"]}


def _gemm_shapes(c):
    rng = random.Random(29)
    return [(rng.choice("NT"), rng.choice("NT")) + tuple(_logu(rng, c["lo"], c["hi"]) for _ in range(3))
            for _ in range(c["count"])]


def _prepare_batch_gemm(c, seed):
    g = _gen(seed)
    shapes = _gemm_shapes(c)
    A, B, C = (pg.from_double_dev(_fp64(g, total)) for total in (sum(m * k for _, _, m, _, k in shapes),
                                                                   sum(k * n for _, _, _, n, k in shapes),
                                                                   sum(m * n for _, _, m, n, _ in shapes)))
    W = torch.empty_like(C)
    probs, oa, ob, oc = [], 0, 0, 0
    for ta, tb, m, n, k in shapes:
        probs.append((ta, tb, m, n, k, ALPHA_MINUS_ONE, A[oa:oa + m * k], m if ta == "N" else k, B[ob:ob + k * n],
                      k if tb == "N" else n, pg.P32_ONE, W[oc:oc + m * n], m))
        oa, ob, oc = oa + m * k, ob + k * n, oc + m * n
    return {"plan": pg.BatchGemmPlan(probs), "A": A, "B": B, "C0": C, "C": W}


def _run_batch_gemm(s):
    s["C"].copy_(s["C0"])
    s["plan"].launch()
    return s["C"]


_PREPARE = {"gemm": _prepare_gemm, "host_gemm": _prepare_host_gemm, "lu": _prepare_factor, "chol": _prepare_factor,
            "served": _prepare_served, "batch_solve": _prepare_batch_solve, "batch_gemm": _prepare_batch_gemm}
_RUN = {"gemm": _run_gemm, "host_gemm": _run_host_gemm, "lu": _run_factor, "chol": _run_factor,
        "served": _run_served, "batch_solve": _run_batch_solve, "batch_gemm": _run_batch_gemm}


def prepare(case, seed):
    """What a program holds before the call: operands, plan or server, and output buffers."""
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    """One pass through the public entry points; the outputs it returns are whole."""
    return _RUN[state["kind"]](state)


def exact(case, seed):
    """Every output is a bit pattern or an index: there is no value in 64 bits to be near."""
    return None


def _factor_work(kind, n, nrhs):
    flops = (2.0 / 3.0 if kind == "lu" else 1.0 / 3.0) * n ** 3 + 2.0 * n * n * nrhs
    return {"bytes": 8.0 * n * n + 8.0 * n * nrhs, "flops": flops}


def work(case):
    """A posit multiply and a posit add count as one operation each."""
    k = case["kind"]
    if k in ("gemm", "host_gemm"):
        m, n, kk = case["m"], case["n"], case["k"]
        reads_c = 0 if case.get("beta", HALF) == 0 else 1
        return {"bytes": 4.0 * (m * kk + kk * n + (1 + reads_c) * m * n), "flops": 2.0 * m * n * kk}
    if k in ("lu", "chol"):
        return _factor_work(k, case["n"], case["nrhs"])
    if k == "batch_gemm":
        shapes = _gemm_shapes(case)
        return {"bytes": sum(4.0 * (m * q + q * n + 2 * m * n) for _, _, m, n, q in shapes),
                "flops": sum(2.0 * m * n * q for _, _, m, n, q in shapes)}
    rng = random.Random(23)
    total = {"bytes": 0.0, "flops": 0.0}
    for i, n in enumerate(_sizes(case, 0)):
        kind = ("lu", "chol")[i % 2]
        nrhs = rng.randint(1, 16) if k == "served" else 1
        w = _factor_work(kind, n, nrhs)
        if k == "served" and i % 10 in (2, 5, 9):  # cached factor: the solve only
            w = {"bytes": 4.0 * n * n + 8.0 * n * nrhs, "flops": 2.0 * n * n * nrhs}
        total = {q: total[q] + w[q] for q in total}
    return total
