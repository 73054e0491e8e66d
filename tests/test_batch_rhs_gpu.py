"""Batched problems with many right-hand sides: the places where the threads are dealt out over
rows and right-hand sides -- rows against the team's width (32, 256, 512), right-hand sides one
short of, at and past a team's share, past what fits in shared memory, side by side or one by
one -- on a CTA and, where there are more problems than CTAs, on a warp each; against the oracle
bit for bit.  Which problems go where is checked without a GPU."""
import ctypes

import numpy as np
import pytest

import oracle

# (n, right-hand sides)
SPECS = [(1, 3), (1, 40), (2, 15), (2, 16), (4, 4), (4, 5), (4, 65), (5, 300), (11, 17), (16, 16), (17, 33), (31, 5),
         (32, 4), (32, 15), (32, 16), (32, 70), (33, 5), (33, 8), (33, 150), (64, 17), (85, 9), (128, 21), (129, 5),
         (200, 50), (224, 6), (225, 9), (256, 33), (257, 6), (300, 60), (520, 5)]


def _plan_problems(pg, specs):
    return (pg._BatchProblem * len(specs))(*(pg._BatchProblem(kind, n, n, nrhs, n, None, None, None, None)
                                             for kind, n, nrhs in specs))


def test_routes():
    import posit_gpu_b200 as pg
    fn = pg._lib.posit_batch_plan_routes

    def routes(specs, sms=148):
        out = (ctypes.c_int * len(specs))()
        assert fn(_plan_problems(pg, specs), len(specs), sms, out) == 0
        return list(out)

    assert routes([(0, 225, 1), (0, 224, 1), (1, 33, 300), (0, 32, 15), (1, 0, 1)]) == [0, 1, 1, 2, 2]
    # many right-hand sides: a CTA, while CTAs are not many turns short
    assert routes([(0, 32, 16), (1, 4, 300), (0, 40, 2), (0, 4, 1)]) == [1, 1, 1, 2]
    assert set(routes([(1, 8, 64)] * 888)) == {1}
    assert set(routes([(1, 8, 64)] * 889)) == {2}
    assert routes([(1, 8, 64)] * 889 + [(0, 33, 64), (0, 8, 1)])[-2:] == [1, 2]
    assert set(routes([(1, 8, 64)] * 25, sms=4)) == {2}


def _values(rng, numel, what):
    x = rng.uniform(-1, 1, numel)
    if what == "wide":
        x = np.sign(x) * 10.0 ** rng.uniform(-15, 15, numel)
    u = oracle.from_double(x)
    if what == "special":
        u[rng.integers(0, numel, max(1, numel // 5))] = 0
        u[rng.integers(0, numel, 1 + numel // 50)] = oracle.P32_NAR
    return u


def _matrix(rng, kind, n, what):
    if kind == 1:
        X = rng.uniform(-1, 1, (n, n))
        if what == "wide":  # a graded matrix: entries over many binades
            d = 10.0 ** rng.uniform(-7, 7, n)
            return oracle.from_double(((X @ X.T / n + np.eye(n)) * np.outer(d, d)).reshape(-1))
        return oracle.from_double((X @ X.T / n + np.eye(n)).reshape(-1))
    A = _values(rng, n * n, "wide" if what == "wide" else "uniform")
    if what == "special" and n > 2:
        A.reshape(n, n)[1] = 0  # a singular matrix: zero pivots, quotients by zero
    return A


def _run(pg, rng, specs, what):
    import torch
    keep, probs, want = [], [], []
    for kind, n, nrhs in specs:
        lda, ldb = n, n + 2
        A, B = _matrix(rng, kind, n, what), _values(rng, ldb * nrhs, what)
        F, X, piv = A.copy(), B.copy(), np.zeros(n, np.int32)
        if kind == 0:
            info = oracle.orc.orc_rgetrf(n, n, F, lda, piv, 32)
            oracle.orc.orc_rgetrs(b"N", n, nrhs, F, lda, piv, X, ldb)
        else:
            info = oracle.orc.orc_rpotrf(b"L", n, F, lda, 32)
            if info == 0:
                oracle.orc.orc_rpotrs(b"L", n, nrhs, F, lda, X, ldb)
        want.append((X, info))
        t = [torch.from_numpy(v.view(np.int32).copy()).cuda() for v in (A, B)]
        t += [torch.zeros(n, dtype=torch.int32, device="cuda"), torch.full((1,), -7, dtype=torch.int32, device="cuda")]
        keep.append(t)
        probs.append(pg._BatchProblem(kind, n, lda, nrhs, ldb, *(x.data_ptr() for x in t)))
    h = ctypes.c_void_p()
    assert pg._lib.posit_batch_plan_create((pg._BatchProblem * len(probs))(*probs), len(probs), ctypes.byref(h)) == 0
    assert pg._lib.posit_batch_plan_launch(h, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    pg._lib.posit_batch_plan_destroy(h)
    for spec, (A, B, piv, info), (X, wi) in zip(specs, keep, want):
        assert int(info.item()) == wi, (what, spec)
        assert np.array_equal(B.cpu().numpy().view(np.uint32), X), (what, spec)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("what", ["uniform", "wide", "special"])
def test_many_right_hand_sides(cuda_ok, what, kind):
    import posit_gpu_b200 as pg
    rng = np.random.default_rng(3 + kind)
    _run(pg, rng, [(kind, n, nrhs) for n, nrhs in SPECS if what == "uniform" or n < 200], what)


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["uniform", "special"])
def test_many_problems_with_many_right_hand_sides(cuda_ok, what):
    """More such problems than CTAs take in a few turns: a warp each, whatever fits side by side."""
    import posit_gpu_b200 as pg
    rng = np.random.default_rng(9)
    sizes = [(1, 20), (3, 16), (4, 31), (7, 33), (13, 90), (16, 16), (17, 40), (31, 36), (32, 33), (32, 16)]
    _run(pg, rng, [(q & 1, *sizes[q // 2 % len(sizes)]) for q in range(1000)], what)


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["uniform", "special"])
def test_few_many_right_hand_sides_beside_longer_problems(cuda_ok, what):
    """Where a few problems with many right-hand sides do not bound the launch, it takes the kernels
    with a thread per row; they solve any number all the same."""
    import posit_gpu_b200 as pg
    rng = np.random.default_rng(12)
    _run(pg, rng, [(0, 620, 1), (0, 300, 8), (1, 240, 6), (0, 200, 1), (0, 40, 7), (1, 36, 9), (1, 12, 5), (0, 7, 9)],
         what)
