"""The batched factor-and-solve at the edges of its forms -- a warp per problem (n <= 32), 256
threads with panels of 16 columns, 512 threads with panels of 32 from 225 rows, narrower
panels beyond 512 -- with few and many right-hand sides, padded leading dimensions, ties,
singular and NaR matrices and values outside the fast window, against the oracle bit for bit."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(rng, kind, n, lda, what):
    if kind == 1:
        X = rng.uniform(-1, 1, (n, n))
        S = X @ X.T / n + np.eye(n)
        if what == "special":
            S[n // 2, n // 2] = -1.0
        M = np.zeros((n, lda))
        M[:, :n] = S
    else:
        M = rng.uniform(-1, 1, (n, lda))
        if what == "ties":
            M = rng.choice([-1.0, 1.0, 0.5, -0.5], (n, lda)) + np.eye(n, lda)
        elif what == "wide":
            M = np.sign(M) * 10.0 ** rng.uniform(-15, 15, (n, lda))
    A = oracle.from_double(M.reshape(-1)).reshape(n, lda)
    if what == "special" and kind == 0:
        A[0] = 0
        A[0, 0] = oracle.P32_NAR
        A[min(2, n - 1)] = 0
    return A.reshape(-1)


@pytest.mark.parametrize("what", ["uniform", "ties", "wide", "special"])
def test_batch_shapes(cuda_ok, what):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(["uniform", "ties", "wide", "special"].index(what))
    specs = [(kind, n, nrhs) for kind in (0, 1) for n, nrhs in
             ((1, 1), (2, 3), (15, 1), (31, 2), (32, 5), (33, 1), (47, 12), (64, 1), (65, 3), (130, 9), (224, 1),
              (225, 2), (257, 17), (290, 1))]
    if what == "uniform":
        specs += [(0, 620, 1), (1, 620, 3), (1, 1100, 1)]
    keep, probs, want = [], [], []
    for kind, n, nrhs in specs:
        lda, ldb = n + 3, n + 1
        A, B = _matrix(rng, kind, n, lda, what), oracle.from_double(rng.uniform(-1, 1, ldb * nrhs))
        F, X, piv = A.copy(), B.copy(), np.zeros(n, np.int32)
        if kind == 0:
            info = oracle.orc.orc_rgetrf(n, n, F, lda, piv, 32)
            oracle.orc.orc_rgetrs(b"N", n, nrhs, F, lda, piv, X, ldb)
        else:
            info = oracle.orc.orc_rpotrf(b"L", n, F, lda, 32)
            if info == 0:
                oracle.orc.orc_rpotrs(b"L", n, nrhs, F, lda, X, ldb)
        want.append((F, X, piv, info))
        t = [torch.from_numpy(v.view(np.int32).copy()).cuda() for v in (A, B)]
        t += [torch.zeros(n, dtype=torch.int32, device="cuda"), torch.full((1,), -7, dtype=torch.int32, device="cuda")]
        keep.append(t)
        probs.append(pg._BatchProblem(kind, n, lda, nrhs, ldb, *(x.data_ptr() for x in t)))
    arr = (pg._BatchProblem * len(probs))(*probs)
    h = ctypes.c_void_p()
    assert pg._lib.posit_batch_plan_create(arr, len(probs), ctypes.byref(h)) == 0
    assert pg._lib.posit_batch_plan_launch(h, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    pg._lib.posit_batch_plan_destroy(h)
    for (kind, n, nrhs), (A, B, piv, info), (F, X, wp, wi) in zip(specs, keep, want):
        what_ = (what, kind, n, nrhs)
        assert int(info.item()) == wi, what_
        assert np.array_equal(B.cpu().numpy().view(np.uint32), X), what_
        got = A.cpu().numpy().view(np.uint32).reshape(n, n + 3)
        exp = F.reshape(n, n + 3)
        if kind == 0:
            assert np.array_equal(piv.cpu().numpy(), wp), what_
            assert np.array_equal(got, exp), what_
        elif wi == 0:
            assert np.array_equal(got, exp), what_
