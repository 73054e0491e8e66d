"""The panel kernels at the edges of rows per CTA (128), CTAs (8), slots per thread and panel
widths (the Cholesky panel's 32 columns; the column padding of 8), against the oracle bit for
bit: ties, zero columns, NaR over zeros, values outside the fast window; a Cholesky that fails
in the first, a middle and the last column of a panel leaves the same info."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matrix(rng, m, n, kind):
    A = rng.uniform(-1, 1, (n, m))  # row c: column c
    if kind == "ties":
        A = rng.choice([-1.0, 1.0, 0.5, -0.5, 2.0], (n, m))
    elif kind == "wide":
        A = np.sign(A) * 10.0 ** rng.uniform(-18, 18, (n, m))
    A = oracle.from_double(A.reshape(-1)).reshape(n, m)
    if kind == "special":
        A[min(3, n - 1)] = 0
        A[0, 1:] = 0
        A[0, 0] = oracle.P32_NAR
    return A.reshape(-1)


@pytest.mark.parametrize("kind", ["uniform", "ties", "wide", "special"])
@pytest.mark.parametrize("m,n,nb", [(1, 1, 8), (31, 33, 16), (33, 31, 9), (129, 40, 17), (257, 70, 25), (1030, 40, 31),
                                    (2100, 34, 33), (8300, 12, 5)])
def test_lu_panels(cuda_ok, m, n, nb, kind):
    import torch

    import posit_gpu_b200 as pg
    A = _matrix(np.random.default_rng(m), m, n, kind)
    want, piv = A.copy(), np.zeros(min(m, n), np.int32)
    info = oracle.orc.orc_rgetrf(m, n, want, m, piv, nb)
    dA = torch.from_numpy(A.view(np.int32).copy()).cuda()
    dp, di = (torch.zeros(k, dtype=torch.int32, device="cuda") for k in (min(m, n), 1))
    pg.Rgetrf_dev(m, n, dA, m, dp, di, nb=nb)
    assert int(di.item()) == info
    assert np.array_equal(dp.cpu().numpy(), piv)
    assert np.array_equal(dA.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("n,nb,bad", [(1, 8, -1), (33, 32, -1), (65, 31, -1), (200, 32, -1), (513, 24, -1),
                                      (700, 32, 32), (700, 32, 47), (700, 32, 63), (100, 32, 99)])
def test_cholesky_panels(cuda_ok, n, nb, bad):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (n, n))
    S = X @ X.T / n + np.eye(n)
    if bad >= 0:
        S[bad, bad] = -1.0
    A = oracle.from_double(S.reshape(-1))
    want = A.copy()
    info = oracle.orc.orc_rpotrf(b"L", n, want, n, nb)
    dA, di = torch.from_numpy(A.view(np.int32).copy()).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    pg.Rpotrf_dev("L", n, dA, n, di, nb=nb)
    assert int(di.item()) == info == (bad + 1 if bad >= 0 else 0)
    got = dA.cpu().numpy().view(np.uint32).reshape(n, n)
    low = np.triu(np.ones((n, n), bool))  # rows are columns here
    done = low if bad < 0 else low & (np.arange(n)[:, None] < bad // nb * nb)
    assert np.array_equal(got[done], want.reshape(n, n)[done])
