"""LU blocks that go by inner panels: wider than 32 columns, or with more rows than the cluster
panel holds at their width (4864 rows of 32 columns, 6144 of 24), down to inner panels of 16;
remainders of one column; blocks beyond 8192 rows, which keep their two launches per column.
Against the oracle at the same block size bit for bit: ties, values outside the fast window, zero
pivots over and under a NaR (interchanges across the inner panels)."""
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
        for c in {min(3, n - 1), n // 2, n - 1}:  # zero columns in the first, a middle and the last panel
            A[c] = 0
        A[0, 1:] = 0
        A[0, 0] = oracle.P32_NAR
    return A.reshape(-1)


# 33 = 32 + 1, 65 = 2 * 32 + 1; 4900 x 32 = 24 + 8; 6200 x 32 = 16 + 16; 6200 x 24 = 16 + 8
CASES = [(33, 33, 33), (40, 90, 40), (100, 100, 64), (129, 96, 96), (300, 130, 65), (513, 200, 512), (1030, 70, 48),
         (4900, 40, 32), (6200, 34, 32), (6200, 30, 24), (5000, 41, 40), (8300, 36, 34)]


@pytest.mark.parametrize("kind", ["uniform", "ties", "wide", "special"])
@pytest.mark.parametrize("m,n,nb", CASES)
def test_lu(cuda_ok, m, n, nb, kind):
    import torch

    import posit_gpu_b200 as pg
    A = _matrix(np.random.default_rng(m + nb), m, n, kind)
    want, piv = A.copy(), np.zeros(min(m, n), np.int32)
    info = oracle.orc.orc_rgetrf(m, n, want, m, piv, nb)
    dA = torch.from_numpy(A.view(np.int32).copy()).cuda()
    dp, di = (torch.zeros(k, dtype=torch.int32, device="cuda") for k in (min(m, n), 1))
    pg.Rgetrf_dev(m, n, dA, m, dp, di, nb=nb)
    assert int(di.item()) == info
    assert np.array_equal(dp.cpu().numpy(), piv)
    assert np.array_equal(dA.cpu().numpy().view(np.uint32), want)
