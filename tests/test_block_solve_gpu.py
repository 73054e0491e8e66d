"""The axpy-form solves by blocks of 32 rows on one to eight CTAs, at the edges of blocks,
warps and CTAs (512 rows each), with zero multipliers over NaR coefficients (skipped, as the
reference does), NaR right-hand sides, values outside the fast window and long interchange
sequences: Rgetrs 'N' against the oracle bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["uniform", "wide", "zeros", "nar"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 100, 511, 512, 513, 1040, 1537, 4128])
def test_rgetrs_blocks(cuda_ok, n, kind):
    import torch

    import posit_gpu_b200 as pg
    if n > 1100 and kind in ("wide", "nar"):
        pytest.skip("the large sizes differ in the dealing of blocks only")
    rng = np.random.default_rng(n)
    nrhs, lda = 3, n + 3
    A = rng.uniform(-1, 1, (n, lda)) * (1.0 if n < 200 else 8.0 / n)  # row c: column c
    if kind == "wide":
        A = np.sign(A) * 10.0 ** rng.uniform(-25, 25, (n, lda))
    A[np.arange(n), np.arange(n)] = rng.uniform(1, 2, n)
    A = oracle.from_double(A.reshape(-1))
    B = oracle.from_double(rng.uniform(-1, 1, nrhs * n))
    ipiv = (np.arange(n) + rng.integers(0, n - np.arange(n), n) + 1).astype(np.int32)
    if kind == "zeros":
        B[n // 3:n] = 0
        B[n:n + n // 2] = 0
        ipiv = (np.arange(n) + 1).astype(np.int32)
        A[min(1, n - 1)] = oracle.P32_NAR  # column 0 of L: b_0 is zero in the second right-hand side
    if kind == "nar":
        B[n // 2] = oracle.P32_NAR
        A[(n - 1) * lda] = oracle.P32_NAR  # U's last column
    want = B.copy()
    oracle.orc.orc_rgetrs(b"N", n, nrhs, A, lda, ipiv, want, n)
    dA, dB = (torch.from_numpy(x.view(np.int32).copy()).cuda() for x in (A, B))
    pg.Rgetrs_dev("N", n, nrhs, dA, lda, torch.from_numpy(ipiv).cuda(), dB, n)
    assert np.array_equal(dB.cpu().numpy().view(np.uint32), want)
