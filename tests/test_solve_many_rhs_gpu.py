"""The axpy-form solves (Rgetrs 'N', Rpotrs) with many right-hand sides: the cluster that solves one
shrinks as they become many, down to one CTA; every size against the oracle bit for bit, zero and
NaR right-hand sides and a singular matrix among them.  The rule itself is checked without a GPU."""
import numpy as np
import pytest

import oracle


def test_cluster_rule():
    import posit_gpu_b200 as pg
    ctas = pg._lib.posit_solve_cluster_ctas
    assert [ctas(n, 1) for n in (1, 512, 513, 1024, 2048, 4096, 16384)] == [1, 1, 2, 2, 4, 8, 8]
    # enough right-hand sides for all SMs: a CTA each
    assert [ctas(n, 1024) for n in (512, 1024, 2048, 4096)] == [1, 1, 1, 1]
    # what one right-hand side takes is the most (in between, turns decide: more need not mean fewer)
    for n in (600, 2048, 4096, 8192, 30000, 100000, 202752):
        c = [ctas(n, r) for r in (1, 15, 16, 32, 33, 74, 75, 148, 5000)]
        assert c[0] == min(8, (n + 511) // 512) and min(c) >= 1 and max(c) == c[0]
    # long columns need their CTAs
    assert ctas(200000, 1024) == 8


# (n, right-hand sides): 1, 2, 3, 4, 6 and 8 CTAs, and more clusters than run at a time
CASES = [(40, 200), (513, 3), (513, 80), (1030, 33), (1060, 50), (1600, 16), (2100, 21), (2100, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,nrhs", CASES)
def test_solves(cuda_ok, n, nrhs):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(n + nrhs)
    # a triangular pair of moderate size: the solves do not ask how the factor came about
    A = oracle.from_double(rng.uniform(-1, 1, (n, n)) / np.sqrt(n) + np.diag(rng.uniform(1, 2, n))).reshape(-1)
    if n == 513:
        A.reshape(n, n)[100, 100] = 0  # a quotient by zero
    B = oracle.from_double(rng.uniform(-1, 1, n * nrhs))
    B[:n] = 0
    B[n:n + 50] = 0
    B[2 * n + n // 2] = oracle.P32_NAR
    piv = (np.arange(n) + 1 + rng.integers(0, np.maximum(1, n - np.arange(n)))).astype(np.int32)
    dA, dp = torch.from_numpy(A.view(np.int32)).cuda(), torch.from_numpy(piv).cuda()
    # the oracle on a sample of the right-hand sides: they do not meet
    cols = sorted({0, 1, 2, nrhs // 2, nrhs - 1} & set(range(nrhs)))
    for solve in ("getrs", "potrs"):
        dB = torch.from_numpy(B.view(np.int32).copy()).cuda()
        want = np.concatenate([B[c * n:(c + 1) * n] for c in cols])
        if solve == "getrs":
            pg.Rgetrs_dev("N", n, nrhs, dA, n, dp, dB, n)
            oracle.orc.orc_rgetrs(b"N", n, len(cols), A, n, piv, want, n)
        else:
            pg.Rpotrs_dev("L", n, nrhs, dA, n, dB, n)
            oracle.orc.orc_rpotrs(b"L", n, len(cols), A, n, want, n)
        got = dB.cpu().numpy().view(np.uint32)
        for q, c in enumerate(cols):
            assert np.array_equal(got[c * n:(c + 1) * n], want[q * n:(q + 1) * n]), (solve, c)
