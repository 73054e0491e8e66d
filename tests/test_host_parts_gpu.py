"""Host-matrix Rgemm large enough to go through in stretches of columns, against the device
entry on the same operands: transposed B, ragged last stretch, padded leading dimensions, beta
0, and C inside A's or B's address range (one stretch)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,ta,tb,beta,inside", [
    (1100, 1030, 1000, "N", "N", 0x38000000, ""), (1100, 1030, 1000, "T", "T", 0x38000000, ""),
    (1024, 1025, 1024, "N", "T", 0, ""), (700, 2100, 800, "T", "N", 0x40000000, ""),
    (2050, 2055, 2049, "N", "N", 0x40000000, ""), (1024, 1024, 1024, "N", "N", 0x40000000, "A"),
    (1024, 1024, 1024, "N", "T", 0x40000000, "B")])
def test_stretches_match_the_device(cuda_ok, m, n, k, ta, tb, beta, inside):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(m + n)
    ar, ac = (m, k) if ta == "N" else (k, m)
    br, bc = (k, n) if tb == "N" else (n, k)
    lda, ldb, ldc = ar + 3, br + 1, m + 5
    sizes = [lda * ac, ldb * bc, ldc * n]
    whole = oracle.from_double(rng.uniform(-1, 1, sum(sizes)))
    A, B, C = np.split(whole.copy(), np.cumsum(sizes)[:2])
    if inside == "A":
        C, ldc = A, lda
    elif inside == "B":
        C, ldc = B, ldb
    d = [torch.from_numpy(x.view(np.int32).copy()).cuda() for x in (A, B, C)]
    pg.Rgemm_dev(ta, tb, m, n, k, oracle.P32_MINUS_ONE, d[0], lda, d[1], ldb, beta, d[2], ldc)
    want = d[2].cpu().numpy().view(np.uint32)
    pg.Rgemm(ta, tb, m, n, k, oracle.P32_MINUS_ONE, A, lda, B, ldb, beta, C, ldc)
    assert np.array_equal(C, want)
