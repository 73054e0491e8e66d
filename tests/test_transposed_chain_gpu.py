"""The transposed triangular solves' warp chain on both sides of its groups (16 addends),
runs (8), windows (512) and storage forms (five bytes an addend from 8941 rows), on values that stay in
one binade, wander across powers of two, change fraction width, go wide, cancel to zero or
hold a NaR: Rpotrs 'L' and 'U' against the oracle bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 8, 9, 16, 17, 18, 33, 65, 66, 80, 130, 527, 530, 1060]


def _triangle(rng, n, kind):
    T = rng.uniform(-1, 1, (n, n))
    if kind == "calm":  # the running value moves by 1e-4 of itself
        T *= 1e-4
    elif kind == "near":  # around a power of two, steps of 1/100
        T *= 0.01
    elif kind == "wide":
        T = np.sign(T) * 10.0 ** rng.uniform(-12, 6, (n, n))
    elif kind == "ties":
        T = rng.choice([-1.0, 1.0, 0.5, 2.0 ** -26, -(2.0 ** -27), 0.0, 2.0 ** -28], (n, n))
    np.fill_diagonal(T, 1.0 if kind == "ties" else rng.uniform(1, 2, n))
    return T


def _check(pg, torch, uplo, n, nrhs, A, B):
    want = B.copy()
    oracle.orc.orc_rpotrs(uplo.encode(), n, nrhs, A, n, want, n)
    dA, dB = (torch.from_numpy(x.view(np.int32).copy()).cuda() for x in (A, B))
    pg.Rpotrs_dev(uplo, n, nrhs, dA, n, dB, n)
    assert np.array_equal(dB.cpu().numpy().view(np.uint32), want), (uplo, n, nrhs)


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("kind", ["calm", "near", "wide", "ties", "nar"])
def test_chain_edges(cuda_ok, kind, uplo):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(["calm", "near", "wide", "ties", "nar"].index(kind))
    for n in SIZES:
        A = oracle.from_double(_triangle(rng, n, kind).reshape(-1, order="F"))
        B = oracle.from_double(rng.choice([-1, 1], 3 * n) * rng.uniform(0.9, 1.1, 3 * n))
        B[::11] = 0
        if kind == "nar" and n > 2:
            A[(n - 1) if uplo == "L" else (n - 1) * n] = oracle.P32_NAR
        _check(pg, torch, uplo, n, 3, A, B)


def test_chain_on_patterns(cuda_ok):
    import torch

    import posit_gpu_b200 as pg
    n, rng = 9000, np.random.default_rng(9)
    A = np.zeros((n, n), np.uint32)  # row c holds column c of a banded lower triangle
    for d in range(60):
        v = oracle.from_double(rng.uniform(1, 2, n) if d == 0 else rng.uniform(-1, 1, n) * 0.05)
        A[np.arange(n - d), np.arange(d, n)] = v[:n - d]
    _check(pg, torch, "L", n, 1, A.reshape(-1), oracle.from_double(rng.uniform(-1, 1, n)))
