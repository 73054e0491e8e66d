"""Products of few rows or columns, and others around the lines between the GEMM's routes: the
route each takes (checked without a GPU) and the result on every transpose case against the oracle
bit for bit.  A tile that is mostly padding costs what a full one does."""
import numpy as np
import pytest

import oracle

STAGED, F64X32, F32X32 = 0, 1, 2


def test_routes():
    import posit_gpu_b200 as pg
    route = pg._lib.posit_rgemm_route
    # half of a 64-wide tile, or more, would be padding
    for m, n, k in [(8192, 32, 8192), (32, 8192, 4096), (8192, 1, 8192), (1, 8192, 8192), (16384, 8, 128),
                    (65536, 4, 64), (100000, 32, 32), (16384, 1, 1024), (12800, 32, 512), (3300, 129, 1024)]:
        assert route(m, n, k) != STAGED, (m, n, k)
    # full tiles in numbers
    for m, n, k in [(8192, 8192, 8192), (8128, 8128, 64), (8128, 8128, 32), (4096, 4096, 64), (2049, 1537, 3001),
                    (1024, 1024, 1024), (2048, 2048, 2048)]:
        assert route(m, n, k) == STAGED, (m, n, k)
    for m, n, k in [(1, 1, 1), (48, 48, 32), (256, 256, 256), (320, 320, 300), (8, 8, 8192)]:
        assert route(m, n, k) == F32X32, (m, n, k)
    for m, n, k in [(1200, 1200, 32), (51200, 8, 128), (1400, 1400, 16), (4800, 96, 512)]:
        assert route(m, n, k) == F64X32, (m, n, k)
    assert route(0, 5, 5) == route(5, 0, 5) == route(5, 5, 0) == -1
    # more 32-wide tiles than a grid has rows of
    assert route(1, 65535 * 32, 1) != STAGED and route(1, 65535 * 32 + 1, 1) == STAGED


# (m, n, k, route)
CASES = [(6500, 31, 90, F32X32), (33, 6500, 90, F32X32), (9601, 1, 150, F32X32), (1, 9601, 150, F32X32),
         (4801, 95, 40, F64X32), (25700, 7, 30, F64X32), (1250, 1190, 21, F64X32), (1300, 1230, 130, STAGED),
         (800, 810, 300, F32X32)]


@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
def test_skinny_products(cuda_ok, ta, tb):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(5)
    for m, n, k, route in CASES:
        assert pg._lib.posit_rgemm_route(m, n, k) == route, (m, n, k)
        ra, ca = (m, k) if ta == "N" else (k, m)
        rb, cb = (k, n) if tb == "N" else (n, k)
        A, B, C = (oracle.from_double(rng.uniform(-1, 1, v)) for v in (ra * ca, rb * cb, m * n))
        A[rng.integers(0, A.size)] = oracle.P32_NAR
        d = [torch.from_numpy(v.view(np.int32).copy()).cuda() for v in (A, B, C)]
        pg.Rgemm_dev(ta, tb, m, n, k, oracle.P32_MINUS_ONE, d[0], ra, d[1], rb, oracle.P32_ONE, d[2], m)
        assert oracle.rgemm(ta, tb, m, n, k, oracle.P32_MINUS_ONE, A, ra, B, rb, oracle.P32_ONE, C, m) == 0
        assert np.array_equal(d[2].cpu().numpy().view(np.uint32), C), (m, n, k)
        assert pg.device_error() == 0


@pytest.mark.gpu
def test_more_columns_than_a_grid_of_narrow_tiles(cuda_ok):
    import torch

    import posit_gpu_b200 as pg
    m, n, k = 2, 65535 * 32 + 70, 3
    rng = np.random.default_rng(6)
    A, B = (oracle.from_double(rng.uniform(-1, 1, v)) for v in (m * k, k * n))
    C = np.zeros(m * n, np.uint32)
    d = [torch.from_numpy(v.view(np.int32).copy()).cuda() for v in (A, B, C)]
    pg.Rgemm_dev("N", "N", m, n, k, oracle.P32_ONE, d[0], m, d[1], k, 0, d[2], m)
    assert oracle.rgemm("N", "N", m, n, k, oracle.P32_ONE, A, m, B, k, 0, C, m) == 0
    assert np.array_equal(d[2].cpu().numpy().view(np.uint32), C)
