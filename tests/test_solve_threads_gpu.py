"""Solves of very different orders issued by several threads at once, each on its own stream:
every call succeeds and gives the bits it gives alone (a kernel's shared-memory limit is shared
by all threads of the process)."""
import threading

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

ORDERS = [40, 1500, 300, 4100, 90, 2600, 700, 3300]


def test_solves_from_threads(cuda_ok):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(5)
    jobs = []
    for n in ORDERS:  # triangles with few entries off the diagonal, so that a solve is short
        A = np.zeros((n, n), np.uint32)
        np.fill_diagonal(A, oracle.from_double(rng.uniform(1, 2, n)))
        A[n // 2, :n // 2] = A[: n // 2, n // 2] = oracle.from_double(rng.uniform(-1, 1, n // 2))
        b = oracle.from_double(rng.uniform(-1, 1, n))
        ipiv = np.minimum(np.arange(1, n + 1) + rng.integers(0, 3, n), n).astype(np.int32)
        jobs.append([torch.from_numpy(x.reshape(-1).view(np.int32).copy()).cuda() for x in (A, b, ipiv)])
    torch.cuda.synchronize()

    def solve(i, stream):
        n, (A, b, ipiv) = ORDERS[i], jobs[i]
        x, y = b.clone(), b.clone()
        pg.Rgetrs_dev("N", n, 1, A, n, ipiv, x, n, stream=stream)
        pg.Rpotrs_dev("L", n, 1, A, n, y, n, stream=stream)
        return x, y

    alone = [solve(i, None) for i in range(len(ORDERS))]
    torch.cuda.synchronize()
    failures = []

    def worker(i):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                got = [solve(i, st) for _ in range(30)]
                st.synchronize()
            for x, y in got:
                assert torch.equal(x, alone[i][0]) and torch.equal(y, alone[i][1])
        except Exception as exc:  # noqa: BLE001 -- reported by the main thread
            failures.append((ORDERS[i], repr(exc)))

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(len(ORDERS))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
