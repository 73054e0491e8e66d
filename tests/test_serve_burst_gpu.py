"""A server with an order window admits a burst largest work first also when it has nothing else to
do as the burst begins, and when the request ahead of it ends in the middle of it; with the
window off requests go in arrival order at once."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _requests(rng, sizes):
    return [(n, oracle.from_double(rng.uniform(-1, 1, n * n)), oracle.from_double(rng.uniform(-1, 1, n)),
             np.zeros(n, np.uint32)) for n in sizes]


def _admitted(res):
    """Request numbers in the order of admission: submitted within moments, they differ by it."""
    return sorted(range(len(res)), key=lambda i: res[i]["queue_ms"])


@pytest.mark.parametrize("ahead", [0, 40])
def test_burst_on_an_idle_server(cuda_ok, ahead):
    import posit_gpu_b200 as pg
    rng = np.random.default_rng(5)
    sizes = [300, 900, 400, 600]
    reqs, first = _requests(rng, sizes), _requests(rng, [ahead] if ahead else [])
    with pg.Server(max_inflight=1, lanes=2, batch_max_n=64, order_window_ms=60000) as srv:
        t0 = [srv.submit(0, n, 1, A, B, X) for n, A, B, X in first]
        res = [srv.wait(t) for t in [srv.submit(0, n, 1, A, B, X) for n, A, B, X in reqs]]
        assert all(srv.wait(t)["status"] == 0 for t in t0)
    assert all(r["status"] == 0 for r in res)
    assert [sizes[i] for i in _admitted(res)] == [900, 600, 400, 300]


def test_arrival_order_without_a_window(cuda_ok):
    import posit_gpu_b200 as pg
    rng = np.random.default_rng(6)
    reqs = _requests(rng, [300, 900, 400, 600])
    with pg.Server(max_inflight=1, lanes=2, batch_max_n=64) as srv:
        res = [srv.wait(t) for t in [srv.submit(0, n, 1, A, B, X) for n, A, B, X in reqs]]
    assert all(r["status"] == 0 for r in res)
    assert _admitted(res) == [0, 1, 2, 3]
