"""The bench's roofline line names the kernel that ran and takes the instruction and traffic
figures, which are the staged main kernel's, for that one only."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402
from posit_gpu_b200 import perf  # noqa: E402


@pytest.mark.parametrize("m,n,k,kernel", [(8192, 8192, 8192, "gemm_main_kernel<0>"),
                                          (512, 512, 512, "gemm_fused_kernel<0, 2, 2>"),
                                          (1200, 1200, 32, "gemm_fused_kernel<0, 4, 2>")])
def test_kernel_and_figures(monkeypatch, m, n, k, kernel):
    import posit_gpu_b200 as pg
    monkeypatch.setattr(perf, "inst_count_current", lambda: True)
    route = pg._lib.posit_rgemm_route(m, n, k)
    r = bench.gemm_roofline(route, m, n, k, 1e-3, 1965.0)
    assert r["kernel"] == kernel and r["main_kernel_ms"] == 1.0
    assert r["posit_gop_s_main_kernel"] == round(2.0 * m * n * k / 1e-3 / 1e9, 2)
    figures = ("achieved", "frac", "traffic", "warp_inst_per_mad", "fp64_pipe_frac", "inst_source")
    for key in figures:
        assert (r[key] is None) == (route != 0), key
    if route == 0:
        assert r["traffic"] == perf.MAIN_KERNEL_DRAM_BYTES_PER_MAD * m * n * k


def test_stale_counts_and_trailing_shapes(monkeypatch):
    monkeypatch.setattr(perf, "inst_count_current", lambda: False)
    r = bench.gemm_roofline(0, 8192, 8192, 8192, 0.3, 1965.0)
    assert r["achieved"] is r["frac"] is r["fp64_pipe_frac"] is None and r["inst_source_stale"]
    assert bench.gemm_roofline(0, 8128, 8128, 64, 1e-3, 1965.0, 64)["traffic"] == perf.trailing_traffic(64)
    assert bench.gemm_roofline(2, 128, 128, 64, 1e-3, 1965.0, 64)["traffic"] is None
