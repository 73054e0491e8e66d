"""Figures the benchmark's roofline uses, with where each one comes from.

The GEMM main kernel runs each posit multiply-add as FP64 operations plus a little
integer work (posit32.cuh, f64_posit_mac): it is bound by instruction issue -- each SM
sub-partition (4 per SM, 148 SMs on B200) issues at most one warp instruction per cycle --
with the FP64 pipe (half rate) the busiest pipe: an FP64 warp instruction takes two issue
slots, so the issue figure below cannot reach 1 (6 of 14 instructions take two).  The roofline therefore compares the
kernel's issued warp instructions per second with 148 * 4 * f_SM warp instructions per
second, f_SM being the SM clock sampled during the run.  The instruction count per posit
multiply-add is a property of the compiled kernel (its fast path is branch-free),
measured with ncu on the same kernel and recorded here.
"""

import hashlib
import os

SM_COUNT = 148
SMSP_PER_SM = 4
SM_MAX_MHZ = 1965.0

# Warp instructions issued by gemm_main_kernel per posit multiply-add:
# smsp__inst_executed.sum / (m*n*k) for one NN launch at m = n = k = 4096
# (30,100,779,008 / 68,719,476,736 = 0.4380, i.e. 14.02 thread instructions).  Of those,
# 6 per multiply-add run on the FP64 pipe (DMUL, DFMA, 4 DADD; smsp__inst_executed_pipe_fp64.sum
# 12,952,535,040 = 0.1885): FP64 pipe 61.7 %, ALU pipe 41.7 %, LSU 46.1 %, issue 71.7 % busy in
# the same capture.
WARP_INST_PER_MAD = 0.4380
FP64_WARP_INST_PER_MAD = 6 / 32
INST_SOURCE = ("ncu, gemm_main_kernel<0>, NN 4096^3 U[-1,1] "
               "(profiles/gemm_main_kernel_nn_4096.md)")
# DRAM bytes (read + write) per posit multiply-add of the same launch:
# (3,935,058,432 + 70,387,968) / 68,719,476,736.
MAIN_KERNEL_DRAM_BYTES_PER_MAD = 0.0583


def issue_peak_warp_inst_per_s(sm_mhz):
    return SM_COUNT * SMSP_PER_SM * float(sm_mhz) * 1e6


def fp64_pipe_peak_warp_inst_per_s(sm_mhz):
    """FP64 pipe: 16 lanes per SM sub-partition per cycle, i.e. half a warp instruction."""
    return SM_COUNT * SMSP_PER_SM * 0.5 * float(sm_mhz) * 1e6


# The instruction count above belongs to one build of the main kernel.  It is tied to
# that build by a SHA-256 over the sources that define the kernel's instruction stream
# (gemm.cu and the headers it includes) and the compiler flags (build.py's ARCH and CFLAGS);
# the benchmark recomputes the digest and, when it differs, marks the count stale and
# reports no roofline fraction from it.
KERNEL_SOURCES = ["csrc/gemm.cu", "csrc/gemm.cuh", "csrc/gemm_tile.cuh", "csrc/posit32.cuh"]
INST_SOURCE_DIGEST = "54aed4f387b4609bc67e2a97ff14d8745f33f5a74caa3839ff5ec8225e792bcf"


def kernel_source_digest():
    from . import build as _build
    here = os.path.dirname(os.path.abspath(__file__))
    h = hashlib.sha256()
    for rel in KERNEL_SOURCES:
        with open(os.path.join(here, rel), "rb") as fh:
            h.update(rel.encode() + b"\0" + fh.read() + b"\0")
    h.update(b"flags\0" + " ".join(_build.ARCH + _build.CFLAGS).encode() + b"\0")
    return h.hexdigest()


def inst_count_current():
    """True when WARP_INST_PER_MAD was measured on the kernel sources present now."""
    return INST_SOURCE_DIGEST is not None and kernel_source_digest() == INST_SOURCE_DIGEST


# DRAM bytes (read + write) of one main-kernel launch at the LU trailing-update shapes
# m = n = 8192 - b, k = b (key b), from ncu dram__bytes_read.sum + dram__bytes_write.sum
# of that launch.  Empty until measured; the benchmark then reports no traffic figure for
# the shape rather than one scaled from another shape.
TRAILING_TRAFFIC_BYTES = {16: 483767040, 32: 482796544, 64: 483489024, 128: 484047104, 256: 482452992}
TRAILING_TRAFFIC_SOURCE = ("ncu --metrics dram__bytes_read.sum,dram__bytes_write.sum, gemm_main_kernel<0>, "
                           "one launch per shape (profiles/gemm_main_kernel_lu_trailing.md)")


def trailing_traffic(k):
    return TRAILING_TRAFFIC_BYTES.get(int(k))
