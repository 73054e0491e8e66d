"""posit_rgemm on host matrices, its host code run without a GPU against a stand-in for the CUDA
runtime (host_parts_stub.cpp): when device memory runs out anywhere in the call, the call says so
and C is untouched (with beta != 0 a half-updated C could not be computed again); when it does
not, all of C is written, and every allocation is given back."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import posit_gpu_b200 as pg
from posit_gpu_b200.build import ARCH, CSRC, NVCC

HERE = os.path.dirname(os.path.abspath(__file__))
MARK = 0x12345678
E_NO_MEMORY = -3


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("host_parts")
    stub, capi = str(out / "stub.o"), str(out / "capi.o")
    cuda = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-I", cuda, "-c",
                           os.path.join(HERE, "host_parts_stub.cpp"), "-o", stub])
    subprocess.check_call([NVCC, *ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-c", os.path.join(CSRC, "capi.cu"),
                           "-o", capi])
    so = str(out / "libhostparts.so")
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, stub, capi])
    lib = ctypes.CDLL(so)
    lib.fake_peak.restype = ctypes.c_size_t
    lib.posit_rgemm.argtypes = pg._lib.posit_rgemm.argtypes
    return lib


def _call(lib, m, n, k, beta, fail_at):
    A, B, C = np.ones(m * k, np.uint32), np.ones(k * n, np.uint32), np.full(m * n, 7, np.uint32)
    lib.fake_reset(fail_at)
    p = [ctypes.c_void_p(x.ctypes.data) for x in (A, B, C)]
    rc = lib.posit_rgemm(b"N", b"N", m, n, k, 0xC0000000, p[0], m, p[1], k, beta, p[2], m)
    assert lib.fake_live() == 0
    return rc, C


# one piece; two and four stretches of columns, the last one narrower
@pytest.mark.parametrize("m,n,k", [(100, 90, 80), (1024, 1100, 1024), (2048, 2080, 2048)])
@pytest.mark.parametrize("beta", [0, 0x40000000])
def test_all_or_nothing(lib, m, n, k, beta):
    rc, C = _call(lib, m, n, k, beta, 0)
    assert rc == 0 and (C == MARK).all()
    allocs = lib.fake_allocs()
    assert allocs >= 1
    for fail_at in range(1, allocs + 1):
        rc, C = _call(lib, m, n, k, beta, fail_at)
        assert rc == E_NO_MEMORY, fail_at
        assert (C == 7).all(), fail_at
