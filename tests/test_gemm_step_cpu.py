"""The FP64 multiply-add step without an exactness test, and the rounding outside the fast
window, against the oracle.  The same header the CUDA kernels compile, built for the host
(tests/host_core_check.cpp)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle

HERE = os.path.dirname(os.path.abspath(__file__))
U32 = np.ctypeslib.ndpointer(dtype=np.uint32, flags="C_CONTIGUOUS")


@pytest.fixture(scope="module")
def mac(tmp_path_factory):
    out = tmp_path_factory.mktemp("hc") / "libhc.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", str(out),
                           os.path.join(HERE, "host_core_check.cpp")])
    fn = ctypes.CDLL(str(out)).hc_f64_mac_n
    fn.argtypes = [U32, U32, U32, U32, ctypes.c_long, ctypes.c_int]
    fn.restype = ctypes.c_long
    return fn


def _at_scale(rng, scale):
    """Posits of the given scales with random, all-zero, all-one and one-bit fractions."""
    n = scale.size
    k = scale >> 2
    run = np.where(k < 0, -k, k + 1)
    frac = rng.integers(0, 2**32, n, dtype=np.uint64)
    pick = rng.integers(0, 6, n)
    frac = np.where(pick == 0, 0, frac)
    frac = np.where(pick == 1, 2**32 - 1, frac)
    frac = np.where(pick == 2, np.uint64(1) << rng.integers(0, 32, n).astype(np.uint64), frac).astype(np.uint64)
    regime = np.where(k < 0, 1, (np.uint64(1) << run.astype(np.uint64)) * 2 - 2).astype(np.uint64)
    body = (regime << np.uint64(34)) | ((scale & 3).astype(np.uint64) << np.uint64(32)) | frac  # run+1+2+32 bits
    drop = run + 35 - 31
    u = (body >> drop.astype(np.uint64)).astype(np.uint32)
    u = np.where(u == 0, 1, np.minimum(u, 0x7FFFFFFF)).astype(np.uint32)
    return np.where(rng.integers(0, 2, n) == 1, (0 - u.astype(np.int64)) & 0xFFFFFFFF, u).astype(np.uint32)


def _want(c, t, a):
    p, out = np.empty_like(c), np.empty_like(c)
    oracle.orc.orc_p32_mul_n(t, a, p, c.size)
    oracle.orc.orc_p32_add_n(c, p, out, c.size)
    return out


@pytest.mark.parametrize("what", ["gaps", "edges", "products"])
@pytest.mark.parametrize("use_table", [1, 0])
def test_step_without_exactness_test_matches_oracle(mac, what, use_table):
    """gaps: every pair of scales 20..40 apart, where the FP64 sum is inexact; edges: sums
    around both ends of the fast window and beyond; products: products there."""
    rng = np.random.default_rng({"gaps": 1, "edges": 2, "products": 3}[what])
    n = 1_500_000
    if what == "gaps":
        sc = rng.integers(-120, 121, n)
        st = np.clip(sc - rng.integers(20, 41, n), -120, 120)
        c, t, a = _at_scale(rng, sc), _at_scale(rng, st), np.full(n, oracle.P32_ONE, np.uint32)
        swap = rng.integers(0, 2, n) == 1
        c[swap], t[swap] = t[swap], c[swap]
    else:
        side = np.where(rng.integers(0, 2, n) == 1, 1, -1)
        sc = np.clip(side * rng.integers(100, 121, n), -120, 120)
        c = _at_scale(rng, sc)
        if what == "edges":
            t = _at_scale(rng, np.clip(sc + rng.integers(-6, 7, n), -120, 120))
            a = np.full(n, oracle.P32_ONE, np.uint32)
        else:
            st = rng.integers(-120, 121, n)
            t, a = _at_scale(rng, st), _at_scale(rng, np.clip(sc - st + rng.integers(-3, 4, n), -120, 120))
    got = np.empty_like(c)
    flagged = mac(c, t, a, got, n, use_table)
    assert np.array_equal(got, _want(c, t, a))
    if what == "gaps":
        assert flagged < n // 4  # an inexact sum is not flagged, only a result outside the window is
