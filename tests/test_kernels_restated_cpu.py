"""What the kernels compute with, on the CPU: the quotient and the root from FP64 with their integer
fallback near half way between two posits, against the oracle on constructed ties, near-ties, the
edges of the fast window, zeros and NaR; and the present panels' and adding warp's algorithms,
restated (host_kernels_check.cpp), against the reference's recursion and plain additions."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle

HERE = os.path.dirname(os.path.abspath(__file__))
U32 = np.ctypeslib.ndpointer(dtype=np.uint32, flags="C_CONTIGUOUS")
I32 = np.ctypeslib.ndpointer(dtype=np.int32, flags="C_CONTIGUOUS")


@pytest.fixture(scope="module")
def hk(tmp_path_factory):
    out = tmp_path_factory.mktemp("hk") / "libhk.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-o", str(out),
                           os.path.join(HERE, "host_kernels_check.cpp")])
    lib = ctypes.CDLL(str(out))
    lib.hk_div_n.argtypes = [U32, U32, U32, ctypes.c_long]
    lib.hk_sqrt_n.argtypes = [U32, U32, ctypes.c_long]
    lib.hk_lu_panel.argtypes = [U32, ctypes.c_int, ctypes.c_int, I32]
    lib.hk_chol_panel.argtypes = [U32, ctypes.c_int, ctypes.c_int]
    lib.hk_warp_chain.argtypes = [ctypes.c_uint32, U32, ctypes.c_int, ctypes.c_int,
                                  np.ctypeslib.ndpointer(dtype=np.int64, flags="C_CONTIGUOUS")]
    lib.hk_plain_chain.argtypes = [ctypes.c_uint32, U32, ctypes.c_int, ctypes.c_int]
    for f in ("hk_div_n", "hk_sqrt_n"):
        getattr(lib, f).restype = ctypes.c_long
    for f in ("hk_warp_chain", "hk_plain_chain"):
        getattr(lib, f).restype = ctypes.c_uint32
    return lib


def _div(hk, t, a):
    t, a = (np.ascontiguousarray(x, np.uint32) for x in (t, a))
    got, want = np.empty_like(t), np.empty_like(t)
    near = hk.hk_div_n(t, a, got, t.size)
    oracle.orc.orc_p32_div_n(t, a, want, t.size)
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, [(hex(t[i]), hex(a[i]), hex(got[i]), hex(want[i])) for i in bad[:3]]
    return near


def _fraction_bits(x):
    e = np.floor(np.log2(np.abs(x))).astype(int)
    k = e >> 2
    run = np.where(k < 0, -k, k + 1)
    return e, np.maximum(28 - run, 0)


def _neighbours(u, by):
    """Patterns `by` steps away, without passing zero or NaR."""
    v = (u.astype(np.int64) + by) & 0xFFFFFFFF
    ok = ((v ^ u) & 0x80000000 == 0) & (v & 0x7FFFFFFF != 0)
    return np.where(ok, v, u).astype(np.uint32)


def test_quotient_on_ties_and_near_ties(hk):
    rng = np.random.default_rng(1)
    n = 300_000
    # z of moderate precision, the divisor a power of two or of few bits: a (z + half a step) is a posit
    z = np.ldexp(rng.uniform(1, 2, n), rng.integers(-90, 90, n)) * rng.choice([-1, 1], n)
    z = oracle.to_double(oracle.from_double(z))
    e, fb = _fraction_bits(z)
    tie = z + np.ldexp(1.0, e - fb - 1)
    a = np.ldexp(rng.choice([1.0, 1.5, 1.25, 1.125], n), -e + rng.integers(-3, 4, n)) * rng.choice([-1, 1], n)
    a = oracle.to_double(oracle.from_double(a))
    t = oracle.from_double(tie * a)
    ua = oracle.from_double(a)
    exact = oracle.to_double(t) == tie * a
    near = _div(hk, t, ua)
    assert exact.sum() > n // 4 and near >= exact.sum() // 2  # the integer quotient decides these
    for by in (-2, -1, 1, 2):
        _div(hk, _neighbours(t, by), ua)
    # any divisor: quotients as near to half way as posits t get
    a = oracle.to_double(oracle.from_double(rng.uniform(1, 2, n)))
    ua = oracle.from_double(a)
    t = oracle.from_double(tie / np.ldexp(1.0, e) * a)
    for by in (-1, 0, 1):
        _div(hk, _neighbours(t, by), ua)


def test_quotient_next_to_half_way(hk):
    """Quotients 2^-51 to 2^-56 of their size away from half way between two posits: the FP64 value
    of most is half way itself, and only the integer quotient knows the side.  t = (a h -+ 1) / 2^28 with the 29-bit odd
    h half way and a its inverse modulo 2^28 (or less that)."""
    rng = np.random.default_rng(6)
    h = (rng.integers(2**27, 2**28, 40_000, dtype=np.uint64) * np.uint64(2) + np.uint64(1))
    inv = h.copy()  # 3 bits right; doubled by each step
    for _ in range(5):
        inv = inv * (np.uint64(2) - h * inv)
    m = np.uint64(2**28)
    total = 0
    for a, r in ((inv % m, 1), ((m - inv % m) % m, -1)):
        ok = (a < 2**27) & (a > 2**23)  # t of at most 28 bits; 1 / (a h) below 2^-50
        A, H = a[ok], h[ok]
        t = (A.astype(object) * H.astype(object) - r)
        assert all(v % 2**28 == 0 for v in t)
        t = np.array([v >> 28 for v in t], np.float64)
        ut, ua = (oracle.from_double(x / 2.0 ** np.floor(np.log2(x))) for x in (t, A.astype(np.float64)))
        assert _div(hk, ut, ua) == ut.size
        total += ut.size
    assert total > 20_000


def test_quotient_everywhere_else(hk):
    rng = np.random.default_rng(2)
    n = 500_000
    _div(hk, rng.integers(0, 2**32, n, dtype=np.uint64), rng.integers(0, 2**32, n, dtype=np.uint64))
    x, y = (oracle.from_double(rng.uniform(-1, 1, n)) for _ in range(2))
    _div(hk, x, y)
    # both edges of the fast window and beyond, where quotients saturate
    wide = [oracle.from_double(np.ldexp(rng.uniform(1, 2, n), s * rng.integers(40, 121, n))) for s in (1, -1)]
    _div(hk, wide[0], wide[1])
    _div(hk, wide[1], wide[0])
    pw = np.array([1 << i for i in range(31)], np.uint64)
    edge = np.concatenate([pw, pw - 1, pw + 1, [0, 0x80000000, 0x7FFFFFFF, 0xFFFFFFFF, 0x40000000, 0xC0000000]])
    edge = np.concatenate([edge, (2**32 - edge) % 2**32]).astype(np.uint32)
    T, A = np.meshgrid(edge, edge)
    _div(hk, T.reshape(-1), A.reshape(-1))


def test_root(hk):
    rng = np.random.default_rng(3)
    n = 300_000

    def check(a):
        a = np.ascontiguousarray(a, np.uint32)
        got, want = np.empty_like(a), np.empty_like(a)
        near = hk.hk_sqrt_n(a, got, a.size)
        oracle.orc.orc_p32_sqrt_n(a, want, a.size)
        bad = np.nonzero(got != want)[0]
        assert bad.size == 0, [(hex(a[i]), hex(got[i]), hex(want[i])) for i in bad[:3]]
        return near

    check(rng.integers(1, 2**31, n, dtype=np.uint64))
    check(oracle.from_double(np.ldexp(rng.uniform(1, 4, n), rng.integers(-120, 119, n))))
    # squares of values half way between two posits, and their neighbours
    z = oracle.to_double(oracle.from_double(np.ldexp(rng.integers(2**10, 2**13, n) / 2.0**10, rng.integers(-58, 58, n))))
    e, fb = _fraction_bits(z)
    tie = oracle.from_double((z + np.ldexp(1.0, e - fb - 1)) ** 2)
    for by in (-1, 0, 1):
        check(_neighbours(tie, by))
    check(oracle.from_double(z * z))  # exact ones
    # as for the quotient: a = (h^2 - c) / 2^s with a small c, h odd and half way; square roots of c
    # modulo 2^s lifted from the four modulo 8
    total = 0
    for s in (29, 30):
        for c in range(-31, 33, 8):
            roots = [1, 3, 5, 7]
            for bit in range(3, s):
                roots = [x for r in roots for x in (r, r + 2**bit) if (x * x - c) % 2 ** (bit + 1) == 0]
            a = [(r * r - c) >> s for r in roots if 2**28 < r < 2**29]
            a = sorted({v for v in a if 0 < v < 2**28})
            if a:
                x = np.array(a, np.float64)
                # an even power of two away from the root's own scale
                check(oracle.from_double(x * 2.0 ** (-28 if s == 30 else -27)))
                total += check(oracle.from_double(x * 2.0 ** (-28 + s % 2)))
    assert total >= 16, total
    check(np.array([1, 2, 3, 0x7FFFFFFF, 0x7FFFFFFE, 0x40000000, 0x40000001, 0x3FFFFFFF], np.uint32))


def _panels(rng):
    for M, jb in ((1, 1), (5, 3), (40, 16), (300, 24), (130, 64)):
        yield "random", M, jb, rng.uniform(-1, 1, (jb, M))
    for M, jb in ((64, 16), (200, 24)):
        yield "ties", M, jb, rng.choice([-1.0, 1.0, 0.5, -0.5, 2.0], (jb, M))
    A = rng.uniform(-1, 1, (16, 100))
    A[5], A[:, 30] = 0, 0
    yield "zero column", 100, 16, A
    for M in (80, 1000):
        A = rng.uniform(-1, 1, (16, M))
        A[0] = 0
        A[0, 0] = np.nan
        yield "NaR over zeros", M, 16, A
    A = rng.uniform(-1, 1, (8, 90))
    A[3] = np.nan
    yield "NaR column", 90, 8, A
    yield "wide", 120, 12, rng.choice([-1, 1], (12, 120)) * 10.0 ** rng.uniform(-18, 18, (12, 120))


def test_lu_panel(hk):
    for name, M, jb, A in _panels(np.random.default_rng(4)):
        g = oracle.from_double(A.reshape(-1))
        o = g.copy()
        pg_, po = np.zeros(jb, np.int32), np.zeros(jb, np.int32)
        assert hk.hk_lu_panel(g, M, jb, pg_) == oracle.orc.orc_rgetrf2(M, jb, o, M, po), name
        assert np.array_equal(pg_, po), name
        assert np.array_equal(g, o), name


@pytest.mark.parametrize("M,jb,bad", [(1, 1, -1), (16, 16, -1), (100, 16, -1), (300, 24, -1), (257, 32, -1),
                                      (200, 32, 20), (60, 16, 0)])
def test_cholesky_panel(hk, M, jb, bad):
    rng = np.random.default_rng(M)
    X = rng.uniform(-1, 1, (M, M))
    S = X @ X.T / M + np.eye(M)
    if bad >= 0:
        S[bad, bad] = -1.0
    full = oracle.from_double(S.reshape(-1))
    panel = full[:M * jb].copy()
    info = oracle.orc.orc_rpotrf(b"L", M, full, M, jb)
    assert hk.hk_chol_panel(panel, M, jb) == info == (bad + 1 if bad >= 0 else 0)
    if bad < 0:
        low = np.arange(M)[None, :] >= np.arange(jb)[:, None]  # row c: column c
        assert np.array_equal(panel.reshape(jb, M)[low], full[:M * jb].reshape(jb, M)[low])


def test_adding_warp(hk):
    rng = np.random.default_rng(5)
    stats = np.zeros(4, np.int64)
    for trial in range(400):
        n = int(rng.choice([1, 7, 15, 16, 17, 63, 64, 65, 511, 512, 513, 700, 1500, 3000]))
        kind = trial % 8
        if kind == 0:  # calm: small terms on a large value
            q = rng.uniform(-1, 1, n) * 1e-4
        elif kind == 1:  # terms of the value's size: crossings everywhere
            q = rng.uniform(-1, 1, n)
        elif kind == 2:  # ties: terms that are odd halves of the value's spacing
            q = rng.choice([-1, 1], n) * np.ldexp(rng.choice([1.0, 3.0, 5.0], n), -28 - rng.integers(0, 3, n))
        elif kind == 3:  # near a power of two, over and back
            q = rng.choice([-1, 1], n) * 2.0 ** -rng.integers(20, 28, n)
        elif kind == 4:  # wide range
            q = rng.choice([-1, 1], n) * 10.0 ** rng.uniform(-20, 20, n)
        elif kind == 5:  # cancelling to zero
            q = np.repeat(rng.uniform(-1, 1, (n + 1) // 2), 2)[:n] * np.tile([1, -1], (n + 1) // 2)[:n]
        elif kind == 6:  # slow growth through many binades
            q = np.abs(rng.uniform(0, 1, n)) * 3
        else:  # sums below and above the fast window
            q = rng.choice([-1, 1], n) * 2.0 ** rng.choice([-118, -110, 108, 112], n)
        uq = oracle.from_double(q)
        t0 = int(oracle.from_double(np.array([[1.0, 0.0, 1.0 - 2**-27, -2.0, rng.uniform(-16, 16)][trial % 5]]))[0])
        pos = int(rng.integers(0, min(n, 40)))
        got = hk.hk_warp_chain(t0, uq, pos, n, stats)
        assert got == hk.hk_plain_chain(t0, uq, pos, n), (trial, kind, n, pos)
    assert (stats > 50).all(), stats  # whole windows, cut ones, blocks and blocks redone
