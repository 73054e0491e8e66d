"""The GEMM's routes on both sides of every tile edge, against the oracle bit for bit.
Separate operands take the fused route (32x32 tiles, or 64x32 where they are many) but
for the one size beyond 2^24 multiply-adds, which is staged; so are A, B and C inside one matrix,
whose address ranges meet (64x64 tiles of 32-row blocks, an odd count of blocks among them)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (31, 33, 15), (32, 32, 16), (33, 65, 17), (64, 64, 33), (97, 95, 48), (65, 2400, 20),
         (1500, 640, 18), (1217, 1100, 19), (1153, 1089, 7), (4000, 100, 9)]


def _values(rng, numel, kind):
    x = rng.uniform(-1, 1, numel)
    if kind == "wide":
        x = np.sign(x) * 10.0 ** rng.uniform(-20, 20, numel)
    u = oracle.from_double(x)
    if kind == "nar":
        u[rng.integers(0, numel, 2)] = oracle.P32_NAR
    return u


@pytest.mark.parametrize("kind", ["uniform", "wide", "nar"])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T")])
@pytest.mark.parametrize("staged", [False, True])
def test_routes_match_oracle(cuda_ok, staged, ta, tb, kind):
    import torch

    import posit_gpu_b200 as pg
    rng = np.random.default_rng(7 + 10 * staged)
    alphas = [oracle.P32_ONE, oracle.P32_MINUS_ONE, oracle.p32(0.7)]
    for i, (m, n, k) in enumerate(SIZES):
        if kind != "uniform" and m * n * k > 10_000_000:
            continue
        ra, ca = (m, k) if ta == "N" else (k, m)
        rb, cb = (k, n) if tb == "N" else (n, k)
        ld = max(ra, rb, m)
        whole = _values(rng, ld * (ca + cb + n), kind)
        alpha, beta = alphas[i % 3], [oracle.P32_ONE, 0, oracle.p32(0.5)][i % 3]
        oA, oB, oC = 0, ld * ca, ld * (ca + cb)
        want = whole.copy()
        assert oracle.rgemm(ta, tb, m, n, k, alpha, whole[oA:oB], ld, whole[oB:oC], ld, beta, want[oC:], ld) == 0
        if staged:
            # interleave: rows of C between the columns of A, so that the ranges meet
            big = ra + m
            AC = np.zeros(big * max(ca, n), np.uint32)
            for j in range(ca):
                AC[j * big:j * big + ra] = whole[oA + j * ld:oA + j * ld + ra]
            for j in range(n):
                AC[j * big + ra:j * big + ra + m] = whole[oC + j * ld:oC + j * ld + m]
            dAC = torch.from_numpy(AC.view(np.int32)).cuda()
            dB = torch.from_numpy(whole[oB:oC].view(np.int32).copy()).cuda()
            pg.Rgemm_dev(ta, tb, m, n, k, alpha, dAC, big, dB, ld, beta, dAC[ra:], big)
            out = dAC.cpu().numpy().view(np.uint32)
            got = np.concatenate([out[j * big + ra:j * big + ra + m] for j in range(n)])
        else:
            d = [torch.from_numpy(whole[a:b].view(np.int32).copy()).cuda() for a, b in ((oA, oB), (oB, oC), (oC, None))]
            pg.Rgemm_dev(ta, tb, m, n, k, alpha, d[0], ld, d[1], ld, beta, d[2], ld)
            out = d[2].cpu().numpy().view(np.uint32)
            got = np.concatenate([out[j * ld:j * ld + m] for j in range(n)])
        ref = np.concatenate([want[oC + j * ld:oC + j * ld + m] for j in range(n)])
        assert np.array_equal(got, ref), (m, n, k, alpha, beta)
        assert pg.device_error() == 0
