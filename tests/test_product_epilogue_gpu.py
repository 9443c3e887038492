"""The product GEMM's epilogue (csrc/crt.cu, k_crt_product): inner dimensions around the line
(448) past which the middle sum is reduced first, one-CTA and paired tiles, ragged rows and columns,
with entries whose residues' digits are large and of one sign.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _primes(n):
    out, c = [], 65535
    while len(out) < n:
        if all(c % d for d in range(3, 256, 2)):
            out.append(c)
        c -= 2
    return out


@pytest.mark.parametrize("k", [1, 63, 64, 65, 447, 448, 449, 511, 512])
@pytest.mark.parametrize("m,n", [(3, 5), (130, 66)])
def test_middle_sum_bound(g, k, m, n):
    rng = random.Random(k * 5 + m)
    ps = _primes(6)
    # residues near -p/2 and p/2: digits 128 * 256 + (-128 .. 127), for as many moduli as fit
    mod = 1
    for p in ps[:4]:
        mod *= p

    def crt(rs):
        v = 0
        for p, r in zip(ps, rs):
            q = mod // p
            v += r * q * pow(q, -1, p)
        return v % mod

    ext = [crt([(s * (p // 2 - d)) % p for p in ps[:4]]) for s in (1, -1) for d in (0, 1, 127, 128)]
    A = [rng.choice(ext) * rng.choice((1, 1, -1)) for _ in range(m * k)]
    B = [rng.choice(ext) * rng.choice((1, 1, -1)) for _ in range(k * n)]
    dA, dB = g.DeviceMatrix.from_ints(m, k, A, 2), g.DeviceMatrix.from_ints(k, n, B, 2)
    dC = g.DeviceMatrix(m, n, 6)
    g.default_handle().matmul(dC, dA, dB, path=g.PATH_CRT)
    assert dC.to_ints() == [sum(A[y * k + i] * B[i * n + x] for i in range(k)) for y in range(m) for x in range(n)]
