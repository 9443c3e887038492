"""The limb form's products on the tensor cores (csrc/limb_tc.cu) against Python
integers: tiles of several rows and of several column windows, remainders in every
dimension, exact accumulation at the largest digit sums, chunks of the inner
dimension, C += A*B, strided views and results that do not fit.  Integer work: exact."""
import ctypes
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    f = gbmm.lib().gbmmx_limb_tc
    f.argtypes, f.restype = [ctypes.c_int32], ctypes.c_int32
    old = f(1)
    yield gbmm
    f(old)


def _vals(rng, n, bits, kind):
    if kind == "ones":
        return [((1 << bits) - 1) * rng.choice((-1, 1)) for _ in range(n)]
    if kind == "max":  # one sign: the columns add up
        return [(1 << bits) - 1] * n
    return [0 if rng.random() < 0.1 else rng.getrandbits(rng.choice((bits, max(1, bits // 3)))) * rng.choice((-1, 1))
            for _ in range(n)]


def _ref(K, M, N, A, B, C=None):
    return [(C[y * N + x] if C else 0) + sum(A[y * M + k] * B[k * N + x] for k in range(M))
            for y in range(K) for x in range(N)]


def _gemm_ran(g, fn):
    g.profile(1)
    fn()
    ran = "k_ltc_gemm" in g.profile_read()
    g.profile(0)
    return ran


@pytest.mark.parametrize("K,M,N,ba,bb,kind", [
    (1, 1, 1, 32, 32, "max"), (9, 5, 3, 1, 64, "rand"), (17, 16, 129, 128, 128, "rand"), (5, 40, 7, 256, 250, "ones"),
    (3, 33, 130, 512, 512, "ones"), (7, 31, 20, 513, 480, "rand"), (4, 60, 33, 1024, 1024, "max"),
    (4, 19, 9, 1056, 1057, "rand"), (3, 70, 128, 2048, 2048, "max"), (2, 9, 257, 96, 2080, "rand"),
    (6, 9, 40, 2080, 96, "rand"), (2, 300, 3, 4096, 4096, "max"), (2, 21, 6, 4128, 1000, "ones"),
])
@pytest.mark.parametrize("acc", [False, True])
def test_limb_tc_product(g, K, M, N, ba, bb, kind, acc):
    rng = random.Random(K * 7919 + M * 31 + N + ba + bb)
    A, B = _vals(rng, K * M, ba, kind), _vals(rng, M * N, bb, kind)
    la, lb = (ba + 31) // 32, (bb + 31) // 32
    dA, dB = g.DeviceMatrix.from_ints(K, M, A, la), g.DeviceMatrix.from_ints(M, N, B, lb)
    C = _vals(rng, K * N, ba + bb, "rand") if acc else None
    cn = la + lb + 2
    if acc:
        dC = g.DeviceMatrix.from_ints(K, N, C, cn)
    else:
        dC = g.DeviceMatrix.from_ints(K, N, [-1 << (32 * cn - 40)] * (K * N), cn)  # stale limbs
    h = g.default_handle()
    ran = _gemm_ran(g, lambda: h.matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE, accumulate=acc))
    assert ran
    assert dC.to_ints() == _ref(K, M, N, A, B, C)


def test_limb_tc_views_and_cancellation(g):
    rng = random.Random(5)
    K, M, N, bits = 11, 13, 21, 700
    A, B = _vals(rng, K * M, bits, "rand"), _vals(rng, M * N, bits, "rand")
    dA, dB = g.DeviceMatrix.from_ints(K, M, A, 22), g.DeviceMatrix.from_ints(M, N, B, 22)
    sub = lambda X, cols, r0, c0, r, c: [X[(r0 + i) * cols + c0 + j] for i in range(r) for j in range(c)]
    a, b = sub(A, M, 2, 1, 7, 9), sub(B, N, 1, 3, 9, 14)
    # C holds -(A B) and a little more: results of either sign close to zero
    c = [-v + rng.choice((-1, 0, 1, 1 << 40)) for v in _ref(7, 9, 14, a, b)]
    big = [0] * (20 * 30)
    for i in range(7):
        for j in range(14):
            big[(3 + i) * 30 + 5 + j] = c[i * 14 + j]
    dC = g.DeviceMatrix.from_ints(20, 30, big, 46)
    h = g.default_handle()
    h.matmul(dC.view(3, 5, 7, 14), dA.view(2, 1, 7, 9), dB.view(1, 3, 9, 14), path=g.PATH_LIMB, method=g.METHOD_NAIVE,
             accumulate=True)
    got = dC.to_ints()
    exp = _ref(7, 9, 14, a, b, c)
    for i in range(20):
        for j in range(30):
            inside = 3 <= i < 10 and 5 <= j < 19
            assert got[i * 30 + j] == (exp[(i - 3) * 14 + j - 5] if inside else 0)


def test_limb_tc_result_that_does_not_fit(g):
    A, B = [(1 << 512) - 1] * 16, [(1 << 512) - 1] * 16
    dA, dB = g.DeviceMatrix.from_ints(4, 4, A, 16), g.DeviceMatrix.from_ints(4, 4, B, 16)
    dC = g.DeviceMatrix(4, 4, 32)  # the sum of four products needs 1026 bits
    g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE)
    with pytest.raises(g.GbmmError) as e:
        dC.download()
    assert e.value.status == g.ERR_CAPACITY


@pytest.mark.parametrize("N,cutoff,bits", [(64, 16, 700), (96, 24, 1024), (66, 33, 130), (8, 4, 1600), (8, 4, 2400)])
def test_limb_tc_winograd_leaves(g, N, cutoff, bits):
    """Leaves on the tensor cores; sums and combinations in segments of an entry's limbs
    (up to 96, up to 136 limbs) and one thread per entry (longer)."""
    rng = random.Random(N + bits)
    A, B = _vals(rng, N * N, bits, "ones"), _vals(rng, N * N, bits, "rand")
    nl = (bits + 31) // 32
    dA, dB = g.DeviceMatrix.from_ints(N, N, A, nl), g.DeviceMatrix.from_ints(N, N, B, nl)
    cn = g.limbs_needed(nl, nl, N, method=g.METHOD_WINOGRAD, cutoff=cutoff)
    d1, d2 = g.DeviceMatrix(N, N, cn), g.DeviceMatrix(N, N, cn)
    assert _gemm_ran(g, lambda: g.mat_mul_winograd(N, d1, dA, dB, cutoff=cutoff))
    f = g.lib().gbmmx_limb_tc
    f(0)
    assert not _gemm_ran(g, lambda: g.mat_mul(N, N, N, d2, dA, dB))
    f(1)
    assert d1.to_ints() == d2.to_ints()
