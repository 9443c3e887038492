"""Winograd trees that stop above the cutoff where the tensor cores take larger leaves faster
(csrc/limb_tc.cu, ltc_wino_levels): one and several levels, leaves of odd and of 128 columns, results
with as few limbs as they need, against the CUDA-core tree of full depth and exact
products.  Integer work: exact."""
import ctypes
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


@pytest.mark.parametrize("N,bits,cutoff,extra", [(64, 512, 16, 1), (64, 1000, 8, 1), (60, 700, 15, 0), (72, 640, 9, 1),
                                                 (128, 300, 32, 0), (256, 64, 16, 1)])
def test_fewer_levels(g, N, bits, cutoff, extra):
    rng = random.Random(N + bits)
    top = (1 << bits) - 1
    kinds = [lambda: rng.getrandbits(bits), lambda: top, lambda: rng.getrandbits(rng.randint(1, bits)), lambda: 0]
    A = [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(N * N)]
    B = [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(N * N)]
    for i in range(N):  # a row and a column of extremes: the largest entry
        A[i] = -top
        B[i * N] = top
    nl = (bits + 31) // 32
    need = -(-(2 * bits + N.bit_length()) // 32)
    dA, dB = g.DeviceMatrix.from_ints(N, N, A, nl), g.DeviceMatrix.from_ints(N, N, B, nl)
    f = g.lib().gbmmx_limb_tc
    f.argtypes, f.restype = [ctypes.c_int32], ctypes.c_int32
    got = []
    for mode in (-1, 0):
        old = f(mode)
        try:
            dC = g.DeviceMatrix(N, N, need + extra)
            g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_WINOGRAD, cutoff=cutoff)
        finally:
            f(old)
        got.append(dC.to_ints())
    assert got[0] == got[1]
    for y, x in [(0, 0), (0, N - 1), (N - 1, 0)] + [(rng.randrange(N), rng.randrange(N)) for _ in range(64)]:
        assert got[0][y * N + x] == sum(A[y * N + k] * B[k * N + x] for k in range(N))


@pytest.mark.parametrize("limbs", [46, 47, 66, 67, 94, 95, 96, 134, 135, 136, 137, 270, 271, 272, 400])
def test_sums_and_combinations_by_length(g, limbs):
    """Sums and combinations with their limbs split among threads: blocks of 32, 16 and 8
    entries at the edges of their ranges, carries and borrows through whole segments."""
    N, bits = 6, 32 * limbs
    rng = random.Random(limbs)
    top = (1 << bits) - 1
    kinds = [lambda: rng.getrandbits(bits), lambda: top, lambda: 1 << (32 * rng.randrange(limbs)), lambda: 0,
             lambda: top - (1 << (32 * rng.randrange(limbs))), lambda: 1]
    A = [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(N * N)]
    B = [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(N * N)]
    dA, dB = g.DeviceMatrix.from_ints(N, N, A, limbs), g.DeviceMatrix.from_ints(N, N, B, limbs)
    dC = g.DeviceMatrix(N, N, 2 * limbs + 1)
    g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_WINOGRAD, cutoff=3)
    assert dC.to_ints() == [sum(A[y * N + k] * B[k * N + x] for k in range(N)) for y in range(N) for x in range(N)]
