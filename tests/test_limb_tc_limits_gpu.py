"""The limb form's products on the tensor cores (csrc/limb_tc.cu) at the edges of what the
per-entry kernel takes: more rows than a grid dimension has blocks, and inner dimensions
that run in several chunks.  A chunk's partial sum may be longer than the result (and
than C); only the exact result has to fit, and one that does not leaves C as it was.
Integer work: exact."""
import ctypes
import random

import numpy as np
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


def _limb(g, dC, dA, dB, acc=False):
    """The product on the tensor cores, without recursion."""
    g.profile(1)
    try:
        g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE, accumulate=acc)
        assert "k_ltc_gemm" in g.profile_read()
    finally:
        g.profile(0)


@pytest.mark.parametrize("rows", [4 * 65535, 4 * 65535 + 1, 300001])
def test_rows_past_a_grid_dimension(g, rows):
    k, n = 2, 8
    rng = np.random.default_rng(rows)
    A = rng.integers(-2 ** 30, 2 ** 30, (rows, k))
    B = rng.integers(-2 ** 30, 2 ** 30, (k, n))
    dA, dB, dC = g.DeviceMatrix(rows, k, 1), g.DeviceMatrix(k, n, 1), g.DeviceMatrix(rows, n, 3)
    for d, X in ((dA, A), (dB, B)):
        x = X.reshape(-1)
        d.upload(np.abs(x).astype(np.uint32).reshape(1, -1), np.sign(x).astype(np.int32))
    _limb(g, dC, dA, dB)
    limbs, sizes = dC.download()
    mag = limbs[0].astype(np.int64) + (limbs[1].astype(np.int64) << 32)
    assert not limbs[2].any()
    assert (np.sign(sizes) * mag == (A @ B).reshape(-1)).all()
    assert (np.abs(sizes) == (limbs[0] != 0).astype(int) * (limbs[1] == 0) + 2 * (limbs[1] != 0)).all()


def _chunk(la, lb):
    """terms of one chunk: the column sums of their byte digits stay inside 32 bits"""
    return 131071 // ((4 * min(la, lb) + 15) // 16 * 16 + 2)


@pytest.mark.parametrize("la,lb", [(128, 128), (64, 64), (32, 40), (40, 16), (64, 3)])
@pytest.mark.parametrize("acc", [False, True])
def test_partial_sums_longer_than_c(g, la, lb, acc):
    """Two terms of the first chunk (and the old C) add up past C's planes, the second
    chunk's take the excess away: the result needs every limb that C has."""
    kc = _chunk(la, lb)
    M, n = kc + 3, 2
    a, b = (1 << 32 * la) - 1, (1 << 32 * lb) - 1
    row = [0] * M
    row[0] = row[kc - 1] = a
    row[kc] = -a
    if acc:
        row[M - 1] = -a
    A = row + [-v for v in row]
    B = [b] * (M * n)
    C = [a * b, a * b, -a * b, -a * b] if acc else [5] * 4  # else stale
    exp = [a * b, a * b, -a * b, -a * b]
    dA, dB = g.DeviceMatrix.from_ints(2, M, A, la), g.DeviceMatrix.from_ints(M, n, B, lb)
    dC = g.DeviceMatrix.from_ints(2, n, C, la + lb)
    _limb(g, dC, dA, dB, acc)
    assert dC.to_ints() == exp


@pytest.mark.parametrize("la,lb", [(128, 128), (32, 40), (64, 3)])
@pytest.mark.parametrize("at", [0, -1])
@pytest.mark.parametrize("acc", [False, True])
def test_result_that_does_not_fit_leaves_c(g, la, lb, at, acc):
    """Four terms of one sign, in the first or in the last chunk; the other entries are written."""
    kc = _chunk(la, lb)
    M, n = 2 * kc + 5, 2
    a, b = (1 << 32 * la) - 1, (1 << 32 * lb) - 1
    A = [0] * M + [0] * M
    A[0:4] = [a] * 4
    if at:
        A[0:M] = A[0:M][::-1]
    A[M] = A[2 * M - 1] = 3
    dA, dB = g.DeviceMatrix.from_ints(2, M, A, la), g.DeviceMatrix.from_ints(M, n, [b] * (M * n), lb)
    dC = g.DeviceMatrix.from_ints(2, n, [7, -9, 11, 0], la + lb)
    g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE, accumulate=acc)
    with pytest.raises(g.GbmmError) as e:
        dC.download()
    assert e.value.status == g.ERR_CAPACITY
    old = [11, 0] if acc else [0, 0]
    assert dC.to_ints() == [7, -9, old[0] + 6 * b, old[1] + 6 * b]


@pytest.mark.parametrize("K,M,N,la,lb", [(2, 3 * 255 + 1, 3, 128, 127), (9, 2 * 1985 + 7, 3, 16, 16), (1, 2, 5, 16, 16),
                                         (3, 2 * 1008, 129, 32, 31), (17, 7282, 2, 4, 3)])
@pytest.mark.parametrize("acc", [False, True])
def test_many_chunks(g, K, M, N, la, lb, acc):
    rng = random.Random(K + M + N)
    top = lambda n: (1 << 32 * n) - 1
    pick = lambda n: rng.choice((top(n), top(n), rng.getrandbits(32 * n), 1)) * rng.choice((-1, 1))
    A, B = [pick(la) for _ in range(K * M)], [pick(lb) for _ in range(M * N)]
    C = [pick(la + lb) if acc else 0 for _ in range(K * N)]
    exp = [C[y * N + x] + sum(A[y * M + k] * B[k * N + x] for k in range(M)) for y in range(K) for x in range(N)]
    cn = max(1, max((abs(v).bit_length() + 31) // 32 for v in exp + C))
    dA, dB = g.DeviceMatrix.from_ints(K, M, A, la), g.DeviceMatrix.from_ints(M, N, B, lb)
    dC = g.DeviceMatrix.from_ints(K, N, C, cn)
    _limb(g, dC, dA, dB, acc)
    assert dC.to_ints() == exp


def test_carries_of_many_chunks(g):
    """260 chunks of the largest column sums (every digit 127): a segment's carry passes 32 bits."""
    nl = 128
    K = 260 * _chunk(nl, nl)
    v = int.from_bytes(b"\x7f" * (4 * nl), "little")
    dA, dB, dC = g.DeviceMatrix(1, K, nl), g.DeviceMatrix(K, 1, nl), g.DeviceMatrix(1, 1, 2 * nl + 1)
    for d in (dA, dB):
        d.limbs_t.fill_(0x7f7f7f7f)
        d.sizes_t.fill_(nl)
    _limb(g, dC, dA, dB)
    assert dC.to_ints() == [K * v * v]
