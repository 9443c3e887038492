"""Per-entry products of few entries of 3 to 8 limbs, cut into 2 x 2 limb blocks (csrc/limb.cu,
choose_mm_for): every pair of lengths, thin top limbs, both sides of the line at 4096 entries,
C += A B, and Winograd leaves.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _vals(rng, n, limbs):
    top = (1 << (32 * limbs)) - 1
    kinds = [lambda: rng.getrandbits(32 * limbs), lambda: top, lambda: rng.getrandbits(rng.randint(1, 32 * limbs)),
             lambda: 1 << (32 * limbs - 1), lambda: 0, lambda: 1]
    return [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(n)]


def _case(g, m, k, n, la, lb, accumulate=False, **opts):
    rng = random.Random(m + 3 * k + 5 * n + 7 * la + 11 * lb)
    A, B, C = _vals(rng, m * k, la), _vals(rng, k * n, lb), _vals(rng, m * n, la + lb)
    dA, dB = g.DeviceMatrix.from_ints(m, k, A, la), g.DeviceMatrix.from_ints(k, n, B, lb)
    dC = g.DeviceMatrix.from_ints(m, n, C, la + lb + 2)
    g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, accumulate=accumulate, **opts)
    assert dC.to_ints() == [(C[y * n + x] if accumulate else 0) + sum(A[y * k + i] * B[i * n + x] for i in range(k))
                            for y in range(m) for x in range(n)]


@pytest.mark.parametrize("la", range(1, 9))
@pytest.mark.parametrize("lb", range(1, 9))
def test_lengths(g, la, lb):
    _case(g, 5, 19, 7, la, lb, accumulate=(la + lb) % 2 == 1, method=g.METHOD_NAIVE)


@pytest.mark.parametrize("m,n", [(64, 64), (17, 241), (1, 4096), (1, 1)])
@pytest.mark.parametrize("la,lb", [(4, 3), (8, 8), (5, 7)])
def test_line(g, m, n, la, lb):
    _case(g, m, 3, n, la, lb, method=g.METHOD_NAIVE)


def test_winograd_leaves(g):
    _case(g, 16, 16, 16, 6, 7, method=g.METHOD_WINOGRAD, cutoff=4)
