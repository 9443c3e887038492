"""Digits and residues in one kernel (csrc/crt.cu, k_crt_residue2): rows of one to eight
64-digit slots, ragged columns and plane rows, one and several column tiles, more units than
CTA pairs, operands of different lengths, one operand only, limb halves read in place,
grouped launches, and the line past which the two-kernel form is taken.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _vals(rng, n, bits):
    kinds = [lambda: rng.getrandbits(bits), lambda: (1 << bits) - 1, lambda: rng.getrandbits(rng.randint(1, bits)),
             lambda: 1 << (bits - 1), lambda: 0, lambda: 1]
    return [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(n)]


def _exact(A, B, m, k, n):
    return [sum(A[y * k + i] * B[i * n + x] for i in range(k)) for y in range(m) for x in range(n)]


@pytest.mark.parametrize("m,k,n,ba,bb", [
    (1, 1, 1, 40, 40), (3, 5, 2, 512, 512), (8, 32, 8, 513, 1024), (9, 33, 7, 1500, 1025), (16, 31, 17, 2048, 2049),
    (5, 64, 40, 2560, 3000), (33, 21, 9, 3584, 3585), (7, 63, 65, 4095, 4096), (64, 64, 64, 1024, 1024),
    (2, 96, 3, 4096, 4097), (11, 40, 5, 6000, 900), (96, 100, 90, 300, 260), (130, 200, 120, 64, 4096),
    # padding: 8 x the entries in two kernels' and one kernel's range, one side each, 5.3 x
    (2200, 4, 2, 600, 500), (2, 4, 2200, 500, 600), (2040, 4, 3, 600, 500), (1, 1700, 1, 300, 2000), (2800, 6, 2, 200, 90)])
def test_products(g, m, k, n, ba, bb):
    rng = random.Random(m * 7 + k * 11 + n * 13 + ba + bb)
    A, B = _vals(rng, m * k, ba), _vals(rng, k * n, bb)
    la, lb = (ba + 31) // 32, (bb + 31) // 32
    dA, dB = g.DeviceMatrix.from_ints(m, k, A, la), g.DeviceMatrix.from_ints(k, n, B, lb)
    dC = g.DeviceMatrix(m, n, la + lb + 1)
    for _ in range(2):  # the second run finds the first's planes in the workspace
        g.default_handle().matmul(dC, dA, dB, path=g.PATH_CRT)
    assert dC.to_ints() == _exact(A, B, m, k, n)


@pytest.mark.parametrize("m,k,n,ba,bb", [(24, 16, 40, 20000, 4000), (40, 16, 24, 4000, 20000), (24, 20, 33, 19000, 2500)])
def test_operand_split_in_place(g, m, k, n, ba, bb):
    rng = random.Random(ba * 3 + bb)
    A, B = _vals(rng, m * k, ba), _vals(rng, k * n, bb)
    la, lb = (ba + 31) // 32, (bb + 31) // 32
    dA, dB = g.DeviceMatrix.from_ints(m, k, A, la), g.DeviceMatrix.from_ints(k, n, B, lb)
    dC = g.DeviceMatrix(m, n, la + lb + 1)
    g.default_handle().matmul(dC, dA, dB)
    assert dC.to_ints() == _exact(A, B, m, k, n)
