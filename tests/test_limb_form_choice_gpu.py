"""Which form a limb product takes by the estimate (csrc/limb_tc.cu, ltc_pays): few terms and long
entries, where the tensor form's last kernel alone takes longer than the CUDA cores do, stay on
the CUDA cores; sums long enough run on the tensor cores.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


@pytest.mark.parametrize("m,k,n,la,lb,tensor", [
    (16, 20, 64, 128, 16, False), (2, 1, 441, 136, 121, False), (11, 4, 60, 108, 102, False), (64, 1, 64, 128, 16, False),
    (16, 4, 512, 8, 8, False), (128, 128, 128, 16, 16, True), (64, 64, 64, 33, 33, True), (238, 3, 415, 9, 2, True),
    (16, 512, 64, 128, 16, True)])
def test_form(g, m, k, n, la, lb, tensor):
    rng = random.Random(m + k + n + la)
    A = [rng.getrandbits(32 * la) * rng.choice((-1, 1)) for _ in range(m * k)]
    B = [rng.getrandbits(32 * lb) * rng.choice((-1, 1)) for _ in range(k * n)]
    dA, dB = g.DeviceMatrix.from_ints(m, k, A, la), g.DeviceMatrix.from_ints(k, n, B, lb)
    dC = g.DeviceMatrix(m, n, la + lb + 1)
    g.profile(1)
    g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE)
    ran = g.profile_read()
    g.profile(0)
    assert ("k_ltc_gemm" in ran) == tensor, ran
    got = dC.to_ints()
    for _ in range(60):
        y, x = rng.randrange(m), rng.randrange(n)
        assert got[y * n + x] == sum(A[y * k + i] * B[i * n + x] for i in range(k))
