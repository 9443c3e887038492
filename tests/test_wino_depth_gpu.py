"""The depth that Winograd's tree runs to (csrc/limb_tc.cu, ltc_wino_levels) and the form of
its leaves, read from the launches: one launch of the sums and one of the combinations a
level.  The cutoff's depth with the tensor cores off, fewer levels and leaves on the
tensor cores where the estimate says so, the cutoff's where it does not.  Integer work: exact."""
import ctypes
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


@pytest.mark.parametrize("N,limbs,cutoff,full,levels,tensor", [(64, 16, 16, 2, 1, True), (128, 32, 32, 2, 1, True), (256, 3, 32, 3, 1, True),
                                                               (128, 8, 16, 3, 1, True), (16, 4, 8, 1, 1, False)])
def test_levels_and_leaves(g, N, limbs, cutoff, full, levels, tensor):
    rng = random.Random(N + limbs)
    A, B = ([rng.getrandbits(32 * limbs) * rng.choice((-1, 1)) for _ in range(N * N)] for _ in range(2))
    dA, dB = g.DeviceMatrix.from_ints(N, N, A, limbs), g.DeviceMatrix.from_ints(N, N, B, limbs)
    f = g.lib().gbmmx_limb_tc
    f.argtypes, f.restype = [ctypes.c_int32], ctypes.c_int32
    got = []
    for mode, depth, gemm in ((-1, levels, tensor), (0, full, False)):
        dC = g.DeviceMatrix(N, N, g.limbs_needed(limbs, limbs, N, cutoff=cutoff))
        old = f(mode)
        g.profile(1)
        try:
            g.default_handle().matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_WINOGRAD, cutoff=cutoff)
            ran = g.profile_read()
        finally:
            g.profile(0)
            f(old)
        assert ran["k_wino_sums"][0] == ran["k_wino_combine"][0] == depth, (mode, ran)
        assert ("k_ltc_gemm" in ran) == gemm, (mode, ran)
        got.append(dC.to_ints())
    assert got[0] == got[1]
    for _ in range(32):
        y, x = rng.randrange(N), rng.randrange(N)
        assert got[0][y * N + x] == sum(A[y * N + k] * B[k * N + x] for k in range(N))
