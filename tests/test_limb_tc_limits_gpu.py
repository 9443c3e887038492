"""The limb form's products on the tensor cores (csrc/limb_tc.cu) at the edges of what the
per-entry kernel takes: more rows than a grid dimension has blocks.  Integer work: exact."""
import ctypes

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
