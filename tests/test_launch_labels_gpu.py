"""gbmm_profile names the kernels that ran: the one-kernel residues, and the three forms of
an elementwise signed sum."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _ran(g, fn):
    g.profile(1)
    fn()
    ran = set(g.profile_read())
    g.profile(0)
    return ran


@pytest.mark.parametrize("limbs,names", [(128, {"k_crt_residue2"}), (129, {"k_crt_digits", "k_crt_residue"})])
def test_residues(g, limbs, names):
    n = 32
    A, B = [3] * n * n, [5] * n * n
    dA, dB = g.DeviceMatrix.from_ints(n, n, A, limbs), g.DeviceMatrix.from_ints(n, n, B, limbs)
    dC = g.DeviceMatrix(n, n, 4)
    ran = _ran(g, lambda: g.default_handle().matmul(dC, dA, dB, path=g.PATH_CRT))
    assert ran == names | {"k_crt_product", "k_crt_recon"}
    assert dC.to_ints() == [15 * n] * (n * n)


@pytest.mark.parametrize("cols,limbs,pad,name", [(80 * 1024, 3, 0, "k_mpz_addsub_vec"), (1000, 3, 0, "k_mpz_lin2"),
                                                 (80 * 1024, 3, 1, "k_mpz_lin2"), (40, 1100, 0, "k_mpz_addsub")])
def test_signed_sums(g, cols, limbs, pad, name):
    """pad: a plane stride that is no multiple of four entries (no 16-byte loads)."""
    mats = [g.DeviceMatrix.from_ints(1, cols + pad, [v] * (cols + pad), limbs) for v in (-7, 20, 0)]
    views = [m.view(0, 0, 1, cols) for m in mats]
    for v in views:
        v.rs = cols
    assert _ran(g, lambda: g.mpz_add(views[2], views[0], views[1])) == {name}
    assert mats[2].to_ints() == [13] * cols + [0] * pad
