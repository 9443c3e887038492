"""Signed sums with an entry's limbs split among threads (csrc/limb.cu, k_mpz_lin2) and the
vectorised mpn_add_n / mpn_sub_n (k_mpn_addsub_n_vec): segment edges, carries and borrows
through whole segments, results of either sign, in-place calls, results that do not
fit, remainders of four operands.  Integer work: exact."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _vals(rng, n, limbs):
    top = 1 << (32 * limbs)
    kinds = [lambda: rng.getrandbits(32 * limbs), lambda: top - 1, lambda: 1 << (32 * rng.randrange(limbs)),
             lambda: top - (1 << (32 * rng.randrange(limbs))), lambda: rng.getrandbits(32 * rng.randint(1, limbs)),
             lambda: 0, lambda: 1]
    return [rng.choice(kinds)() * rng.choice((-1, 1)) for _ in range(n)]


@pytest.mark.parametrize("ul,vl", [(1, 1), (7, 8), (8, 8), (9, 3), (127, 128), (128, 129), (131, 130), (500, 511),
                                   (512, 40), (600, 1023), (1023, 1023), (1100, 90)])
@pytest.mark.parametrize("sub", [False, True])
def test_mat_addsub_segments(g, ul, vl, sub):
    rng = random.Random(ul * 31 + vl + sub)
    rows, cols = 3, 37
    U, V = _vals(rng, rows * cols, ul), _vals(rng, rows * cols, vl)
    for i in range(0, len(U), 4):  # cancel down to a small value of either sign
        m = min(ul, vl)
        U[i] = rng.getrandbits(32 * m)
        V[i] = (U[i] + rng.choice((-1, 0, 1))) * (1 if sub else -1)
        if abs(V[i]) >> (32 * vl):
            V[i] = 0
    cap = max(ul, vl) + 1
    exp = [u - v if sub else u + v for u, v in zip(U, V)]
    du, dv = g.DeviceMatrix.from_ints(rows, cols, U, ul), g.DeviceMatrix.from_ints(rows, cols, V, vl)
    dw = g.DeviceMatrix.from_ints(rows, cols, [-(1 << (32 * cap - 1))] * (rows * cols), cap)
    (g.mat_sub if sub else g.mat_add)(dw, du, dv)
    assert dw.to_ints() == exp
    # in place: W = U
    duw = g.DeviceMatrix.from_ints(rows, cols, U, cap)
    (g.mpz_sub if sub else g.mpz_add)(duw, duw, dv)
    assert duw.to_ints() == exp


@pytest.mark.parametrize("u,v,cap", [((1 << 256) - 1, 1, 8), (-(1 << 256) + 1, -1, 8), (1 << 256, -1, 8)])
def test_mat_add_that_does_not_fit(g, u, v, cap):
    du, dv = g.DeviceMatrix.from_ints(1, 1, [u], 9), g.DeviceMatrix.from_ints(1, 1, [v], 9)
    dw = g.DeviceMatrix(1, 1, cap)
    g.mat_add(dw, du, dv)  # the last case: an operand longer than W is refused whatever the sum
    with pytest.raises(g.GbmmError) as e:
        dw.download()
    assert e.value.status == g.ERR_CAPACITY


@pytest.mark.parametrize("nb,n,off", [(155648, 5, 0), (155651, 1, 0), (160001, 9, 0), (155649, 4, 1)])
@pytest.mark.parametrize("sub", [False, True])
def test_mpn_addsub_n_vec(g, oracle, nb, n, off, sub):
    import torch
    rng = np.random.default_rng(nb + n + sub)
    ld = (nb + off + 3) // 4 * 4
    u = rng.integers(0, 2**32, size=(n, nb), dtype=np.uint64).astype(np.uint32)
    v = rng.integers(0, 2**32, size=(n, nb), dtype=np.uint64).astype(np.uint32)
    u[:, ::7], v[0, ::7], v[1:, ::7] = (0 if sub else 0xFFFFFFFF), 1, 0  # a carry through every limb
    exp_r, exp_c = oracle.mpn_add_n(u, v, sub=sub)

    def dev(a):
        t = torch.zeros((n, ld), dtype=torch.int32, device="cuda")
        t[:, off:off + nb] = torch.from_numpy(a.view(np.int32)).cuda()
        return t.view(-1)[off:]

    du, dv, dr = dev(u), dev(v), torch.zeros(n * ld, dtype=torch.int32, device="cuda")[off:]
    cy = torch.zeros(nb + 4, dtype=torch.int32, device="cuda")
    (g.mpn_sub_n if sub else g.mpn_add_n)(dr, du, dv, n, ld, nb, cy)
    got = torch.cat([dr, torch.zeros(off, dtype=torch.int32, device="cuda")]).cpu().numpy().view(np.uint32).reshape(n, ld)
    assert (got[:, :nb] == exp_r).all()
    assert (cy.cpu().numpy().view(np.uint32)[:nb] == exp_c).all() and not cy[nb:].any()


@pytest.mark.parametrize("rows,cols,ul,vl", [(363, 362, 3, 5), (256, 513, 6, 6)])
@pytest.mark.parametrize("sub", [False, True])
def test_mat_addsub_four_entries_per_thread(g, rows, cols, ul, vl, sub):
    """131406 and 131328 entries: the vectorised form, with a remainder of four or none."""
    rng = random.Random(rows + ul + sub)
    n = rows * cols
    U, V = _vals(rng, n, ul), _vals(rng, n, vl)
    for i in range(0, n, 5):
        V[i] = (U[i] + rng.choice((-1, 0, 1))) * (1 if sub else -1) if ul < vl else V[i]
    exp = [u - v if sub else u + v for u, v in zip(U, V)]
    du, dv = g.DeviceMatrix.from_ints(rows, cols, U, ul), g.DeviceMatrix.from_ints(rows, cols, V, vl)
    dw = g.DeviceMatrix(rows, cols, max(ul, vl) + 1)
    (g.mat_sub if sub else g.mat_add)(dw, du, dv)
    assert dw.to_ints() == exp


def test_mat_add_errors_leave_the_neighbours(g):
    rows, cols = 363, 362
    n = rows * cols
    U, V = [5] * n, [7] * n
    U[4], V[9] = 1 << 96, (1 << 64) - 1  # longer than W; a carry out of W
    U[9] = 1
    du, dv = g.DeviceMatrix.from_ints(rows, cols, U, 4), g.DeviceMatrix.from_ints(rows, cols, V, 4)
    dw = g.DeviceMatrix(rows, cols, 2)
    g.mat_add(dw, du, dv)
    with pytest.raises(g.GbmmError) as e:
        dw.download()
    assert e.value.status == g.ERR_CAPACITY
    got = dw.to_ints()
    assert [got[i] for i in range(n) if i not in (4, 9)] == [12] * (n - 2) and got[4] == 0
