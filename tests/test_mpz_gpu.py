"""mpz mul / addmul / submul with the operands staged on chip (csrc/limb.cu,
k_mpz_mulops_sm) against Python integers: lengths around the 4-limb blocks, short and zero
entries, results of either sign around zero, strided views (no 16-byte loads), results
that do not fit, and operands too long to stage.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _vals(rng, n, limbs):
    return [0 if rng.random() < 0.1 else rng.getrandbits(32 * rng.randint(1, limbs)) * rng.choice((-1, 1))
            for _ in range(n)]


@pytest.mark.parametrize("ul,vl,rows,cols", [(1, 1, 1, 1), (2, 4, 9, 31), (1, 9, 5, 33), (3, 3, 4, 40), (3, 5, 7, 19), (4, 4, 16, 16), (16, 16, 5, 129),
                                             (17, 2, 9, 67), (40, 33, 3, 50), (700, 3, 2, 33), (1200, 1200, 1, 3)])
@pytest.mark.parametrize("op", ["mul", "addmul", "submul"])
@pytest.mark.parametrize("view", [False, True])
def test_mpz_mulops_on_chip(g, ul, vl, rows, cols, op, view):
    rng = random.Random(ul * 100 + vl + rows + cols + len(op) + view)
    n = rows * cols
    U, V = _vals(rng, n, ul), _vals(rng, n, vl)
    U[0], V[0] = (1 << (32 * ul)) - 1, -((1 << (32 * vl)) - 1)
    W = _vals(rng, n, ul + vl)
    for i in range(0, n, 3):  # w close to -(u v) or u v
        W[i] = U[i] * V[i] * (1 if op == "submul" else -1) + rng.choice((-1, 0, 1))
    cap = ul + vl + 1

    def mat(vals, nl):
        if not view:
            m = g.DeviceMatrix.from_ints(rows, cols, vals, nl)
            return m, m.mat
        big = [0] * ((rows + 1) * (cols + 3))
        for r in range(rows):
            for c in range(cols):
                big[(r + 1) * (cols + 3) + c + 1] = vals[r * cols + c]
        m = g.DeviceMatrix.from_ints(rows + 1, cols + 3, big, nl)
        return m, m.view(1, 1, rows, cols)

    (mu, du), (mv, dv), (mw, dw) = mat(U, ul), mat(V, vl), mat(W, cap)
    getattr(g, "mpz_" + op)(dw, du, dv)
    got = mw.to_ints()
    if view:
        got = [got[(r + 1) * (cols + 3) + c + 1] for r in range(rows) for c in range(cols)]
    s = {"mul": (0, 1), "addmul": (1, 1), "submul": (1, -1)}[op]
    assert got == [s[0] * w + s[1] * u * v for u, v, w in zip(U, V, W)]


@pytest.mark.parametrize("w,ok", [(0, False), (-1, True), (1, False)])
def test_mpz_addmul_result_at_the_capacity(g, w, ok):
    # u v + w against 4 limbs: 2^128 does not fit, 2^128 - 1 does
    du, dv = g.DeviceMatrix.from_ints(1, 1, [1 << 64], 3), g.DeviceMatrix.from_ints(1, 1, [1 << 64], 3)
    dw = g.DeviceMatrix.from_ints(1, 1, [w], 4)
    g.mpz_addmul(dw, du, dv)
    if ok:
        assert dw.to_ints() == [(1 << 128) + w]
    else:
        with pytest.raises(g.GbmmError) as e:
            dw.download()
        assert e.value.status == g.ERR_CAPACITY
