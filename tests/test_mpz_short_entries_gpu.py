"""mpz mul / addmul / submul of entries shorter than their planes (csrc/limb.cu,
k_mpz_mulops_sm): the limbs that the sizes name are what counts, in the result and in
what is read.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


@pytest.mark.parametrize("cap,longest", [(9, 1), (16, 4), (33, 5), (64, 8), (64, 63), (130, 12), (500, 3)])
@pytest.mark.parametrize("n", [1, 33, 200])
@pytest.mark.parametrize("op", ["mul", "addmul", "submul"])
def test_short_entries(g, cap, longest, n, op):
    """Lengths that differ from block to block of 32 entries, with whole blocks of zeros."""
    rng = random.Random(cap * 31 + longest + n)
    val = lambda i: 0 if (i // 32) % 3 == 1 else rng.getrandbits(32 * rng.randint(0, longest)) * rng.choice((-1, 1))
    U, V = [val(i) for i in range(n)], [val(i) for i in range(n)]
    W = [rng.getrandbits(32 * rng.randint(0, 2 * longest)) * rng.choice((-1, 1)) for _ in range(n)]
    U[-1], V[-1] = (1 << 32 * longest) - 1, 1 - (1 << 32 * longest)
    du, dv = g.DeviceMatrix.from_ints(1, n, U, cap), g.DeviceMatrix.from_ints(1, n, V, cap + 1)
    for wcap in (2 * longest + 1, 2 * cap + 2):
        dw = g.DeviceMatrix.from_ints(1, n, W, wcap)
        getattr(g, "mpz_" + op)(dw, du, dv)
        s = {"mul": (0, 1), "addmul": (1, 1), "submul": (1, -1)}[op]
        assert dw.to_ints() == [s[0] * w + s[1] * u * v for u, v, w in zip(U, V, W)]


def test_planes_above_the_sizes_are_not_read(g):
    """The same 2^20 entries of 4 limbs through views of 8 and of 64 planes: 33 MB of
    operand limbs are read either way, not 537.  (The factor of two and a half leaves room
    for a form of the kernel that the planes choose.)"""
    import torch
    n = 1 << 20
    mats = []
    for seed in (1, 2):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        m = g.DeviceMatrix(1, n, 64)
        m.limbs_t[:4 * n].random_(-2 ** 31, 2 ** 31, generator=gen)
        m.limbs_t[3 * n:4 * n] |= 1
        m.sizes_t.fill_(4)
        mats.append(m)
    dw = g.DeviceMatrix(1, n, 8)
    ms = {}
    for planes in (8, 64):
        views = []
        for m in mats:
            v = m.mat
            v.nlimbs = planes
            views.append(v)
        best = 1e9
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            g.mpz_mul(dw, *views)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        ms[planes] = best
    assert ms[64] < 2.5 * ms[8], ms


@pytest.mark.parametrize("wcap", [4, 9, 30])
def test_lengths_around_the_result_planes(g, wcap):
    """Factors of one limb more than W that cancel into it, zero products of long factors, and
    products that do not fit, which fail without touching the entries of other blocks."""
    cap, n = 40, 300
    top = (1 << 32 * wcap) - 1
    rng = random.Random(wcap)
    pool = [(1 << 32 * wcap, 1, -top), (1, -(1 << 32 * wcap), top), (top, 1, 0), (3, -5, 15), ((1 << 32 * cap) - 1, 0, -top),
            (0, (1 << 32 * cap) - 1, 7), (1 << 16, 1 << 32 * wcap - 17, 5)]
    rows = [rng.choice(pool) for _ in range(n)]
    U, V, W = (list(c) for c in zip(*rows))
    du, dv, dw = g.DeviceMatrix.from_ints(1, n, U, cap), g.DeviceMatrix.from_ints(1, n, V, cap), g.DeviceMatrix.from_ints(1, n, W, wcap)
    g.mpz_addmul(dw, du, dv)
    exp = [w + u * v for u, v, w in rows]
    assert max(abs(x) for x in exp) <= top
    assert dw.to_ints() == exp
    U[5] = V[5] = (1 << 32 * cap) - 1
    du, dv, dw = g.DeviceMatrix.from_ints(1, n, U, cap), g.DeviceMatrix.from_ints(1, n, V, cap), g.DeviceMatrix.from_ints(1, n, W, wcap)
    g.mpz_addmul(dw, du, dv)
    with pytest.raises(g.GbmmError) as e:
        dw.download()
    assert e.value.status == g.ERR_CAPACITY
    assert dw.to_ints()[128:] == exp[128:]
