"""A batch takes a limb plan from the tuning table only where the table's time is one
that a batch can reach: gbmm_autotune times products one by one, and a single product's
limb form may run on the tensor cores, a batch's does not."""
import math
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _key(*dims):
    key = 0
    for d in dims:
        key = key << 8 | (0 if d <= 1 else round(math.log2(d)))
    return key


@pytest.mark.parametrize("n,limbs,plan,reached", [(128, 16, 0, False), (128, 32, 1, False), (16, 4, 0, True),
                                                  (24, 8, 0, True)])
def test_batch_plans_from_the_table(g, n, limbs, plan, reached, tmp_path):
    rng = random.Random(n + limbs)
    A, B = ([rng.getrandbits(32 * limbs) * rng.choice((-1, 1)) for _ in range(n * n)] for _ in range(2))
    dA, dB = g.DeviceMatrix.from_ints(n, n, A, limbs), g.DeviceMatrix.from_ints(n, n, B, limbs)
    dC = g.DeviceMatrix(n, n, 2 * limbs + 4)
    table = tmp_path / "tune.json"
    table.write_text('[\n  {"key": %d, "plan": %d, "ms": 0.01}\n]\n' % (_key(n, n, n, limbs, limbs), plan))
    h = g.Handle()
    assert g.lib().gbmm_tune_load(h.h, str(table).encode()) == g.OK
    # one product runs the table's plan as the table timed it
    g.profile(1)
    h.matmul(dC, dA, dB)
    ran = g.profile_read()
    g.profile(0)
    assert ("k_ltc_gemm" in ran) == (not reached) and not any(k.startswith("k_crt") for k in ran)
    one = dC.to_ints()
    arr = h.jobs([(dC, dA, dB)])
    (_, chosen), = h.matmul_batched(arr, plans=True)
    assert chosen == (plan if reached else g.PLAN_CRT)
    assert dC.to_ints() == one
    for _ in range(20):
        y, x = rng.randrange(n), rng.randrange(n)
        assert one[y * n + x] == sum(A[y * n + k] * B[k * n + x] for k in range(n))
    h.close()
