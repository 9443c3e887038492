"""The block edge (4 or 8 limbs) of the batched product on chip (csrc/limb.cu,
gbmm_mpn_mul_basecase): lengths whose padding to blocks of 8 costs an SM a CTA, in batches
that fill the GPU and that do not.  Integer work: exact."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILLS = 152 * 5 * 128 + 5  # operands of a batch that fills every SM


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _operands(n, nb, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.empty((n, nb), dtype=torch.int32, device="cuda").random_(-2 ** 31, 2 ** 31, generator=gen)


@pytest.mark.parametrize("un,vn", [(96, 41), (100, 8), (61, 41), (176, 41), (104, 48)])
@pytest.mark.parametrize("nb", [33, 5000, FILLS])
def test_products(g, un, vn, nb):
    import torch
    u, v = _operands(un, nb, un), _operands(vn, nb, vn)
    r = torch.zeros((un + vn, nb), dtype=torch.int32, device="cuda")
    g.mpn_mul_basecase(r, u, un, v, vn, nb, nb)
    rng = random.Random(nb)
    val = lambda t, b: int.from_bytes(t[:, b].cpu().numpy().astype(np.int32).tobytes(), "little")
    for b in [0, nb - 1] + [rng.randrange(nb) for _ in range(30)]:
        assert val(r, b) == val(u, b) * val(v, b)


def test_shorter_products_are_not_slower(g):
    """96 x 41 limbs against 96 x 48 (a sixth more limb products): blocks of 8 would give the
    first the second's time."""
    import torch
    nb, ms = 40000, {}
    u = _operands(96, nb, 1)
    for vn in (41, 48):
        v, r = _operands(vn, nb, 2), torch.zeros((96 + vn, nb), dtype=torch.int32, device="cuda")
        best = 1e9
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(5):
                g.mpn_mul_basecase(r, u, 96, v, vn, nb, nb)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        ms[vn] = best
    assert ms[41] < 0.95 * ms[48], ms
