"""A batch's grouped reconstructions (csrc/crt.cu, crt_group_launch): products by base-256 tables
(up to 940 moduli) and by base-128 ones (up to 1023), directly and as limb-half splits joined
afterwards, alone and in every mixture, the two forms side by side on two streams.  Eager call,
capturing call, replays, each with new inputs.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu

DIRECT256, DIRECT128 = [(12, 9, 7, 4000, 4000), (40, 3, 33, 900, 64)], [(12, 9, 7, 8000, 8000), (3, 20, 50, 15400, 200)]
SPLIT256, SPLIT128 = [(10, 6, 9, 20000, 4000)], [(8, 5, 11, 20000, 5600), (30, 4, 3, 5600, 20000)]


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


@pytest.mark.parametrize("specs", [DIRECT128, SPLIT128, DIRECT256 + DIRECT128, DIRECT256 + SPLIT128, SPLIT256 + DIRECT128,
                                   SPLIT256 + SPLIT128, DIRECT256 + SPLIT256, DIRECT256 + DIRECT128 + SPLIT256 + SPLIT128])
def test_forms(g, specs):
    import torch
    rng = random.Random(len(specs) * 7 + specs[0][3])
    val = lambda bits: rng.choice((rng.getrandbits(bits), (1 << bits) - 1, rng.getrandbits(rng.randint(1, bits)), 0)) * rng.choice((-1, 1))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        h = g.Handle()
        mats = []
        for m, k, n, ba, bb in specs:
            la, lb = (ba + 31) // 32, (bb + 31) // 32
            mats.append((g.DeviceMatrix(m, k, la), g.DeviceMatrix(k, n, lb), g.DeviceMatrix(m, n, la + lb + 1)))
        jobs = h.jobs([(c, a, b) for a, b, c in mats], path=g.PATH_CRT)
        for call in range(4):
            exp = []
            for (m, k, n, ba, bb), (a, b, c) in zip(specs, mats):
                A, B = [val(ba) for _ in range(m * k)], [val(bb) for _ in range(k * n)]
                a.upload(*g.ints_to_planes(A, a.nlimbs))
                b.upload(*g.ints_to_planes(B, b.nlimbs))
                c.limbs_t.fill_(0x5a5a5a5a)
                exp.append([sum(A[y * k + i] * B[i * n + x] for i in range(k)) for y in range(m) for x in range(n)])
            h.matmul_batched(jobs, path=g.PATH_CRT)
            for (a, b, c), e in zip(mats, exp):
                assert c.to_ints() == e
        h.close()
