"""Digits and residues in one kernel (csrc/crt.cu, k_crt_residue2) in a batch's grouped
launch: operands of one to eight 64-digit slots as units of one launch, beside rows past 512
digits in the two-kernel form and a limb-half split read in place.  Eager call, capturing
call and replay, with new inputs for each.  Integer work: exact."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


SPECS = [(9, 33, 7, 1500, 60), (40, 31, 17, 4096, 4095), (8, 32, 8, 513, 1024), (1, 1, 1, 40, 2000), (65, 64, 30, 300, 3000),
         (24, 20, 33, 4097, 700), (33, 21, 9, 9000, 4096), (24, 16, 40, 20000, 4000), (40, 16, 24, 4000, 20000)]


def test_grouped_products_of_mixed_row_lengths(g):
    import torch
    rng = random.Random(77)
    val = lambda bits: rng.choice((rng.getrandbits(bits), (1 << bits) - 1, rng.getrandbits(rng.randint(1, bits)), 0, 1)) * rng.choice((-1, 1))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        h = g.Handle()
        mats = []
        for m, k, n, ba, bb in SPECS:
            la, lb = (ba + 31) // 32, (bb + 31) // 32
            mats.append((g.DeviceMatrix(m, k, la), g.DeviceMatrix(k, n, lb), g.DeviceMatrix(m, n, la + lb + 1)))
        jobs = h.jobs([(c, a, b) for a, b, c in mats], path=g.PATH_CRT)
        for call in range(3):
            exp = []
            for (m, k, n, ba, bb), (a, b, c) in zip(SPECS, mats):
                A, B = [val(ba) for _ in range(m * k)], [val(bb) for _ in range(k * n)]
                a.upload(*g.ints_to_planes(A, a.nlimbs))
                b.upload(*g.ints_to_planes(B, b.nlimbs))
                exp.append([sum(A[y * k + i] * B[i * n + x] for i in range(k)) for y in range(m) for x in range(n)])
            g.profile(1 if call == 0 else 0)
            h.matmul_batched(jobs, path=g.PATH_CRT)
            if call == 0:
                ran = g.profile_read()
                g.profile(0)
                # one grouped launch of each form
                assert ran["k_crt_residue2"][0] == 1 and ran["k_crt_residue"][0] >= 1
            for (a, b, c), e in zip(mats, exp):
                assert c.to_ints() == e
        h.close()
