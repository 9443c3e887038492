"""gbmm_matmul_host with CRT plans whose product is not the one that was asked for: a
limb-half split (its halves are one product, C the shifted sum of its parts) and
Winograd's tree with CRT leaves (whose sums read B first).  Neither may start on A alone
nor return C in ranges of a stage within.  Bit-exact against Python integers."""
import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _spec(g, rng, K, M, N, ba, bb):
    import torch
    pin = lambda a: torch.from_numpy(a).pin_memory().numpy()
    A = [rng.getrandbits(ba) * rng.choice((-1, 1)) for _ in range(K * M)]
    B = [rng.getrandbits(bb) * rng.choice((-1, 1)) for _ in range(M * N)]
    la, lb = (ba + 31) // 32, (bb + 31) // 32
    planes = [tuple(pin(x) for x in g.ints_to_planes(v, nl)) for v, nl in ((A, la), (B, lb))]
    C = (pin(np.zeros((la + lb + 4, K * N), dtype=np.uint32)), pin(np.zeros(K * N, dtype=np.int32)))
    exp = [sum(A[y * M + k] * B[k * N + x] for k in range(M)) for y in range(K) for x in range(N)]
    return (K, M, N, planes[0], planes[1], C), exp


def _run(g, h, spec, exp, **kw):
    Cl, Cs = spec[5]
    for jobs in (1, 2, 1, 2):
        Cl[:], Cs[:] = 0x5a5a5a5a, 3
        chosen = h.matmul_host(h.host_jobs([spec] * jobs, **kw))
        assert set(chosen) == {g.PATH_CRT}
        assert g.planes_to_ints(Cl, Cs) == exp


@pytest.mark.parametrize("K,M,N,ba,bb", [(150, 64, 120, 4096, 2048), (150, 64, 120, 2048, 4096), (40, 30, 50, 1024, 1024)])
def test_split_plan(g, tmp_path, K, M, N, ba, bb):
    lg = lambda d: round(math.log2(d))
    key = 0
    for d in (K, M, N, ba // 32, bb // 32):
        key = key << 8 | lg(d)
    table = tmp_path / "tune.json"
    table.write_text('[\n  {"key": %d, "plan": %d, "ms": 0.01}\n]\n' % (key, g.PLAN_CRT_SPLIT))
    spec, exp = _spec(g, random.Random(K + ba), K, M, N, ba, bb)
    h = g.Handle()
    assert g.lib().gbmm_tune_load(h.h, str(table).encode()) == g.OK
    _run(g, h, spec, exp)
    h.close()


@pytest.mark.parametrize("n,bits,cutoff", [(64, 1024, 32), (96, 700, 24)])
def test_tree_with_crt_leaves(g, n, bits, cutoff):
    spec, exp = _spec(g, random.Random(n + bits), n, n, n, bits, bits)
    h = g.Handle()
    _run(g, h, spec, exp, path=g.PATH_CRT, method=g.METHOD_WINOGRAD_CRT, cutoff=cutoff)
    h.close()
