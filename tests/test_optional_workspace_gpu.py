"""The workspace with which limb products run on the tensor cores is optional: a call
that the plain workspace serves is not refused, does not end a stream capture, does not
grow the workspace past what later calls need, gives nothing up for a refused part and
stays inside a device budget."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g(built_lib):
    import gbmm
    gbmm.default_handle()
    return gbmm


def _case(g, n, limbs, seed):
    rng = random.Random(seed)
    A, B = ([rng.getrandbits(32 * limbs) * rng.choice((-1, 1)) for _ in range(n * n)] for _ in range(2))
    dA, dB = g.DeviceMatrix.from_ints(n, n, A, limbs), g.DeviceMatrix.from_ints(n, n, B, limbs)
    return A, B, dA, dB, g.DeviceMatrix(n, n, 2 * limbs + 1)


def _check(A, B, n, dC, samples=40):
    got, rng = dC.to_ints(), random.Random(n)
    for _ in range(samples):
        y, x = rng.randrange(n), rng.randrange(n)
        assert got[y * n + x] == sum(A[y * n + k] * B[k * n + x] for k in range(n))


def test_capture_after_a_call_with_a_smaller_workspace(g):
    """A limb product needs the plain workspace only, which the warm-up call left: it can be
    captured, and the graph's replay computes it."""
    import torch
    n, limbs = 64, 33
    A, B, dA, dB, dC = _case(g, n, limbs, 1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        h = g.Handle()
        small = _case(g, 4, 2, 2)
        h.matmul(small[4], small[2], small[3], path=g.PATH_LIMB, method=g.METHOD_NAIVE)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            h.matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE)
        graph.replay()
        torch.cuda.synchronize()
        _check(A, B, n, dC)
        h.close()


def test_workspace_does_not_double_on_the_optional_part(g):
    """A CRT product that needs a little more than the optional workspace of an earlier limb
    product gets what it needs, not twice that workspace."""
    import torch
    limb, crt = _case(g, 256, 64, 3), _case(g, 192, 64, 4)
    h = g.Handle()
    h.matmul(*[_case(g, 16, 64, 5)[i] for i in (4, 2, 3)], path=g.PATH_CRT)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    h.matmul(limb[4], limb[2], limb[3], path=g.PATH_LIMB, method=g.METHOD_NAIVE)
    _check(limb[0], limb[1], 256, limb[4], 8)
    free1 = torch.cuda.mem_get_info()[0]
    assert free0 - free1 > 80 << 20  # the optional workspace of the product (digits and columns)
    h.matmul(crt[4], crt[2], crt[3], path=g.PATH_CRT)
    _check(crt[0], crt[1], 192, crt[4], 8)
    free2 = torch.cuda.mem_get_info()[0]
    # 258 moduli: planes of A, B and the product 38 MB each and the digits 19 MB; the tables 5 MB
    assert free0 - free2 < 160 << 20
    h.close()


def test_graphs_survive_a_refused_request(g):
    """Where the device has no room for the optional part, nothing is given up for it: the
    workspace and the batches captured in it stay, and the product runs without."""
    import ctypes
    import torch
    f = g.lib().gbmmx_extra_room
    f.argtypes, f.restype = [ctypes.c_int64], ctypes.c_int64
    n = 64
    A, B, dA, dB, dC = _case(g, n, 33, 6)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        h = g.Handle()
        small = _case(g, 8, 2, 7)
        jobs = h.jobs([(small[4], small[2], small[3])], path=g.PATH_LIMB)

        def replayed():  # the library times launches, not the kernels of a replay
            g.profile(1)
            h.matmul_batched(jobs, path=g.PATH_LIMB)
            torch.cuda.synchronize()
            ran = g.profile_read()
            g.profile(0)
            return ran == {}

        h.matmul_batched(jobs, path=g.PATH_LIMB)
        h.matmul_batched(jobs, path=g.PATH_LIMB)
        assert replayed()
        old = f(0)
        try:
            h.matmul(dC, dA, dB, path=g.PATH_LIMB, method=g.METHOD_NAIVE)
        finally:
            f(old)
        assert replayed()
        _check(A, B, n, dC)
        h.close()


def test_device_budget_covers_blocked_limb_products(g):
    """A product that runs out of core under a device budget takes no optional workspace
    beside its blocks (its footprint counts the plain workspace)."""
    import numpy as np
    import torch
    n, limbs = 96, 32
    rng = random.Random(8)
    A, B = ([rng.getrandbits(32 * limbs) * rng.choice((-1, 1)) for _ in range(n * n)] for _ in range(2))
    (Al, As), (Bl, Bs) = g.ints_to_planes(A, limbs), g.ints_to_planes(B, limbs)
    Cl, Cs = np.zeros((2 * limbs + 1, n * n), dtype=np.uint32), np.zeros(n * n, dtype=np.int32)
    h = g.Handle()
    spec = [(n, n, n, (Al, As), (Bl, Bs), (Cl, Cs))]
    for budget in (0, 12 << 20):
        h.set_device_budget(budget)
        g.profile(1)
        h.matmul_host(h.host_jobs(spec, path=g.PATH_LIMB, method=g.METHOD_NAIVE))
        ran = g.profile_read()
        g.profile(0)
        assert ("k_ltc_gemm" in ran) == (budget == 0)
        got = g.planes_to_ints(Cl, Cs)
        for _ in range(40):
            y, x = rng.randrange(n), rng.randrange(n)
            assert got[y * n + x] == sum(A[y * n + k] * B[k * n + x] for k in range(n))
        Cl[:], Cs[:] = 0, 0
    h.close()
