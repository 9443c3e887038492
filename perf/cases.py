"""Performance cases: what programs that use gbmm have it do, each through the
public Python entry points (bachelor-thesis_gb300/gbmm.py), from the smallest calls
to the largest.  Inputs are signed integers drawn on the GPU from a seed: uniform
magnitudes, fair signs, optional exact zeros and short entries.

Kinds of case:
  matmul    Handle.matmul with the dispatcher's own choice of path (C = A*B, C += A*B)
  limb      mat_mul / mat_mul_winograd: the plain limb form that the reference-shaped
            operators run by default
  batched   Handle.matmul_batched: many uneven products in one call, on a stream
  host      Handle.matmul_host: products whose operands and results are in host memory
  mpn_add   mpn_add_n over a batch of operands
  mpn_mul   mpn_mul over a batch of operand pairs
  mpz_addmul  w += u*v, elementwise over a matrix
"""
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bachelor-thesis_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import gbmm  # noqa: E402


def listed():
    return [
        # the smallest product of the benchmark list: launches and host work count
        dict(name="matmul_64_1024b", kind="matmul", K=64, M=64, N=64, bits_a=1024, bits_b=1024,
             zero=0.0, short=0.0, accumulate=False),
        # a medium product with some zero and some 64-bit entries
        dict(name="matmul_256_2048b", kind="matmul", K=256, M=256, N=256, bits_a=2048, bits_b=2048,
             zero=0.05, short=0.05, accumulate=False),
        # the headline product
        dict(name="matmul_512_4096b", kind="matmul", K=512, M=512, N=512, bits_a=4096, bits_b=4096,
             zero=0.0, short=0.0, accumulate=False),
        # a thin panel update C += A*B, the step of a blocked product
        dict(name="addmul_1024x64x1024_2048b", kind="matmul", K=1024, M=64, N=1024, bits_a=2048, bits_b=2048,
             zero=0.0, short=0.0, accumulate=True),
        # odd dimensions, one operand much longer than the other, longer than one digit group
        dict(name="matmul_181x75x133_long", kind="matmul", K=181, M=75, N=133, bits_a=13001, bits_b=6007,
             zero=0.1, short=0.0, accumulate=False),
        # the plain limb form of the medium product (mat_mul's default path)
        dict(name="limb_256_2048b", kind="limb", method="naive", K=256, M=256, N=256, bits_a=2048, bits_b=2048,
             zero=0.05, short=0.05, cutoff=0),
        # Winograd's recursion on the limb form, as a reference program calls it
        dict(name="winograd_128_1024b", kind="limb", method="winograd", K=128, M=128, N=128, bits_a=1024,
             bits_b=1024, zero=0.0, short=0.0, cutoff=32),
        # 64 independent products of uneven shape and length in one call, replayed
        dict(name="batched_64_uneven", kind="batched", jobs=64, shape_seed=2024, max_dim=512, max_bits=16384,
             zero=0.1),
        # a short stream of products from and to pinned host memory
        dict(name="host_4x_192x256x320_2048b", kind="host", jobs=4, K=192, M=256, N=320, bits_a=2048, bits_b=2048,
             zero=0.0),
        # batched mpn and mpz calls over more data than L2 holds
        dict(name="mpn_add_n_1M_x32", kind="mpn_add", nb=1 << 20, n=32),
        dict(name="mpn_mul_256k_32x32", kind="mpn_mul", nb=1 << 18, un=32, vn=32),
        dict(name="mpz_addmul_1024x1024_512b", kind="mpz_addmul", rows=1024, cols=1024, bits_u=512, bits_v=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "limb", "limb", "batched", "host", "mpn_add", "mpn_mul",
                       "mpz_addmul"])
    zero = rng.choice([0.0, 0.05, 0.1])
    while True:
        if kind == "matmul":
            c = dict(kind=kind, K=_log_int(rng, 16, 1024), M=_log_int(rng, 16, 512), N=_log_int(rng, 16, 1024),
                     bits_a=_log_int(rng, 256, 16384), bits_b=_log_int(rng, 256, 16384), zero=zero,
                     short=rng.choice([0.0, 0.05]), accumulate=rng.random() < 0.25)
            limit = work(listed()[2])
        elif kind == "limb":
            method = rng.choice(["naive", "winograd"])
            K, M, N = (_log_int(rng, 16, 256) for _ in range(3))
            if method == "winograd":
                K = M = N = _log_int(rng, 33, 256)
            c = dict(kind=kind, method=method, K=K, M=M, N=N, bits_a=_log_int(rng, 64, 4096),
                     bits_b=_log_int(rng, 64, 4096), zero=zero, short=0.0,
                     cutoff=0 if method == "naive" else rng.choice([16, 32, 64]))
            limit = work(listed()[5])
        elif kind == "batched":
            c = dict(kind=kind, jobs=rng.randint(8, 64), shape_seed=rng.randrange(1 << 20),
                     max_dim=_log_int(rng, 64, 512), max_bits=_log_int(rng, 1024, 16384), zero=zero)
            limit = work(listed()[7])
        elif kind == "host":
            c = dict(kind=kind, jobs=rng.randint(1, 6), K=_log_int(rng, 32, 512), M=_log_int(rng, 32, 512),
                     N=_log_int(rng, 32, 512), bits_a=_log_int(rng, 512, 8192), bits_b=_log_int(rng, 512, 8192),
                     zero=zero)
            limit = work(listed()[8])
        elif kind == "mpn_add":
            c = dict(kind=kind, nb=_log_int(rng, 1 << 10, 1 << 20), n=_log_int(rng, 1, 128))
            limit = work(listed()[9])
        elif kind == "mpn_mul":
            un = _log_int(rng, 2, 128)
            c = dict(kind=kind, nb=_log_int(rng, 1 << 10, 1 << 18), un=un, vn=max(1, int(un * rng.uniform(0.3, 1.0))))
            limit = work(listed()[10])
        else:
            c = dict(kind=kind, rows=_log_int(rng, 16, 1024), cols=_log_int(rng, 16, 1024),
                     bits_u=_log_int(rng, 64, 2048), bits_v=_log_int(rng, 64, 2048))
            limit = work(listed()[11])
        w = work(c)
        if w["bytes"] <= limit["bytes"] and w["flops"] <= limit["flops"]:
            return c


def _limbs(bits):
    return (bits + 31) // 32


def _job_shapes(case):
    rng = random.Random(case["shape_seed"])
    return [tuple(_log_int(rng, 16, case["max_dim"]) for _ in range(3)) +
            tuple(_log_int(rng, 64, case["max_bits"]) for _ in range(2)) for _ in range(case["jobs"])]


def _product_work(K, M, N, ba, bb, limb_form):
    """Bytes of the operands and the result; operations: the schoolbook 32-bit limb
    multiply-adds, or the byte-digit multiply-adds of a product by 16-bit moduli
    (residues, products, reconstruction), whichever is less."""
    la, lb = _limbs(ba), _limbs(bb)
    nbytes = 4 * ((la + 1) * K * M + (lb + 1) * M * N + (la + lb + 2) * K * N)
    flops = 2 * K * M * N * la * lb
    if not limb_form:
        P = (ba + bb + M.bit_length() + 18 + 15) // 16
        flops = min(flops, 2 * (2 * P * (K * M * (ba // 8 + 1) + M * N * (bb // 8 + 1)) + 4 * P * K * M * N +
                                2 * P * K * N * (2 * P)))
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind in ("matmul", "limb"):
        b, f = _product_work(case["K"], case["M"], case["N"], case["bits_a"], case["bits_b"], kind == "limb")
        if case.get("accumulate"):
            b += 4 * (_limbs(case["bits_a"]) + _limbs(case["bits_b"]) + 2) * case["K"] * case["N"]
    elif kind == "batched":
        b = f = 0
        for shape in _job_shapes(case):
            jb, jf = _product_work(*shape, False)
            b, f = b + jb, f + jf
    elif kind == "host":
        b, f = _product_work(case["K"], case["M"], case["N"], case["bits_a"], case["bits_b"], False)
        b, f = b * case["jobs"], f * case["jobs"]
    elif kind == "mpn_add":
        b, f = 4 * case["nb"] * (3 * case["n"] + 1), case["nb"] * case["n"]
    elif kind == "mpn_mul":
        b = 8 * case["nb"] * (case["un"] + case["vn"])
        f = 2 * case["nb"] * case["un"] * case["vn"]
    else:
        lu, lv = _limbs(case["bits_u"]), _limbs(case["bits_v"])
        e = case["rows"] * case["cols"]
        b, f = 4 * e * (lu + lv + 2 * (lu + lv + 1) + 4), 2 * e * lu * lv
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """Every output is a whole number: equal or wrong, nothing to measure against."""
    return None


# ---- inputs ---------------------------------------------------------------------
def _planes(rows, cols, bits, zero, short, gen):
    """(limbs [L, rows*cols], sizes [rows*cols]) int32 on the GPU: uniform magnitudes
    of up to `bits` bits, fair signs, a share of zeros and of 64-bit entries."""
    n, L = rows * cols, _limbs(bits)
    limbs = torch.empty((L, n), dtype=torch.int32, device="cuda")
    limbs.random_(-2 ** 31, 2 ** 31, generator=gen)
    top = bits - 32 * (L - 1)
    if top < 32:
        limbs[L - 1] &= (1 << top) - 1
    u = torch.rand(n, device="cuda", generator=gen)
    if zero:
        limbs.mul_((u >= zero).to(torch.int32))
    if short and L > 2:
        limbs[2:].mul_(((u < zero) | (u >= zero + short)).to(torch.int32))
    size = torch.zeros(n, dtype=torch.int32, device="cuda")
    for i in range(L):
        size = torch.where(limbs[i] != 0, i + 1, size)
    sign = torch.rand(n, device="cuda", generator=gen) < 0.5
    return limbs, torch.where(sign, -size, size).to(torch.int32)


def _matrix(rows, cols, bits, zero, short, gen):
    limbs, sizes = _planes(rows, cols, bits, zero, short, gen)
    m = gbmm.DeviceMatrix(rows, cols, limbs.shape[0])
    m.limbs_t.copy_(limbs.view(-1))
    m.sizes_t.copy_(sizes)
    return m


_stream = None


def _side_stream():
    """The stream that a program keeps for its batched calls (a created stream, so
    that the library may record and replay them)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("matmul", "limb"):
        K, M, N = case["K"], case["M"], case["N"]
        s["A"] = _matrix(K, M, case["bits_a"], case["zero"], case["short"], gen)
        s["B"] = _matrix(M, N, case["bits_b"], case["zero"], case["short"], gen)
        path = gbmm.PATH_LIMB if kind == "limb" else gbmm.PATH_AUTO
        method = gbmm.METHOD_NAIVE if case.get("method") == "naive" else gbmm.METHOD_WINOGRAD
        cn = gbmm.limbs_needed(s["A"].nlimbs, s["B"].nlimbs, M, path=path, method=method,
                               cutoff=case.get("cutoff", 0))
        acc = bool(case.get("accumulate"))
        # an accumulated C starts as some earlier panel's sum, with room to grow
        s["C"] = gbmm.DeviceMatrix(K, N, cn + (1 if acc else 0))
        if acc:
            limbs, sizes = _planes(K, N, case["bits_a"] + case["bits_b"], 0.0, 0.0, gen)
            s["C"].limbs_t[:limbs.numel()].copy_(limbs.view(-1))
            s["C"].sizes_t.copy_(sizes)
        s["h"] = gbmm.default_handle()
    elif kind == "batched":
        shapes = _job_shapes(case)
        mats, entries, limbs = [], 0, 0
        for K, M, N, ba, bb in shapes:
            A, B = _matrix(K, M, ba, case["zero"], 0.0, gen), _matrix(M, N, bb, case["zero"], 0.0, gen)
            cn = A.nlimbs + B.nlimbs + 2
            mats.append((A, B, cn, entries, limbs))
            entries += (K * N + 63) // 64 * 64
            limbs += (cn * K * N + 63) // 64 * 64
        # all results in one allocation, as a program with many small ones lays them out
        s["limbs"] = torch.zeros(limbs, dtype=torch.int32, device="cuda")
        s["sizes"] = torch.zeros(entries, dtype=torch.int32, device="cuda")
        triples = []
        for (K, M, N, ba, bb), (A, B, cn, e0, l0) in zip(shapes, mats):
            c = gbmm.Mat()
            c.rows, c.cols, c.nlimbs, c.rs, c.ld = K, N, cn, N, K * N
            c.limbs = s["limbs"].data_ptr() + 4 * l0
            c.sizes = s["sizes"].data_ptr() + 4 * e0
            triples.append((c, A, B))
        s["mats"] = mats
        s["jobs"] = gbmm.Handle.jobs(triples)
        s["h"] = gbmm.default_handle()
        s["stream"] = _side_stream()
        torch.cuda.synchronize()
    elif kind == "host":
        K, M, N = case["K"], case["M"], case["N"]
        cn = _limbs(case["bits_a"]) + _limbs(case["bits_b"]) + 2
        s["C"], specs = [], []
        for _ in range(case["jobs"]):
            host = []
            for r, c, bits in ((K, M, case["bits_a"]), (M, N, case["bits_b"])):
                limbs, sizes = _planes(r, c, bits, case["zero"], 0.0, gen)
                host.append(tuple(torch.empty(t.shape, dtype=torch.int32, pin_memory=True).copy_(t)
                                  for t in (limbs, sizes)))
            host.append((torch.zeros((cn, K * N), dtype=torch.int32, pin_memory=True),
                         torch.zeros(K * N, dtype=torch.int32, pin_memory=True)))
            s["C"].append(host[2])
            specs.append((K, M, N) + tuple((x.numpy(), y.numpy()) for x, y in host))
        s["specs"] = specs
        s["jobs"] = gbmm.Handle.host_jobs(specs)
        s["h"] = gbmm.default_handle()
    elif kind in ("mpn_add", "mpn_mul"):
        nb = case["nb"]
        un, vn = (case["n"], case["n"]) if kind == "mpn_add" else (case["un"], case["vn"])
        for key, n in (("u", un), ("v", vn)):
            s[key] = torch.empty((n, nb), dtype=torch.int32, device="cuda").random_(-2 ** 31, 2 ** 31, generator=gen)
        s["r"] = torch.zeros((un if kind == "mpn_add" else un + vn, nb), dtype=torch.int32, device="cuda")
        s["cy"] = torch.zeros(nb, dtype=torch.int32, device="cuda")
    else:
        R, C = case["rows"], case["cols"]
        s["u"] = _matrix(R, C, case["bits_u"], 0.0, 0.0, gen)
        s["v"] = _matrix(R, C, case["bits_v"], 0.0, 0.0, gen)
        limbs, sizes = _planes(R, C, case["bits_u"] + case["bits_v"], 0.0, 0.0, gen)
        s["w"] = gbmm.DeviceMatrix(R, C, s["u"].nlimbs + s["v"].nlimbs + 1)
        s["w"].limbs_t[:limbs.numel()].copy_(limbs.view(-1))
        s["w"].sizes_t.copy_(sizes)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "matmul":
        s["h"].matmul(s["C"], s["A"], s["B"], accumulate=case["accumulate"])
        return s["C"].limbs_t, s["C"].sizes_t
    if kind == "limb":
        if case["method"] == "naive":
            gbmm.mat_mul(case["K"], case["M"], case["N"], s["C"], s["A"], s["B"])
        else:
            gbmm.mat_mul_winograd(case["K"], s["C"], s["A"], s["B"], cutoff=case["cutoff"])
        return s["C"].limbs_t, s["C"].sizes_t
    if kind == "batched":
        with torch.cuda.stream(s["stream"]):
            s["h"].matmul_batched(s["jobs"])
        return s["limbs"], s["sizes"]
    if kind == "host":
        s["h"].matmul_host(s["jobs"])
        return s["C"]
    if kind == "mpn_add":
        gbmm.mpn_add_n(s["r"], s["u"], s["v"], case["n"], case["nb"], case["nb"], s["cy"])
        return s["r"], s["cy"]
    if kind == "mpn_mul":
        gbmm.mpn_mul(s["r"], s["u"], case["un"], s["v"], case["vn"], case["nb"], case["nb"])
        return s["r"]
    gbmm.mpz_addmul(s["w"], s["u"], s["v"])
    return s["w"].limbs_t, s["w"].sizes_t
