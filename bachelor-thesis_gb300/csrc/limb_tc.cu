// The limb form's matrix product on the tcgen05 tensor cores: schoolbook column
// sums over byte digits.
//
// Entry (y, x) of C = A B has the digit columns
//     D_t = sum_k sum_{i + j = t} a_i(y, k) b_j(k, x)            (digits base 256),
// which for one y is a GEMM over (k, j): the plain operand is the digit rows of
// B's column x (128 of them are the M rows of a tile, so TMEM lane = x), and the
// other operand is a Hankel matrix built from A's digits, H[t'][j] = a_(T-1-t'-j)
// with t' = T - 1 - t.  Its 8 x 8 core matrix at (t', j) depends on t' + j only, so
// the (W + 16 nb) / 8 core matrices on its diagonals serve a whole W x 16 nb tile:
// the descriptor's two strides are equal, and a digit row expands 8-fold in shared
// memory instead of W-fold.
//
// Exactness: digits are balanced, |d| <= 128 (a row's last digit at most 256), so a
// column gains at most 2^14 per (k, j), plus 2^15 per k for the last digits; the FP32
// accumulators are added into 32-bit integers every LT_FLUSH chunks (at most
// 960 + 32 terms of 2^14 < 2^24), and the caller keeps k (min digits + 2) below 2^17.
//
// After the last K step a tile turns its columns into limbs from carry 0 (two's
// complement, carry out kept per segment); k_ltc_finish resolves the carries between
// segments, adds the old C for C += A B, and writes sign and magnitude.  A longer inner
// dimension runs in chunks: a later chunk's tiles add the earlier ones' limbs and carries
// to theirs, and C, whose planes only the exact result has to fit, is read and written
// once at the end.
//
// Replaces the launcher_mul / launcher_addmul kernels (mat-gpu/mat-core.h:7-137)
// wherever ltc_pays() says so; the CUDA-core kernel (limb.cu) takes the rest.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "digits.cuh"
#include "gbmm_internal.h"
#include "limb_dev.cuh"
#include "tc.cuh"

namespace gbmm {

namespace {
constexpr int LT_STAGES = 6;             // ring of plain digit rows, 64 digits a stage
constexpr int LT_HANKEL = 6;             // ring of Hankel operands, one term k each
constexpr int LT_RAW = 3;                // digit rows a builder warp has in flight
constexpr int LT_FLUSH = 15;             // 64-digit chunks per exact FP32 accumulation
constexpr int LT_CORE = 144;             // bytes between core matrices: 128 + 16, conflict-free 16-byte stores
constexpr uint32_t LT_STAGE = 128 * 128;    // 128 digit rows of 64 digits
constexpr int LT_THREADS = 384;          // warps 0 TMA, 1 MMA, 2..3 Hankel builders, 4..11 epilogue
}  // namespace

// Shape of one launch: `leaves` independent products of m x k by k x n entries.
struct LtcArgs {
    const __nv_bfloat16 *ad;  // A's digit rows [leaf][m][k][dxa]
    int32_t m, n, k;
    int32_t dxa, dxb;  // digits per entry (multiples of 16)
    int32_t T;         // digit columns per entry (T >= dxa + dxb), columns in descending order t' = T - 1 - t
    int32_t W, nW;     // columns per tile and tiles per entry; nY > 1: W = nY T, one tile holds nY rows y
    int32_t nY;
    int32_t seg;       // columns per segment (one thread's columns of one entry)
    int32_t prow, cs;  // digit rows a tile loads, and 64-digit chunks of one k that share a stage
    int32_t nyg;       // groups of nY rows
    int32_t nxt;       // tiles of 128 columns x
    int64_t nitems;
    uint32_t *wl;      // [T / 4][entries] limbs, two's complement per segment
    void *wq;          // [T / seg][entries] carry out of each segment: int32_t, int64_t with `chunks`
    int32_t chunks;    // one of several chunks of the inner dimension
    int32_t later;     // ... and not the first
    int64_t went;      // entries = leaves m n
    int32_t esize, rsize;  // bytes of a Hankel ring entry and of a builder's digit row buffer
};

struct LtcBars {
    uint64_t full[LT_STAGES], empty[LT_STAGES], hfull[LT_HANKEL], hempty[LT_HANKEL], raw[2][LT_RAW], tfull[2], tempty[2];
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ void ltc_abort(LtcBars *b, uint32_t *err) {
    atomicOr(err, DEVERR_TIMEOUT);
    *(volatile int *)&b->abort_flag = 1;
}
__device__ __forceinline__ bool ltc_aborted(LtcBars *b) { return *(volatile int *)&b->abort_flag != 0; }

// One tile: column tile xt of leaf `leaf`, rows yg * nY .., columns t' = t0 .. t0 + W - 1;
// K steps are (k, c) with digit chunk c (64 digits) in [c0, c1].
struct LtcItem {
    int leaf, xt, yg, t0, c0, c1;
};
// (yg, window) fastest: tiles that run together share the plain operand's rows in L2
__device__ __forceinline__ LtcItem ltc_item(const LtcArgs &a, int64_t it) {
    LtcItem r;
    const int64_t per = (int64_t)a.nyg * a.nW;
    const int64_t g = it / per;
    const int q = (int)(it - g * per);
    r.leaf = (int)(g / a.nxt);
    r.xt = (int)(g - (int64_t)r.leaf * a.nxt);
    r.yg = q / a.nW;
    r.t0 = (q - r.yg * a.nW) * a.W;
    // digits j with a nonzero column in the window: T - dxa - t0 - W + 1 <= j <= T - 1 - t0
    // (a tile of several rows covers every column)
    int jlo = 0, jhi = a.dxb - 1;
    if (a.nY == 1) {
        jlo = max(0, a.T - a.dxa - r.t0 - a.W + 1);
        jhi = min(a.dxb - 1, a.T - 1 - r.t0);
        if (jhi < jlo) jlo = jhi = 0;  // padding columns only: one chunk of zeros
    }
    r.c0 = jlo >> 6;
    r.c1 = jhi >> 6;
    return r;
}

// Core matrices of a tile's Hankel operand for one k: rows t' + j - 64 c0 over the
// tile's columns and the digits of its chunks.
__device__ __forceinline__ int ltc_cores(const LtcArgs &a, const LtcItem &I) {
    return (a.W + min(a.dxb, 64 * (I.c1 + 1)) - 64 * I.c0) >> 3;
}

// Descriptor of the Hankel operand: no swizzle, both strides one core matrix.
__device__ __forceinline__ uint64_t sdesc_hankel(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(LT_CORE >> 4) << 16) | ((uint64_t)(LT_CORE >> 4) << 32) |
           ((uint64_t)1 << 46);
}

// What bounds it: the tensor pipe (83 % busy at 256^3, 2048 bits; an MMA of 256 columns, M = 128,
// K = 16 takes 128 clocks) beside the 16 KB of plain rows each K step brings into shared memory.  Every
// MMA covers the tile's W columns: restricting an MMA to the columns that its digits
// reach halves the multiplications, but every change of the column range drains the
// pipe (measured at 256^3, 2048 bits: 4.5 ms with exact ranges, 3.7 ms with one range
// per K step, 2.8 ms without, before the operands had rings of their own).
// CHUNKS: a.chunks, kept out of the common launches' epilogue.
template <bool CHUNKS>
__global__ void __launch_bounds__(LT_THREADS, 1)
    k_ltc_gemm(const __grid_constant__ CUtensorMap tmP, LtcArgs a, uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *hbase = base + LT_STAGES * LT_STAGE, *rbase = hbase + LT_HANKEL * a.esize;
    LtcBars *bars = reinterpret_cast<LtcBars *>(rbase + 2 * LT_RAW * a.rsize);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < LT_STAGES; s++) {
            tc::mbar_init(&bars->full[s], 1);
            tc::mbar_init(&bars->empty[s], 1);
        }
        for (int s = 0; s < LT_HANKEL; s++) {
            tc::mbar_init(&bars->hfull[s], 1);
            tc::mbar_init(&bars->hempty[s], 1);
        }
        for (int s = 0; s < LT_RAW; s++) {
            tc::mbar_init(&bars->raw[0][s], 1);
            tc::mbar_init(&bars->raw[1][s], 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(&bars->tfull[b], 1);
            tc::mbar_init(&bars->tempty[b], 8);
        }
        bars->abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(&bars->tmem_base, 512);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    tc::grid_dep_wait();
    const uint32_t tmem = bars->tmem_base;

    if (warp < 4) {
        if (warp == 0) {
            if (tc::elect_one()) {
                tc::prefetch_tmap(&tmP);
                const uint32_t bytes = (uint32_t)a.prow * 128;
                int st = 0;
                uint32_t ph = 1;  // parity of the phase before the barrier's first: the first round passes at once
                bool ok = true;
                for (int64_t q = blockIdx.x; q < a.nitems && ok && !ltc_aborted(bars); q += gridDim.x) {
                    const LtcItem I = ltc_item(a, q);
                    int row = I.leaf * a.k * a.n + I.xt * 128;  // digit rows are [leaf][k][x]
                    for (int kk = 0; kk < a.k && ok; kk++, row += a.n)
                        for (int c = I.c0; c <= I.c1; c += a.cs) {
                            if (!tc::mbar_wait(&bars->empty[st], ph)) {
                                ltc_abort(bars, err);
                                ok = false;
                                break;
                            }
                            const int nc = min(a.cs, I.c1 - c + 1);
                            uint8_t *sp = base + st * LT_STAGE;
                            tc::mbar_arrive_expect_tx(&bars->full[st], bytes * nc);
                            for (int i = 0; i < nc; i++, sp += bytes)
                                tc::tma_load_2d(sp, &tmP, &bars->full[st], 64 * (c + i), row);
                            if (++st == LT_STAGES) {
                                st = 0;
                                ph ^= 1;
                            }
                        }
                }
            }
        } else if (warp == 1) {
            if (tc::elect_one()) {
                const uint32_t idesc = tc::idesc_bf16_f32(128, (uint32_t)a.W, 0, 0);
                const uint64_t hd0 = sdesc_hankel(tc::smem_u32(hbase)), pd0 = tc::sdesc_kmajor(tc::smem_u32(base));
                const int flush_steps = LT_FLUSH / a.cs;
                int st = 0, eh = 0, fl = 0;
                uint32_t ph = 0, hph = 0;
                bool ok = true;
                for (int64_t q = blockIdx.x; q < a.nitems && ok; q += gridDim.x) {
                    const LtcItem I = ltc_item(a, q);
                    int left = 0;  // K steps left in the current accumulation
                    for (int kk = 0; kk < a.k && ok; kk++) {
                        if (!tc::mbar_wait(&bars->hfull[eh], hph)) {
                            ltc_abort(bars, err);
                            ok = false;
                            break;
                        }
                        uint64_t hd = tc::sdesc_advance(hd0, (uint32_t)(eh * a.esize));
                        int blocks = (min(a.dxb, 64 * (I.c1 + 1)) - 64 * I.c0) >> 4;  // 16-digit blocks of this k
                        for (int c = I.c0; c <= I.c1; c += a.cs) {
                            const int b = fl & 1;
                            bool fresh = left == 0;
                            if (fresh) {
                                left = flush_steps;
                                if (fl >= 2 && !tc::mbar_wait(&bars->tempty[b], ((fl >> 1) & 1) ^ 1)) {
                                    ltc_abort(bars, err);
                                    ok = false;
                                    break;
                                }
                            }
                            if (!tc::mbar_wait(&bars->full[st], ph)) {
                                ltc_abort(bars, err);
                                ok = false;
                                break;
                            }
                            tc::fence_after_sync();
                            uint64_t pd = tc::sdesc_advance(pd0, st * LT_STAGE);
                            const uint32_t d = tmem + 256u * b;
                            left--;
                            const bool last = c + a.cs > I.c1, flush = left == 0 || (last && kk + 1 == a.k);
                            const int nc = min(a.cs, I.c1 - c + 1);
                            for (int i = 0; i < nc; i++) {
#pragma unroll
                                for (int bb = 0; bb < 4; bb++)
                                    if (bb < blocks)
                                        tc::mma_bf16(d, tc::sdesc_advance(pd, bb * 32),
                                                     tc::sdesc_advance(hd, bb * 2 * LT_CORE), idesc,
                                                     fresh && bb == 0 ? 0u : 1u);
                                fresh = false;
                                blocks -= 4;
                                hd = tc::sdesc_advance(hd, 8 * LT_CORE);
                                pd = tc::sdesc_advance(pd, (uint32_t)a.prow * 128);
                            }
                            tc::mma_commit(&bars->empty[st]);
                            if (last) tc::mma_commit(&bars->hempty[eh]);
                            if (flush) {
                                tc::mma_commit(&bars->tfull[b]);
                                left = 0;
                                fl++;
                            }
                            if (++st == LT_STAGES) {
                                st = 0;
                                ph ^= 1;
                            }
                        }
                        if (++eh == LT_HANKEL) {
                            eh = 0;
                            hph ^= 1;
                        }
                    }
                }
            }
        } else {
            // Hankel builders: core matrix s of one k's operand (8 rows of 16 bytes) holds rows
            // v = 8 s + r, row v = digits a_q .. a_(q-7) with q = T - 1 - (t0 + v) - 64 c0, from two
            // aligned octets of the digit row, which a bulk copy has put in one of this
            // warp's buffers (a load from global memory here would stall the proxy fence
            // until it returned).  The two warps take the terms k in turn.
            const int noct = a.dxa >> 3, w = warp & 1;
            uint8_t *rw = rbase + w * LT_RAW * a.rsize;
            int ik0 = 0;       // terms before this tile
            int ri = 0;        // digit rows this warp has requested
            int rc = 0;        // ... and used
            bool ok = true;
            for (int64_t q = blockIdx.x; q < a.nitems && ok; q += gridDim.x) {
                const LtcItem I = ltc_item(a, q);
                const int ncore = ltc_cores(a, I);
                const int o0 = ((a.T - 8 - I.t0) >> 3) - 8 * I.c0;  // exact: multiples of 8
                const int y0 = I.yg * a.nY, ny = min(a.nY, a.m - y0);
                // the octets that exist: [lo, lo + no) of the one row, or all of ny short rows
                const int lo = a.nY > 1 ? 0 : max(0, o0 - ncore);
                const int no = a.nY > 1 ? noct : max(0, min(noct, o0 + 1) - lo);
                const int first = (ik0 ^ w) & 1;
                const __nv_bfloat16 *arow = a.ad + ((int64_t)I.leaf * a.m + y0) * a.k * a.dxa + 8 * lo;
                auto request = [&](int kk) {
                    if (lane == 0) {
                        uint64_t *bar = &bars->raw[w][ri % LT_RAW];
                        tc::mbar_arrive_expect_tx(bar, 16u * no * ny);
                        for (int y = 0; y < ny; y++)
                            if (no)
                                tc::bulk_load(rw + (ri % LT_RAW) * a.rsize + 16 * y * noct,
                                              arow + ((int64_t)y * a.k + kk) * a.dxa, 16u * no, bar);
                    }
                    ri++;
                };
                for (int i = 0, kk = first; i < LT_RAW && kk < a.k; i++, kk += 2) request(kk);
                for (int kk = first; kk < a.k; kk += 2, rc++) {
                    const int ik = ik0 + kk, eh = ik % LT_HANKEL;
                    if (!tc::mbar_wait(&bars->raw[w][rc % LT_RAW], (rc / LT_RAW) & 1) ||
                        (ik >= LT_HANKEL && !tc::mbar_wait(&bars->hempty[eh], ((ik / LT_HANKEL) & 1) ^ 1))) {
                        ltc_abort(bars, err);
                        ok = false;
                        break;
                    }
                    uint8_t *e = hbase + eh * a.esize;
                    const uint4 *r = reinterpret_cast<const uint4 *>(rw + (rc % LT_RAW) * a.rsize);
                    for (int s = lane; s < ncore; s += 32) {
                        int o = o0 - s, ro = -lo;
                        if (a.nY > 1) {
                            const int yy = min(8 * s / a.T, a.nY - 1);
                            o = yy < ny ? o0 + yy * (a.T >> 3) - s : -1;
                            ro = yy * noct;
                        }
                        uint4 hi = make_uint4(0, 0, 0, 0), lw = hi;
                        if (o >= 0 && o < noct) hi = r[ro + o];
                        if (o >= 1 && o - 1 < noct) lw = r[ro + o - 1];
                        const uint32_t X[8] = {hi.w, hi.z, hi.y, hi.x, lw.w, lw.z, lw.y, lw.x};
                        uint8_t *d = e + s * LT_CORE;
#pragma unroll
                        for (int rr = 0; rr < 8; rr++) {
                            uint32_t x[4];
#pragma unroll
                            for (int m = 0; m < 4; m++)
                                x[m] = (rr & 1) ? __byte_perm(X[rr / 2 + m], X[rr / 2 + m + 1], 0x7610)
                                                : __byte_perm(X[rr / 2 + m], 0u, 0x1032);
                            *reinterpret_cast<uint4 *>(d + 16 * rr) = make_uint4(x[0], x[1], x[2], x[3]);
                        }
                    }
                    tc::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&bars->hfull[eh]);
                    if (kk + 2 * LT_RAW < a.k) request(kk + 2 * LT_RAW);
                }
                ik0 += a.k;
            }
        }
    } else {
        // epilogue: quadrant warp % 4 (lane = column x), half hf of the tile's columns
        const int quad = warp & 3, hf = (warp - 4) >> 2;
        const int hc = a.W >> 1;  // this thread's columns, a multiple of 16
        const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(hf * hc);
        int fl = 0;
        bool ok = true;
        for (int64_t q = blockIdx.x; q < a.nitems && ok; q += gridDim.x) {
            const LtcItem I = ltc_item(a, q);
            const int nst = a.k * ((I.c1 - I.c0) / a.cs + 1), per = LT_FLUSH / a.cs, nfl = (nst + per - 1) / per;
            int acc[128];
#pragma unroll
            for (int i = 0; i < 128; i++) acc[i] = 0;
            for (int f = 0; f < nfl; f++, fl++) {
                const int b = fl & 1;
                if (!tc::mbar_wait(&bars->tfull[b], (fl >> 1) & 1)) {
                    ltc_abort(bars, err);
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
#pragma unroll
                for (int ch = 0; ch < 8; ch++) {
                    if (ch * 16 >= hc) continue;
                    uint32_t v[16];
                    tc::tmem_ld16(lb + 256u * b + 16u * ch, v);
                    tc::tmem_ld_wait(v);
#pragma unroll
                    for (int i = 0; i < 16; i++) acc[16 * ch + i] += tc::acc_int(v[i]);
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&bars->tempty[b]);
            }
            if (!ok) break;
            // limbs from the highest t' (lowest digit) up: four columns per limb
            const int x = I.xt * 128 + quad * 32 + lane;
            const bool xok = x < a.n;
            const int col0 = hf * hc;
            long long cy = 0;
            int yy = a.nY > 1 ? (col0 + hc - 4) / a.T : 0;  // row of the group of columns at hand
            int tcol = a.nY > 1 ? a.T - 4 - (col0 + hc - 4 - yy * a.T) : a.T - 4 - (I.t0 + col0 + hc - 4);
            int sleft = a.seg;
            const int y0 = I.yg * a.nY;
            int64_t ent = ((int64_t)I.leaf * a.m + y0 + yy) * a.n + x;
            bool live = xok && y0 + yy < a.m;
            uint32_t *wp = a.wl + (int64_t)(tcol >> 2) * a.went + ent;
#pragma unroll
            for (int g = 31; g >= 0; g--) {
                if (4 * g >= hc) continue;
                // one group at a time: the columns leave no registers for groups formed ahead
                asm volatile("" : "+r"(acc[4 * g]), "+r"(acc[4 * g + 1]), "+r"(acc[4 * g + 2]), "+r"(acc[4 * g + 3]));
                long long v = (long long)acc[4 * g + 3] + (long long)acc[4 * g + 2] * 256 +
                              (long long)acc[4 * g + 1] * 65536 + (long long)acc[4 * g] * 16777216 + cy;
                if (CHUNKS && a.later && live) v += *wp;
                if (live) *wp = (uint32_t)v;
                cy = v >> 32;
                tcol += 4;
                sleft -= 4;
                wp += a.went;
                if (sleft == 0) {
                    // tcol is one past the segment's last column
                    const int64_t qi = (int64_t)(tcol / a.seg - 1) * a.went + ent;
                    if (CHUNKS) {
                        long long *wq = static_cast<long long *>(a.wq) + qi;
                        if (live) *wq = cy + (a.later ? *wq : 0ll);
                    } else if (live) {
                        static_cast<int32_t *>(a.wq)[qi] = (int32_t)cy;
                    }
                    cy = 0;
                    sleft = a.seg;
                    if (a.nY > 1) {
                        yy--;
                        tcol = 0;
                        ent -= a.n;
                        live = xok && y0 + yy < a.m;
                        wp = a.wl + ent;
                    }
                }
            }
        }
    }
    tc::grid_dep_launch();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, 512);
    }
}

// Segments joined: one thread per entry, coalesced over entries.  A first pass
// resolves the carries and finds the sign and size (limbs and old C are read, nothing
// is written, so a result that does not fit C leaves it untouched); the second
// writes the magnitude.  Both passes stream limb planes; the second reads them from
// L2 unless the product is larger.
struct LtcOut {
    gbmm_mat C;      // the product's C (leaves == 1)
    uint32_t *pl;    // Winograd leaves: dense h x h products of pcap planes, leaf after leaf
    int32_t *ps;
    int32_t pcap;
    int32_t accumulate;
};
__global__ void __launch_bounds__(128) k_ltc_finish(LtcArgs a, LtcOut o, uint32_t *err) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.went) return;
    MatArgs C;
    int64_t ic;
    const int64_t mn = (int64_t)a.m * a.n;
    if (o.pl) {
        const int64_t leaf = e / mn;
        C = wt_dense(o.pl, o.ps, leaf, a.m, o.pcap);
        ic = e - leaf * mn;
    } else {
        C = margs(o.C);
        const int64_t y = e / a.n;
        ic = y * C.rs + (e - y * a.n);
    }
    int sc = 0, cn = 0;
    if (o.accumulate) {
        sc = C.sizes[ic];
        cn = min(iabs_d(sc), C.nlimbs);
    }
    const int TL = a.T >> 2, SL = a.seg >> 2;      // limbs in all and per segment (multiples of 4)
    const int LT = (max(TL, cn) + 3) / 4 * 4 + 4;  // limbs processed: room for the last carry
    long long fin = 0;
    int top_nz = 0, top_no = 0, low_nz = LT;  // highest nonzero + 1, highest not all ones + 1, lowest nonzero
    bool neg = false;
    int top = 0;
    for (int pass = 0; pass < 2; pass++) {
        long long c = 0;
        uint32_t n1 = 1;  // the negation's +1
        for (int l0 = 0; l0 < LT; l0 += 4) {
            uint32_t w[4], u[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                w[i] = l0 < TL ? a.wl[(int64_t)(l0 + i) * a.went + e] : 0u;
                u[i] = l0 + i < cn ? C.limbs[(int64_t)(l0 + i) * C.ld + ic] : 0u;
            }
            // the carry out of segment s enters segment s + 1 (also past the last one)
            if (l0 > 0 && l0 <= TL && l0 % SL == 0) {
                const int64_t qi = (int64_t)(l0 / SL - 1) * a.went + e;
                c += a.chunks ? static_cast<const long long *>(a.wq)[qi] : static_cast<const int32_t *>(a.wq)[qi];
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const long long v = (long long)w[i] + c + (sc < 0 ? -(long long)u[i] : (long long)u[i]);
                const uint32_t r = (uint32_t)v;
                c = v >> 32;
                const int l = l0 + i;
                if (pass == 0) {
                    if (r) {
                        top_nz = l + 1;
                        if (low_nz == LT) low_nz = l;
                    }
                    if (r != 0xFFFFFFFFu) top_no = l + 1;
                } else if (l < C.nlimbs) {
                    uint32_t s = r;
                    if (neg) {
                        s = ~r + n1;
                        n1 &= (uint32_t)(r == 0u);
                    }
                    C.limbs[(int64_t)l * C.ld + ic] = s;
                }
            }
        }
        if (pass == 0) {
            fin = c;
            // the exact sum fits LT limbs: what is left is the sign extension
            if (fin != 0 && fin != -1) { atomicOr(err, DEVERR_CAPACITY); return; }
            neg = fin < 0;
            // |v| = ~r + 1: its top limb is the highest one that is not all ones, one more
            // when every limb up to there is zero
            top = !neg ? top_nz : (low_nz >= top_no ? top_no + 1 : top_no);
            if (top > C.nlimbs) { atomicOr(err, DEVERR_CAPACITY); return; }
        }
    }
    for (int l = LT; l < C.nlimbs; l++) C.limbs[(int64_t)l * C.ld + ic] = 0u;
    C.sizes[ic] = neg ? -top : top;
}

// Digit rows of all leaves' operands of a Winograd tree (side 0: A's rows [y][k],
// side 1: B's [k][x]); blockIdx.x = leaf and tile.
__global__ void __launch_bounds__(256)
    k_ltc_wino_digits(WinoTree t, int which, int64_t leaf0, int nbx, int nby, int dx, __nv_bfloat16 *out) {
    const int per = nbx * nby;
    const int64_t leaf = blockIdx.x / per;
    const int b = (int)(blockIdx.x - leaf * per);
    const MatArgs v = wt_operand(t, which, t.levels, leaf0 + leaf);
    DigitArgs a;
    a.limbs = v.limbs;
    a.sizes = v.sizes;
    a.ld = v.ld;
    a.rs = v.rs;
    a.rows = v.rows;
    a.cols = v.cols;
    // quadrants of A and B have one limb less than the sums
    a.nlimbs = v.nlimbs;
    a.transpose = 0;
    a.dxp = dx;
    a.out = out + leaf * v.rows * v.cols * (int64_t)dx;
    digits_block<true>(a, b % nbx, b / nbx, blockIdx.y);
}
// One operand's digit rows; blockIdx.x = tile of 4 rows x 32 columns (rows alone pass a
// grid's 65535 blocks in y from 262141 on).
__global__ void __launch_bounds__(256) k_ltc_digits(DigitArgs a, int nbx) {
    digits_block<true>(a, blockIdx.x % nbx, blockIdx.x / nbx, blockIdx.y);
}

// ---- host side ----------------------------------------------------------------------------
static int ltc_dx(int nl) { return (4 * std::max(nl, 1) + 15) / 16 * 16; }

// Tiles of a product of la x lb limb entries: columns and their split.
static void ltc_shape(LtcArgs &a, int m, int k, int n, int la, int lb, int64_t leaves) {
    memset(&a, 0, sizeof a);
    a.m = m;
    a.k = k;
    a.n = n;
    a.dxa = ltc_dx(la);
    a.dxb = ltc_dx(lb);
    const int T0 = a.dxa + a.dxb;
    if (T0 <= 128) {
        a.T = T0;
        a.nY = 2 * (256 / T0 / 2);
        a.W = a.nY * a.T;
        a.nW = 1;
        a.seg = a.T;
    } else {
        a.nY = 1;
        a.nW = (T0 + 255) / 256;
        a.W = ((T0 + a.nW - 1) / a.nW + 31) / 32 * 32;
        a.T = a.nW * a.W;
        a.seg = a.W / 2;
    }
    // a tile of few columns x packs several chunks into a stage (fewer barrier round trips)
    a.prow = n >= 128 ? 128 : (n + 7) / 8 * 8;
    a.cs = std::min(4, 128 / a.prow);
    a.nyg = (m + a.nY - 1) / a.nY;
    a.nxt = (n + 127) / 128;
    a.nitems = leaves * a.nxt * a.nyg * a.nW;
    a.went = leaves * m * n;
    a.esize = (a.W + a.dxb) / 8 * LT_CORE;
    a.rsize = std::max(a.dxa, a.nY > 1 ? a.nY * a.dxa : 0) * 2;
}
static size_t ltc_smem(const LtcArgs &a) {
    return LT_STAGES * LT_STAGE + (size_t)LT_HANKEL * a.esize + (size_t)2 * LT_RAW * a.rsize + sizeof(LtcBars) + 1024 + 64;
}
// terms k whose column sums stay inside 32 bits: k (min digits + 2) 2^14 < 2^31
static int ltc_kmax(int la, int lb) { return 131071 / (std::min(ltc_dx(la), ltc_dx(lb)) + 2); }
static size_t ltc_align(size_t x) { return (x + 255) & ~(size_t)255; }

// Device workspace of `leaves` products in one launch.
size_t ltc_ws(int m, int k, int n, int la, int lb, int64_t leaves) {
    LtcArgs a;
    const int kc = std::min(k, ltc_kmax(la, lb));
    ltc_shape(a, m, kc, n, la, lb, leaves);
    return ltc_align((size_t)leaves * m * kc * a.dxa * 2) + ltc_align((size_t)leaves * kc * n * a.dxb * 2) +
           ltc_align((size_t)(a.T / 4) * a.went * 4) + ltc_align((size_t)(a.T / a.seg) * a.went * (k > kc ? 8 : 4)) + 2048;
}

// Estimated time of both forms in microseconds; the tensor form is taken when it is
// faster.  Tensor form: 23.5 us of launches and pipeline fill, then per tile and term k 800
// clocks (the Hankel operand's hand-over) plus the MMAs of the chunks the tile reads, over the
// tiles one SM runs, and the finish: 0.215 us a limb of an entry (one thread takes them one after
// the other) or its traffic at 7.4 TB/s of L2.  CUDA cores: limb_us.  Over 1285 products of 1 to 600
// terms the choice costs 1.5 % against the faster form of each, and five take more than 1.08 times the CUDA
// cores' time (1.17 at most; with a constant for the finish 72, 2.5 at most: 16 x 20 x 64 entries of
// 128 and 16 limbs 28 on the CUDA cores, 65 here).  Measured (us, CUDA cores / tensor):
// 32^3 32 limbs 24 / 63, 64^3 16 limbs 59 / 61, 64^3 33 limbs 141 / 95, 128^3 16 limbs 330 / 90,
// 128^3 64 limbs 1813 / 385, 256^3 8 limbs 575 / 163, 256^3 64 limbs 14002 / 2371,
// 256 x 256 x 16 32 limbs 341 / 420 (16 columns use 16 of 128 lanes), 200 x 40 x 60 16 limbs 113 / 53.
// -1 by the estimate, 0 never, 1 wherever the shape allows it: of this thread's calls
static thread_local int t_ltc_mode = -1;
static bool ltc_allowed(const LtcArgs &a, int k, int n, int64_t leaves) {
    return a.went < ((int64_t)1 << 31) && a.nitems < ((int64_t)1 << 31) && ltc_smem(a) <= 227 * 1024 &&
           leaves * k * n < ((int64_t)1 << 30);
}
static double ltc_tensor_us(const LtcArgs &a, int k) {
    // 16-digit blocks a tile reads per k, averaged over the windows
    double nblk = 0;
    for (int w = 0; w < a.nW; w++) {
        int jlo = 0, jhi = a.dxb - 1;
        if (a.nY == 1) {
            jlo = std::max(0, a.T - a.dxa - w * a.W - a.W + 1);
            jhi = std::max(jlo, std::min(a.dxb - 1, a.T - 1 - w * a.W));
        }
        nblk += std::min(a.dxb / 16, 4 * (jhi / 64 + 1)) - 4 * (jlo / 64);
    }
    nblk /= a.nW;
    const double waves = (double)((a.nitems + num_sms() - 1) / num_sms());
    const double limbs = a.T / 4;
    return 23.5 + waves * k * (800.0 + 1.1 * nblk * a.W / 2) / 2070.0 + 0.215 * limbs + a.went * limbs * 16 / 7.4e6;
}
bool ltc_pays(int m, int k, int n, int la, int lb, int64_t leaves, double slack) {
    if (m < 1 || k < 1 || n < 1 || la < 1 || lb < 1 || t_ltc_mode == 0) return false;
    LtcArgs a;
    ltc_shape(a, m, k, n, la, lb, leaves);
    if (!ltc_allowed(a, k, n, leaves)) return false;
    if (t_ltc_mode == 1) return true;
    return ltc_tensor_us(a, k) < slack * limb_us(la, lb, k, leaves * m * n);
}

// Levels of a Winograd tree (1 .. levels, the depth that the cutoff gives) whose sums,
// leaf products and combinations together are estimated fastest.  Each level has 7/8 of the
// multiplications, but leaves of fewer than 128 columns leave lanes of the MMAs idle, and
// the sums and combinations of a level take about 16 us plus their traffic; above the
// cutoff leaves count whose estimate is within LTC_SHALLOW of the CUDA cores'.  So on the
// tensor cores the tree usually stops at blocks of 64 or more, on the CUDA cores at the
// cutoff.  Products, us (levels, and before at the cutoff's depth): 64^3 16 limbs cutoff 16 98 (1; 151 at 2),
// 128^3 32 limbs cutoff 32 389 (1; 623 at 2), 256^3 64 limbs cutoff 32 3001 (1; 8560 at 3),
// 256^3 3 limbs cutoff 32 150 (1; 232 at 3), 512^3 32 limbs cutoff 32 10614 (2; 28664 at 4).
int ltc_wino_levels(int N, int levels, int la, int lb) {
    if (t_ltc_mode != -1) return levels;
    double sums = 0, best = 1e30;
    int pick = levels;
    int64_t np = 1;
    for (int d = 1; d <= levels; d++, np *= 7) {
        const int hh = N >> d;
        const double e = (double)hh * hh;
        sums += 16.0 + np * e * 4.0 * 19.0 * (la + lb) / 4e6;
        LtcArgs a;
        ltc_shape(a, hh, hh, hh, la, lb, 7 * np);
        double t = d == levels ? limb_us(la, lb, hh, 7 * np * hh * hh) : 1e30;
        if (hh <= ltc_kmax(la, lb) && ltc_pays(hh, hh, hh, la, lb, 7 * np, d < levels ? LTC_SHALLOW : 1.0))
            t = std::min(t, ltc_tensor_us(a, hh));
        if (sums + t < best) {
            best = sums + t;
            pick = d;
        }
    }
    return pick;
}
// Whether ltc_wino_leaves() would run in `room` bytes of workspace.
static int64_t ltc_wino_chunk(int hh, int la, int lb, int64_t leaves, size_t room) {
    const int64_t chunk = std::min<int64_t>(leaves, (int64_t)(room / (ltc_ws(hh, hh, hh, la, lb, 1) + 1)));
    return chunk < 1 || (chunk < leaves && chunk < 64) ? 0 : chunk;
}
bool ltc_wino_fits(int hh, int la, int lb, int64_t leaves, size_t room) {
    return ltc_wino_chunk(hh, la, lb, leaves, room) > 0;
}

gbmm_status make_map(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint64_t pitch_elems,
                     uint32_t box_inner, uint32_t box_outer);  // crt.cu

struct LtcBufs {
    __nv_bfloat16 *da = nullptr, *db = nullptr;
};
// Carves the workspace of one launch from the handle's arena; false when it does not fit.
static bool ltc_carve(gbmm_handle h, LtcArgs &a, LtcBufs &w, int64_t leaves) {
    w.da = (__nv_bfloat16 *)arena_alloc(h, (size_t)leaves * a.m * a.k * a.dxa * 2);
    w.db = (__nv_bfloat16 *)arena_alloc(h, (size_t)leaves * a.k * a.n * a.dxb * 2);
    a.wl = (uint32_t *)arena_alloc(h, (size_t)(a.T / 4) * a.went * 4);
    a.wq = arena_alloc(h, (size_t)(a.T / a.seg) * a.went * (a.chunks ? 8 : 4));
    a.ad = w.da;
    return w.da && w.db && a.wl && a.wq;
}
static gbmm_status ltc_gemm(const LtcArgs &a, const LtcBufs &w, int64_t leaves, cudaStream_t s) {
    CUtensorMap tmP;
    GBMM_TRY(make_map(&tmP, w.db, a.dxb, (uint64_t)leaves * a.k * a.n, a.dxb, 64, (uint32_t)a.prow));
    const size_t smem = ltc_smem(a);
    auto kern = a.chunks ? k_ltc_gemm<true> : k_ltc_gemm<false>;
    GBMM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    LaunchScope ls_("k_ltc_gemm", s);
    kern<<<(unsigned)std::min<int64_t>(a.nitems, num_sms()), LT_THREADS, smem, s>>>(tmP, a, device_error_word());
    GBMM_CUDA_TRY(cudaGetLastError());
    return GBMM_OK;
}
static gbmm_status ltc_finish(const LtcArgs &a, const LtcOut &o, cudaStream_t s) {
    LaunchScope ls_("k_ltc_finish", s);
    k_ltc_finish<<<(unsigned)((a.went + 127) / 128), 128, 0, s>>>(a, o, device_error_word());
    GBMM_CUDA_TRY(cudaGetLastError());
    return GBMM_OK;
}

// C = A B or C += A B on the tensor cores; *done = false (nothing launched) when the
// handle's workspace has no room for it.  The caller checked ltc_pays and that
// the inner dimension is not empty.
gbmm_status ltc_matmul(gbmm_handle h, const gbmm_mat &c, const gbmm_mat &a, const gbmm_mat &b, int accumulate,
                       cudaStream_t s, bool *done) {
    *done = false;
    const int K = a.cols, kc = std::min(K, ltc_kmax(a.nlimbs, b.nlimbs));
    const size_t mark = arena_mark(h);
    LtcArgs full;
    ltc_shape(full, a.rows, kc, b.cols, a.nlimbs, b.nlimbs, 1);
    full.chunks = K > kc;
    LtcBufs w;
    if (!ltc_carve(h, full, w, 1)) {
        arena_release(h, mark);
        return GBMM_OK;
    }
    *done = true;
    gbmm_status st = GBMM_OK;
    for (int k0 = 0; k0 < K && st == GBMM_OK; k0 += kc) {
        const int kn = std::min(kc, K - k0);
        LtcArgs q = full;
        q.k = kn;
        q.later = k0 > 0;
        const gbmm_mat ac = sub_view(a, 0, k0, a.rows, kn), bc = sub_view(b, k0, 0, kn, b.cols);
        for (int side = 0; side < 2; side++) {
            const gbmm_mat &x = side ? bc : ac;
            DigitArgs d;
            d.limbs = x.limbs;
            d.sizes = x.sizes;
            d.ld = x.ld;
            d.rs = x.rs;
            d.rows = x.rows;
            d.cols = x.cols;
            d.nlimbs = x.nlimbs;
            d.transpose = 0;
            d.dxp = side ? q.dxb : q.dxa;
            d.out = side ? w.db : w.da;
            const int nbx = (x.cols + 31) / 32;
            const dim3 grid((unsigned)(nbx * ((x.rows + 3) / 4)), (unsigned)((d.dxp / 4 + 63) / 64));
            LaunchScope ls_("k_ltc_digits", s);
            k_ltc_digits<<<grid, 256, 0, s>>>(d, nbx);
            if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) st = cuda_error(e, "k_ltc_digits");
        }
        if (st == GBMM_OK) st = ltc_gemm(q, w, 1, s);
    }
    LtcOut o;
    memset(&o, 0, sizeof o);
    o.C = c;
    o.accumulate = accumulate;
    if (st == GBMM_OK) st = ltc_finish(full, o, s);
    arena_release(h, mark);
    return st;
}

// All leaf products of a Winograd tree, as many leaves per launch as the handle's
// workspace holds; *done as above.
gbmm_status ltc_wino_leaves(gbmm_handle h, const WinoTree &t, int64_t leaves, cudaStream_t s, bool *done) {
    *done = false;
    const int hh = t.N >> t.levels;
    if (hh > ltc_kmax(t.capSA, t.capSB)) return GBMM_OK;
    const size_t room = h->ws.cap - h->ws.top;
    const int64_t chunk = ltc_wino_chunk(hh, t.capSA, t.capSB, leaves, room);
    if (chunk == 0) return GBMM_OK;
    const size_t mark = arena_mark(h);
    gbmm_status st = GBMM_OK;
    for (int64_t l0 = 0; l0 < leaves && st == GBMM_OK; l0 += chunk) {
        const int64_t nl = std::min(chunk, leaves - l0);
        LtcArgs q;
        ltc_shape(q, hh, hh, hh, t.capSA, t.capSB, nl);
        LtcBufs w;
        if (!ltc_carve(h, q, w, nl)) {
            arena_release(h, mark);
            return l0 == 0 ? GBMM_OK : set_error(GBMM_ERR_NOMEM, "winograd leaves: workspace");
        }
        *done = true;
        const int nbx = (hh + 31) / 32, nby = (hh + 3) / 4;
        for (int side = 0; side < 2; side++) {
            const int dx = side ? q.dxb : q.dxa;
            const dim3 grid((unsigned)(nl * nbx * nby), (unsigned)((dx / 4 + 63) / 64));
            LaunchScope ls_("k_ltc_wino_digits", s);
            k_ltc_wino_digits<<<grid, 256, 0, s>>>(t, side, l0, nbx, nby, dx, side ? w.db : w.da);
            if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) st = cuda_error(e, "k_ltc_wino_digits");
        }
        LtcOut o;
        memset(&o, 0, sizeof o);
        o.pl = t.p_limbs[t.levels] + l0 * (int64_t)hh * hh * t.capP;
        o.ps = t.p_sizes[t.levels] + l0 * (int64_t)hh * hh;
        o.pcap = t.capP;
        if (st == GBMM_OK) st = ltc_gemm(q, w, nl, s);
        if (st == GBMM_OK) st = ltc_finish(q, o, s);
        arena_release(h, mark);
    }
    return st;
}

}  // namespace gbmm

// Test hook: the limb form's products on the tensor cores by the estimate (-1, the
// default), never (0) or wherever the shape allows it (1), in the calls of this thread;
// returns its previous setting.
extern "C" int32_t gbmmx_limb_tc(int32_t mode) {
    const int32_t old = gbmm::t_ltc_mode;
    gbmm::t_ltc_mode = mode < 0 ? -1 : (mode ? 1 : 0);
    return old;
}
