// Multi-modular (CRT) form of the exact product C = A * B on the tcgen05
// tensor cores.
//
// Moduli: the P largest primes below 2^16 with prod p_i = Mod > 2^(bitsA +
// bitsB + log2 k + 18).  Every GEMM below multiplies signed 8-bit digits held
// exactly in bf16 and accumulates in FP32; each accumulation is bounded so that
// every partial sum is an integer of magnitude < 2^24, hence exact.
//
//  1. digits    : limb planes -> rows of byte digits (bf16): unsigned bytes, or for
//                 rows longer than 512 digits balanced digits in [-128, 128]; one
//                 row per entry (A in row-major order, B in column-major order).
//  2. residue   : [entries x digits] x [digits x 2P] GEMM with the table
//                 256^j mod p_i (balanced, split in two signed bytes); the
//                 epilogue folds the two halves, reduces mod p_i in FP32,
//                 applies the entry's sign and stores the residue as two
//                 balanced digits in per-modulus planes.  B's table carries the
//                 CRT weight w_i = (Mod/p_i)^-1 mod p_i.
//                 Rows of up to 512 digits take both steps in one kernel, for both
//                 operands at once (2b below).
//  3. product   : for each modulus, A's two digit planes against B's two
//                 (pre-weighted) digit planes in four accumulators;
//                 y_i = 65536 a1 u1 + 256 (a1 u0 + a0 u1) + a0 u0 mod p_i, stored
//                 balanced as two digits in per-modulus planes.
//  4. reconstruct: [entries x 2P] x [2P x (32 + Dout)] GEMM against the digits
//                 of Mod/p_i (and 256*Mod/p_i) plus fixed-point digits of
//                 2^96/p_i; the epilogue gets q = round(sum y_i / p_i) and the
//                 sign of C, folds out q*Mod, carries across the digit columns
//                 and writes sign-magnitude limbs.  C = sum y_i Mod/p_i - q*Mod.
// The CRT itself is the textbook one (HAC 14.5, Knuth 4.3.2); the reference's
// crt.cpp (split / merge of one integer through a tree of coprime pairs) is
// unused by the reference and only the idea carries over.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <utility>
#include <cmath>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "digits.cuh"
#include "gbmm_internal.h"
#include "tc.cuh"

namespace gbmm {

namespace {
constexpr int BM = 128;  // tile rows (TMEM lanes)
constexpr int BK = 64;   // bf16 elements per K step (one 128-byte swizzle row)
constexpr int UK = 16;   // K of one kind::f16 MMA
// residue GEMM: K steps per exact accumulation group: 8 (512 unsigned byte digits,
// 512 * 255 * 128 < 2^24) or, for rows longer than 512 digits, 15 (960 balanced
// digits, 959 * 128 * 128 + 256 * 128 < 2^24)
constexpr int RES_GROUP_STEPS_U = 8, RES_GROUP_STEPS_B = 15;
constexpr int PROD_MAX_K = 512;      // product GEMM: inner dimension of one exact pass
constexpr int SROWS = 32;       // columns before the first output digit in the reconstruction table
constexpr int SUSED = 14;       // of which the fixed-point sum uses the first 14 (98 bits)
constexpr int FIXB = 96;        // fixed-point bits of the 1/p_i weights
constexpr int CTA_THREADS = 192;   // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int CTA_THREADS8 = 320;  // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue (two per lane quadrant)
constexpr int RES_EPI_WARPS = 16;   // residue GEMM: four epilogue warps per lane quadrant
constexpr int RES_THREADS = 32 * (2 + RES_EPI_WARPS);
constexpr int REC_EPI_WARPS = 16;   // reconstruction: four epilogue warps per lane quadrant
constexpr int REC_THREADS = 32 * (2 + REC_EPI_WARPS);
constexpr int RTAB = 256;          // reconstruction table rows are padded to a multiple of this
}  // namespace

struct ModConst {
    int32_t p;
    float inv_p;
    uint32_t mu;   // floor(2^32 / p)
    uint32_t h16;  // 2^16 mod p
    uint32_t w;    // (Mod / p)^-1 mod p
    uint32_t pad[3];
};

// ---- modular helpers (device) ---------------------------------------------------------
// Every value below is an exact integer held in FP32 with magnitude < 2^24, so
// the reductions run on the FMA pipe with no int<->float conversion.
//
// red(x) = x - rint(x / p) * p for |x| < 2^24 and 2^15 < p < 2^16.  The quotient
// is rounded by adding 1.5 * 2^23 inside one FMA (|x / p| < 2^9 keeps the sum in
// the binade where the ulp is 1); with inv_p = fl(1/p) its error against the
// true x / p is at most 2^9 * 2^-24 = 2^-15, so the result lies in
// [-p/2 - 2, p/2 + 2]: congruent to x, not always the balanced representative.
// The second FMA is exact because the true result is a small integer.
// Downstream bounds use |red(x)| <= 32772.
constexpr float RND_MAGIC = 12582912.0f;  // 1.5 * 2^23

// (p, p', fl(1/p), fl(1/p')) of moduli 2i and 2i+1 for the 1024 largest primes
// below 2^16, in descending order: the moduli of every product are a prefix of
// this list.  Warps read one pair at a time (a constant-cache broadcast, no
// shared-memory traffic); each half is a packed operand of the f32x2 arithmetic.
constexpr int CMOD_PAIRS = 512;
__constant__ float4 c_modpair[CMOD_PAIRS];
__device__ __forceinline__ float red(float x, float p, float inv_p) {
    const float q = __fadd_rn(__fmaf_rn(x, inv_p, RND_MAGIC), -RND_MAGIC);
    return __fmaf_rn(-q, p, x);
}
// r (|r| <= 32772) -> two signed byte digits, r = hi * 256 + lo, |hi|, |lo| <= 128
__device__ __forceinline__ void bal_split(float r, float &hi, float &lo) {
    hi = __fadd_rn(__fmaf_rn(r, 1.0f / 256.0f, RND_MAGIC), -RND_MAGIC);
    lo = __fmaf_rn(-hi, 256.0f, r);
}

// ---- the same steps on two values at once (packed f32x2 arithmetic: one FMA-pipe
// instruction per pair; each lane is rounded exactly as the scalar form) --------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(f32x2 r, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// red on both lanes: np = (-p, -p'), ip = (1/p, 1/p')
__device__ __forceinline__ f32x2 red2(f32x2 x, f32x2 np, f32x2 ip) {
    const f32x2 q = add2(fma2(x, ip, pk2(RND_MAGIC, RND_MAGIC)), pk2(-RND_MAGIC, -RND_MAGIC));
    return fma2(q, np, x);
}
__device__ __forceinline__ void bal_split2(f32x2 r, f32x2 &hi, f32x2 &lo) {
    hi = add2(fma2(r, pk2(1.0f / 256.0f, 1.0f / 256.0f), pk2(RND_MAGIC, RND_MAGIC)), pk2(-RND_MAGIC, -RND_MAGIC));
    lo = fma2(hi, pk2(-256.0f, -256.0f), r);
}
struct Barriers {
    uint64_t full[8];
    uint64_t empty[8];
    uint64_t tfull[2];
    uint64_t tempty[2];
    uint32_t tmem_base;
    int abort_flag;
};
constexpr uint32_t SMEM_BARS = 256;  // bytes reserved for Barriers; per-kernel tables follow
static_assert(sizeof(Barriers) <= SMEM_BARS, "barrier block");

__device__ __forceinline__ uint8_t *align1024(uint8_t *p) {
    uintptr_t v = reinterpret_cast<uintptr_t>(p);
    return reinterpret_cast<uint8_t *>((v + 1023) & ~(uintptr_t)1023);
}

// Common prologue: barrier init by thread 0, TMEM allocation by warp 1.
__device__ __forceinline__ void cta_setup(Barriers *bars, int stages, uint32_t tmem_cols, uint32_t full_count,
                                          uint32_t tempty_count) {
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            tc::mbar_init(&bars->full[s], full_count);
            tc::mbar_init(&bars->empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(&bars->tfull[b], 1);
            tc::mbar_init(&bars->tempty[b], tempty_count);
        }
        bars->abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc(&bars->tmem_base, tmem_cols);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
}

__device__ __forceinline__ void cta_teardown(Barriers *bars, uint32_t tmem_cols) {
    tc::fence_before_sync();
    __syncthreads();
    if ((threadIdx.x >> 5) == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(bars->tmem_base, tmem_cols);
    }
}

__device__ __forceinline__ void set_abort(Barriers *bars, uint32_t *err) {
    atomicOr(err, DEVERR_TIMEOUT);
    *(volatile int *)&bars->abort_flag = 1;
}
__device__ __forceinline__ bool aborted(Barriers *bars) { return *(volatile int *)&bars->abort_flag != 0; }

// epilogue warps 2..5 cover TMEM lane quadrants (warp % 4)
__device__ __forceinline__ int epi_row() { return ((threadIdx.x >> 5) & 3) * 32 + (threadIdx.x & 31); }
__device__ __forceinline__ uint32_t lane_base(uint32_t tmem) { return tmem + (((threadIdx.x >> 5) & 3) * 32u << 16); }
__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// A grouped launch runs the tiles of several products in one persistent kernel.
// Job j owns the global tiles [tile0[j], tile0[j + 1]); every role of a CTA walks
// the same tile sequence and looks each tile's job up by binary search.  The job
// records (arguments and 64-byte aligned tensor maps) sit in global memory.
template <typename J>
struct Group {
    const J *jobs;
    const int64_t *tile0;  // njobs + 1 entries, tile0[njobs] = all tiles
    int32_t njobs;
};
__device__ __forceinline__ int group_job(const int64_t *tile0, int n, int64_t T) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(tile0 + mid) <= T) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
// A role's walk through the tiles only moves forward: the current job and its tile
// range are kept until the walk leaves that range, so most tiles need no lookup
// (the binary search is a chain of dependent loads).
struct GroupCursor {
    int j = -1;
    int64_t beg = 0, end = 0;
    template <typename J>
    __device__ __forceinline__ void seek(const Group<J> &g, int64_t T) {
        if (j >= 0 && T < end) return;
        j = group_job(g.tile0, g.njobs, T);
        beg = __ldg(g.tile0 + j);
        end = __ldg(g.tile0 + j + 1);
    }
};

// ======================================================================================
// 1. digits
// ======================================================================================
// One operand of a grouped digits launch: its blocks are (bx, by, bz) in x-fastest
// order, nbx x nby x (chunks of 64 limbs).
struct DigitJob {
    DigitArgs a;
    int32_t nbx, nby;
};

template <bool BAL, bool GRP>
__global__ void __launch_bounds__(256) k_crt_digits(DigitArgs a0, Group<DigitJob> grp) {
    tc::grid_dep_wait();    // the operand this launch reads is complete
    tc::grid_dep_launch();  // the residue GEMM's CTAs may set up while the last blocks run
    if (GRP) {
        const int j = group_job(grp.tile0, grp.njobs, blockIdx.x);
        const DigitJob &J = grp.jobs[j];
        const int b = (int)(blockIdx.x - __ldg(grp.tile0 + j));
        digits_block<BAL>(J.a, b % J.nbx, (b / J.nbx) % J.nby, b / J.nbx / J.nby);
    } else {
        digits_block<BAL>(a0, blockIdx.x, blockIdx.y, blockIdx.z);
    }
}

// ======================================================================================
// 2. residue GEMM (persistent; TMEM double-buffered so a tile's epilogue overlaps
//    the next tile's MMAs; 16 epilogue warps, four per TMEM lane quadrant)
// ======================================================================================
struct ResidueArgs {
    int32_t kdim;  // entry e -> (e / kdim, e % kdim) in digit-row order
    int32_t E;     // entries (digit rows)
    int32_t nk;    // K steps of 64 digits
    int32_t BN, G; // table columns per tile, accumulation groups (G * BN <= 256)
    int32_t P;
    int32_t ncols;  // table columns: two per modulus, padded to whole pairs of moduli
    int32_t n_ntiles;
    int32_t ntiles;
    __nv_bfloat16 *R;  // planes [2P][rowsR][kp]
    int64_t plane;     // rowsR * kp
    int32_t kp;
    int32_t tma_out;  // kdim % 32 == 0: each warp's 32 entries share a plane row; TMA stores
};
// One operand of a grouped residue launch.
struct ResidueJob {
    CUtensorMap tmD, tmT, tmR;
    ResidueArgs a;
};

// shared-memory staging of one epilogue warp's chunk: [32 planes][32 entries] bf16
constexpr int RES_STG_BYTES = 32 * 32 * 2;

// One chunk of 32 accumulator columns (16 moduli) of group g folded into res.
// The table orders each pair of moduli (m, m') as four columns: [lo_m, lo_m',
// hi_m, hi_m'] (the byte digits of 256^j mod p times 1 and 256), so the lo sums and
// the hi sums of a pair come as packed operands: res = red(256 red(s1) + red(s0)
// (+ res)) on both lanes at once.  Each term is an integer of magnitude <= 2^24;
// the sum stays below 257 * 32772 + 32772 < 2^24, so every FP32 step is exact.
__device__ __forceinline__ void residue_fold(const uint32_t (&v)[32], int mi0, bool first, f32x2 (&res)[8]) {
#pragma unroll
    for (int g = 0; g < 8; g++) {
        const float4 pc = c_modpair[(mi0 >> 1) + g];  // (p, p', 1/p, 1/p')
        const f32x2 np = pk2(-pc.x, -pc.y), ip = pk2(pc.z, pc.w);
        const f32x2 s0 = pk2(__uint_as_float(v[4 * g]), __uint_as_float(v[4 * g + 1]));
        const f32x2 s1 = pk2(__uint_as_float(v[4 * g + 2]), __uint_as_float(v[4 * g + 3]));
        f32x2 t = fma2(red2(s1, np, ip), pk2(256.f, 256.f), red2(s0, np, ip));
        if (!first) t = add2(t, res[g]);
        res[g] = red2(t, np, ip);
    }
}

// PAIR: a cluster of two CTAs shares one M = 256 tcgen05.mma.cta_group::2 per K
// slice (issued by the even CTA); each CTA stages its own 128 entries and half of
// the tile's table columns, and keeps its own 128 rows of D in its TMEM.
// GRP: a grouped launch (single CTAs only); every stage is sized for GBN table
// columns (the launch's operands have table tiles of at most GBN columns).
template <int STAGES, bool PAIR, int GS, bool GRP, int GBN = 256>
__global__ void __launch_bounds__(RES_THREADS, 1)
    k_crt_residue(const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmT,
                  const __grid_constant__ CUtensorMap tmR, ResidueArgs a0, Group<ResidueJob> grp, uint32_t *err) {
    static_assert(!GRP || !PAIR, "grouped residue launches use single CTAs");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = align1024(smem_raw);
    constexpr int NP = PAIR ? 2 : 1;    // row blocks per tile (per cluster)
    constexpr int NBUF = PAIR ? 2 : 1;  // staging buffers per epilogue warp
    const uint32_t A_BYTES = BM * 128, B_BYTES = GRP ? (uint32_t)GBN * 128 : (uint32_t)(PAIR ? a0.BN / 2 : a0.BN) * 128,
                   STAGE = A_BYTES + B_BYTES;
    Barriers *bars = reinterpret_cast<Barriers *>(base + STAGES * STAGE);
    uint8_t *stage_out = reinterpret_cast<uint8_t *>(bars) + SMEM_BARS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? tc::cluster_rank() : 0;
    const int64_t t0 = PAIR ? (blockIdx.x >> 1) : blockIdx.x, tstep = PAIR ? (gridDim.x >> 1) : gridDim.x;
    if (PAIR) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < STAGES; s++) {
                tc::mbar_init(&bars->full[s], 1);
                tc::mbar_init(&bars->empty[s], 1);
            }
            for (int b = 0; b < 2; b++) {
                tc::mbar_init(&bars->tfull[b], 1);
                tc::mbar_init(&bars->tempty[b], 2 * RES_EPI_WARPS);  // the even CTA's: every epilogue warp of both CTAs
            }
            bars->abort_flag = 0;
            tc::fence_mbar_init();
        }
        if (warp == 1) {
            tc::tmem_alloc_pair(&bars->tmem_base, 512);
            tc::tmem_relinquish_pair();
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
        tc::fence_after_sync();
    } else {
        cta_setup(bars, STAGES, 512, 1, RES_EPI_WARPS);
    }
    tc::grid_dep_wait();  // the digits this launch reads are complete
    const uint32_t tmem = bars->tmem_base;
    // the last table tile may be narrow: its MMA has only the columns it needs
    // (a multiple of 16, of 32 for a pair so that each CTA stages whole 8-row groups)
    const int ngran = PAIR ? 32 : 16;
    const int64_t total = GRP ? grp.tile0[grp.njobs] : (int64_t)a0.ntiles;
    // global tile T -> its operand's arguments and maps, and the tile within it
    GroupCursor cur;
    auto tile_job = [&](int64_t T, ResidueArgs &a, const CUtensorMap *&mD, const CUtensorMap *&mT,
                        const CUtensorMap *&mR) -> int {
        if (GRP) {
            cur.seek(grp, T);
            const ResidueJob *J = grp.jobs + cur.j;
            a = J->a;
            mD = &J->tmD;
            mT = &J->tmT;
            mR = &J->tmR;
            return (int)(T - cur.beg);
        }
        a = a0;
        mD = &tmD;
        mT = &tmT;
        mR = &tmR;
        return (int)T;
    };

    if (warp == 0) {
        if (tc::elect_one()) {
            if (!GRP) {
                tc::prefetch_tmap(&tmD);
                tc::prefetch_tmap(&tmT);
            }
            int it = 0;
            for (int64_t T = t0; T < total && !aborted(bars); T += tstep) {
                ResidueArgs a;
                const CUtensorMap *mD, *mT, *mR;
                const int t = tile_job(T, a, mD, mT, mR);
                (void)mR;
                const int rb = t / a.n_ntiles;
                const int e0 = rb * (NP * BM) + (int)rank * BM;
                const int n0 = (t - rb * a.n_ntiles) * a.BN;
                const int nn = min(a.BN, (a.ncols - n0 + ngran - 1) / ngran * ngran);
                for (int s = 0; s < a.nk; s++, it++) {
                    const int st = it % STAGES;
                    if (it >= STAGES && !tc::mbar_wait(&bars->empty[st], ((it / STAGES) & 1) ^ 1)) {
                        set_abort(bars, err);
                        break;
                    }
                    uint8_t *sa = base + st * STAGE;
                    if (PAIR) {
                        // this CTA's half of the tile's columns: n0 + rank * nn / 2 onwards
                        const uint32_t full0 = tc::mapa(tc::smem_u32(&bars->full[st]), 0);
                        if (rank == 0) tc::mbar_arrive_expect_tx(&bars->full[st], 2 * STAGE);
                        tc::tma_load_2d_pair(sa, mD, full0, s * BK, (int)e0);
                        tc::tma_load_2d_pair(sa + A_BYTES, mT, full0, s * BK, n0 + (int)rank * (nn / 2));
                    } else {
                        // a grouped stage holds this operand's BN table rows of its 256
                        tc::mbar_arrive_expect_tx(&bars->full[st], GRP ? A_BYTES + (uint32_t)a.BN * 128 : STAGE);
                        tc::tma_load_2d(sa, mD, &bars->full[st], s * BK, (int)e0);
                        tc::tma_load_2d(sa + A_BYTES, mT, &bars->full[st], s * BK, n0);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && tc::elect_one()) {
            int it = 0, lt = 0;
            bool ok = true;
            for (int64_t T = t0; T < total && ok; T += tstep, lt++) {
                ResidueArgs a;
                const CUtensorMap *mD, *mT, *mR;
                const int t = tile_job(T, a, mD, mT, mR);
                (void)mD, (void)mT, (void)mR;
                const int b = lt & 1;
                const int n0 = (t % a.n_ntiles) * a.BN;
                const int nn = min(a.BN, (a.ncols - n0 + ngran - 1) / ngran * ngran);
                const uint32_t idesc = tc::idesc_bf16_f32(PAIR ? 2 * BM : BM, nn, 0, 0);
                if (lt >= 2 && !tc::mbar_wait(&bars->tempty[b], ((lt >> 1) & 1) ^ 1)) { set_abort(bars, err); break; }
                tc::fence_after_sync();
                for (int s = 0; s < a.nk; s++, it++) {
                    const int st = it % STAGES;
                    if (!tc::mbar_wait(&bars->full[st], (it / STAGES) & 1)) { set_abort(bars, err); ok = false; break; }
                    tc::fence_after_sync();
                    const uint32_t sa = tc::smem_u32(base + st * STAGE);
                    // accumulation group s / GS (GS K steps each, a compile-time constant: the
                    // issuing thread is on the critical path)
                    const uint32_t d = tmem + (uint32_t)(256 * b + (s / GS) * a.BN);
                    const uint64_t ad = tc::sdesc_kmajor(sa), bd = tc::sdesc_kmajor(sa + A_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / UK; kk++) {
                        const uint64_t adesc = tc::sdesc_advance(ad, kk * 32), bdesc = tc::sdesc_advance(bd, kk * 32);
                        const uint32_t acc = (s % GS) != 0 || kk != 0;
                        if (PAIR) tc::mma_bf16_pair(d, adesc, bdesc, idesc, acc);
                        else tc::mma_bf16(d, adesc, bdesc, idesc, acc);
                    }
                    if (PAIR) tc::mma_commit_pair(&bars->empty[st], 0x3);
                    else tc::mma_commit(&bars->empty[st]);
                }
                if (ok) {
                    if (PAIR) tc::mma_commit_pair(&bars->tfull[b], 0x3);
                    else tc::mma_commit(&bars->tfull[b]);
                }
            }
        }
    } else {
        // epilogue: warp (2..17) -> lane quadrant warp % 4, column slot (warp - 2) / 4
        // of cpw chunks of 32 columns.  A warp's work on a tile is its live chunks
        // times G groups ("units", one 32-column TMEM load each), chunk-major.  Four
        // warps per scheduler hide the loads' latency.
        const int quad = warp & 3, slot = (warp - 2) >> 2;
        const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t tempty0 = PAIR ? tc::mapa(tc::smem_u32(&bars->tempty[0]), 0) : 0;
        uint16_t *stg = reinterpret_cast<uint16_t *>(stage_out + (warp - 2) * NBUF * RES_STG_BYTES);
        int lt = 0, sbuf = 0;
        for (int64_t T = t0; T < total; T += tstep, lt++) {
            ResidueArgs a;
            const CUtensorMap *mD, *mT, *mR;
            const int t = tile_job(T, a, mD, mT, mR);
            (void)mD, (void)mT;
            const int cpw = max(1, a.BN / 128);                          // chunks per warp
            const int hcols = slot * cpw * 32;                           // the warp's first column in a tile
            const int nch = max(0, min(cpw, (a.BN - hcols) / 32)), G = a.G;
            const int64_t pstep = 2 * a.plane;  // planes of one modulus
            const uint32_t kdim = (uint32_t)a.kdim, E = (uint32_t)a.E;
            const int b = lt & 1;
            const int rb = t / a.n_ntiles;
            const int n0 = (t - rb * a.n_ntiles) * a.BN;
            const uint32_t ew = (uint32_t)rb * (NP * BM) + rank * BM + quad * 32;  // the warp's first entry
            const uint32_t e = ew + lane;
            if (!tc::mbar_wait(&bars->tfull[b], (lt >> 1) & 1)) { set_abort(bars, err); break; }
            tc::fence_after_sync();
            const uint32_t rw = ew / kdim, cw = ew - rw * kdim;  // plane row and column of the warp's box
            const uint32_t re = e / kdim;
            const int64_t off = e < E ? (int64_t)re * a.kp + (e - re * kdim) : 0;
            const int c00 = n0 + hcols;  // the warp's first table column
            const int nlive = max(0, min(nch, (a.ncols - c00 + 31) / 32));
            const int nunits = nlive * G;
            auto release = [&]() {
                // last TMEM read of this tile by this warp: hand the buffer back
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) tc::mbar_arrive_cluster(tempty0 + 8u * b);
                    else tc::mbar_arrive(&bars->tempty[b]);
                }
            };
            if (nunits == 0) {
                release();
                continue;
            }
            f32x2 res[8];  // moduli (mi0 + 2g, mi0 + 2g + 1) of the current chunk
            auto store = [&](int mi0) {
                // bf16 bits of the two balanced byte digits of each residue
                uint16_t hb[16], lbits[16];
#pragma unroll
                for (int g = 0; g < 8; g++) {
                    f32x2 h2, l2;
                    bal_split2(res[g], h2, l2);
                    float h0, h1, l0, l1;
                    upk2(h2, h0, h1);
                    upk2(l2, l0, l1);
                    hb[2 * g] = (uint16_t)(__float_as_uint(h0) >> 16);
                    hb[2 * g + 1] = (uint16_t)(__float_as_uint(h1) >> 16);
                    lbits[2 * g] = (uint16_t)(__float_as_uint(l0) >> 16);
                    lbits[2 * g + 1] = (uint16_t)(__float_as_uint(l1) >> 16);
                }
                if (a.tma_out) {
                    if (ew >= E) return;  // the whole box lies past the last entry
                    if (lane == 0) tc::bulk_wait_read<NBUF - 1>();
                    __syncwarp();
                    uint16_t *buf = stg + sbuf * (RES_STG_BYTES / 2);
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        buf[(2 * j) * 32 + lane] = hb[j];
                        buf[(2 * j + 1) * 32 + lane] = lbits[j];
                    }
                    tc::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        // planes past 2P and rows past the last entry are clipped by the map
                        tc::tma_store_3d(mR, buf, (int)cw, (int)rw, 2 * mi0);
                        tc::bulk_commit_group();
                    }
                    if (NBUF > 1) sbuf ^= 1;
                } else if (e < E) {
                    uint16_t *dst = reinterpret_cast<uint16_t *>(a.R + (int64_t)mi0 * pstep + off);
                    const int nj = a.P - mi0;
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        if (j >= nj) break;
                        dst[j * pstep] = hb[j];
                        dst[j * pstep + a.plane] = lbits[j];
                    }
                }
            };
            int lch = 0, lg = 0;  // the next unit to load
            auto load_next = [&](uint32_t(&v)[32]) {
                tc::tmem_ld32(lb + (uint32_t)(256 * b + lg * a.BN + hcols + lch * 32), v);
                if (++lg == G) {
                    lg = 0;
                    lch++;
                }
            };
            int cch = 0, cg = 0;  // the next unit to fold
            auto consume = [&](const uint32_t(&v)[32]) {
                const int mi0 = (c00 + cch * 32) >> 1;
                residue_fold(v, mi0, cg == 0, res);
                if (cg == G - 1) store(mi0);
                if (++cg == G) {
                    cg = 0;
                    cch++;
                }
            };
            uint32_t va[32];
            for (int u = 0; u < nunits; u++) {
                load_next(va);
                tc::tmem_ld_wait(va);
                if (u + 1 == nunits) release();
                consume(va);
            }
        }
        if (lane == 0) tc::bulk_wait_all();  // staging buffers stay live until the stores finish
        __syncwarp();
    }
    tc::grid_dep_launch();
    if (PAIR) {
        tc::fence_before_sync();
        __syncthreads();
        tc::cluster_sync_all();  // no CTA leaves while its peer may still signal it or write its TMEM
        if (warp == 1) {
            tc::fence_after_sync();
            tc::tmem_dealloc_pair(tmem, 512);
        }
    } else {
        cta_teardown(bars, 512);
    }
}

// ======================================================================================
// 2b. digits and residues of an operand in one kernel, for rows of up to 512 digits
//
// A cluster of two CTAs takes 256 entries (8 plane rows x 32 columns k) and keeps
// their digits in shared memory for all of the table's columns: eight converter warps
// per CTA turn the limb planes into unsigned byte digits in bf16, straight into the
// K-major swizzled operand tiles (64 digits a slot), and the table's column tiles stream
// through a ring.  One M = 256, N = 256 tcgen05.mma.cta_group::2 per K slice.
// Against the digits kernel followed by the streaming GEMM above, which re-read each
// digit tile for every 256 table columns, the digit rows are neither written nor read
// (0.8 GB per operand at 512 x 512 entries of 4096 bits by 516 moduli), and a K step brings 16 KB into
// an SM instead of 48.  With both operands in one launch, us, digits and residues of both
// (two kernels each before): 64 x 64 entries of 1024 bits 16.1 (36.6), 256 x 256 of 2048 bits
// 75 (105), 512 x 512 of 4096 bits 484 (604).  There no unit is saturated (tensor pipe 51 %,
// load/store pipe 40 %, DRAM 33 %): the issue thread waits for the table's tiles and for the
// epilogue in turn, the epilogue for tensor memory.
// ======================================================================================
constexpr int R2_SLOTS = 8;   // digit tiles of 64 digits x 128 entries
// Table tiles of 64 digits x 128 rows, and staging buffers per epilogue warp: what is left of
// shared memory (512 x 512 entries of 4096 bits, us: 5 and 1 515, 4 and 2 527; the epilogue
// storing residues straight to memory, and 6 tiles, 822)
constexpr int R2_STAGES = 5, R2_NBUF = 1;
constexpr int R2_EPI = 8, R2_CONV = 8;  // epilogue and converter warps
constexpr int R2_THREADS = 32 * (2 + R2_EPI + R2_CONV);
constexpr uint32_t R2_TILE = 128 * 128;

struct Residue2Args {
    const uint32_t *limbs;
    const int32_t *sizes;
    int64_t ld, srow, sk;  // entry (plane row, k) at srow * row + sk * k
    int32_t rows, kdim, nlimbs;
    int32_t hrows, hl;     // a limb-half split read in place (0: none): plane rows from hrows on are
                           // the high halves (limbs hl ..) of rows 0 .., the others the low hl limbs
    int32_t nk, ncols, n_ntiles;
    int32_t nkb, ngr;      // blocks of 32 columns k; column-tile groups a row block is split into
    int32_t units;         // row blocks x groups
    int32_t BN;            // table columns per tile (a multiple of 32, at most 256)
};
struct Residue2Job {
    CUtensorMap tmT, tmR;
    Residue2Args a;
};
// unit u: its first plane row, first k and column tiles [j0, j1)
struct Residue2Unit {
    int row0, k0, j0, j1;
};
__device__ __forceinline__ Residue2Unit residue2_unit(const Residue2Args &a, int u) {
    Residue2Unit r;
    const int rb = u / a.ngr, gi = u - rb * a.ngr;
    const int rg = rb / a.nkb;
    r.row0 = rg * 8;
    r.k0 = (rb - rg * a.nkb) * 32;
    r.j0 = (int)((int64_t)a.n_ntiles * gi / a.ngr);
    r.j1 = (int)((int64_t)a.n_ntiles * (gi + 1) / a.ngr);
    return r;
}
struct Residue2Bars {
    uint64_t full[R2_STAGES], empty[R2_STAGES], afull[R2_SLOTS], aempty[R2_SLOTS], tfull[2], tempty[2];
    uint32_t tmem_base;
    int abort_flag;
};

// One or both operands of a product as a kernel parameter (the second with 0 units: none).
struct Residue2Two {
    Residue2Job j[2];
};

template <bool GRP>
__global__ void __launch_bounds__(R2_THREADS, 1)
    k_crt_residue2(const __grid_constant__ Residue2Two two, Group<Residue2Job> grp, uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = align1024(smem_raw);
    uint8_t *tbase = base + R2_SLOTS * R2_TILE, *stage_out = tbase + R2_STAGES * R2_TILE;
    Residue2Bars *bars = reinterpret_cast<Residue2Bars *>(stage_out + R2_EPI * R2_NBUF * RES_STG_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();
    if (threadIdx.x == 0) {
        for (int i = 0; i < R2_STAGES; i++) {
            tc::mbar_init(&bars->full[i], 1);
            tc::mbar_init(&bars->empty[i], 1);
        }
        for (int i = 0; i < R2_SLOTS; i++) {
            tc::mbar_init(&bars->afull[i], 2 * R2_CONV);  // the even CTA's: both CTAs' converter warps
            tc::mbar_init(&bars->aempty[i], 1);
        }
        for (int b = 0; b < 2; b++) {
            tc::mbar_init(&bars->tfull[b], 1);
            tc::mbar_init(&bars->tempty[b], 2 * R2_EPI);
        }
        bars->abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc_pair(&bars->tmem_base, 512);
        tc::tmem_relinquish_pair();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
    tc::fence_after_sync();
    tc::grid_dep_wait();
    const uint32_t tmem = bars->tmem_base;
    auto give_up = [&]() {
        atomicOr(err, DEVERR_TIMEOUT);
        *(volatile int *)&bars->abort_flag = 1;
    };
    const int64_t units0 = two.j[0].a.units;
    const int64_t total = GRP ? grp.tile0[grp.njobs] : units0 + two.j[1].a.units;
    const int64_t t0 = blockIdx.x >> 1, tstep = gridDim.x >> 1;
    GroupCursor cur;
    auto job = [&](int64_t T, Residue2Args &a, const CUtensorMap *&mT, const CUtensorMap *&mR) -> Residue2Unit {
        if (GRP) {
            cur.seek(grp, T);
            const Residue2Job *J = grp.jobs + cur.j;
            a = J->a;
            mT = &J->tmT;
            mR = &J->tmR;
            return residue2_unit(a, (int)(T - cur.beg));
        }
        const int second = T >= units0;
        a = two.j[second].a;
        mT = &two.j[second].tmT;
        mR = &two.j[second].tmR;
        return residue2_unit(a, (int)(T - (second ? units0 : 0)));
    };
    // the column tiles of a unit in order jj = 0, 1, ..: the narrow last tile first, so that
    // the digit slots come free one K step at a time during a whole tile
    auto col_tile = [](const Residue2Args &a, const Residue2Unit &U, int jj, int &n0, int &nn) {
        const int n = U.j1 - U.j0, j = U.j0 + (jj + n - 1) % n;
        n0 = j * a.BN;
        nn = min(a.BN, (a.ncols - n0 + 31) / 32 * 32);
    };

    if (warp == 0) {
        if (tc::elect_one()) {
            int st = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int64_t T = t0; T < total && ok; T += tstep) {
                Residue2Args a;
                const CUtensorMap *mT, *mR;
                const Residue2Unit U = job(T, a, mT, mR);
                for (int jj = 0; jj < U.j1 - U.j0 && ok; jj++) {
                    int n0, nn;
                    col_tile(a, U, jj, n0, nn);
                    for (int s = 0; s < a.nk; s++) {
                        if (!tc::mbar_wait(&bars->empty[st], ph)) {
                            give_up();
                            ok = false;
                            break;
                        }
                        const uint32_t full0 = tc::mapa(tc::smem_u32(&bars->full[st]), 0);
                        if (rank == 0) tc::mbar_arrive_expect_tx(&bars->full[st], 2 * a.BN / 2 * 128);
                        tc::tma_load_2d_pair(tbase + st * R2_TILE, mT, full0, s * BK, n0 + (int)rank * (nn / 2));
                        if (++st == R2_STAGES) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && tc::elect_one()) {
            const uint64_t ad0 = tc::sdesc_kmajor(tc::smem_u32(base)), bd0 = tc::sdesc_kmajor(tc::smem_u32(tbase));
            int st = 0, lt = 0;
            uint32_t ph = 0, sc = 0;  // sc: digit slots used before this unit
            bool ok = true;
            for (int64_t T = t0; T < total && ok; T += tstep) {
                Residue2Args a;
                const CUtensorMap *mT, *mR;
                const Residue2Unit U = job(T, a, mT, mR);
                (void)mT, (void)mR;
                const int nj = U.j1 - U.j0;
                for (int jj = 0; jj < nj && ok; jj++, lt++) {
                    int n0, nn;
                    col_tile(a, U, jj, n0, nn);
                    const uint32_t idesc = tc::idesc_bf16_f32(2 * BM, (uint32_t)nn, 0, 0);
                    const int b = lt & 1;
                    if (lt >= 2 && !tc::mbar_wait(&bars->tempty[b], ((lt >> 1) & 1) ^ 1)) { give_up(); ok = false; break; }
                    const uint32_t d = tmem + 256u * b;
                    for (int s = 0; s < a.nk; s++) {
                        const uint32_t slot = (sc + s) % R2_SLOTS;
                        if (jj == 0 && !tc::mbar_wait(&bars->afull[slot], ((sc + s) / R2_SLOTS) & 1)) { give_up(); ok = false; break; }
                        if (!tc::mbar_wait(&bars->full[st], ph)) { give_up(); ok = false; break; }
                        tc::fence_after_sync();
                        const uint64_t ad = tc::sdesc_advance(ad0, slot * R2_TILE), bd = tc::sdesc_advance(bd0, st * R2_TILE);
#pragma unroll
                        for (int kk = 0; kk < BK / UK; kk++)
                            tc::mma_bf16_pair(d, tc::sdesc_advance(ad, kk * 32), tc::sdesc_advance(bd, kk * 32), idesc,
                                              s != 0 || kk != 0);
                        tc::mma_commit_pair(&bars->empty[st], 0x3);
                        if (jj + 1 == nj) tc::mma_commit_pair(&bars->aempty[slot], 0x3);
                        if (++st == R2_STAGES) {
                            st = 0;
                            ph ^= 1;
                        }
                    }
                    if (ok) tc::mma_commit_pair(&bars->tfull[b], 0x3);
                }
                sc += (uint32_t)a.nk;
            }
        }
    } else if (warp < 2 + R2_EPI) {
        // epilogue: lane quadrant warp % 4 (one plane row, lane = k), four of a tile's (up to)
        // eight 32-column chunks
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 128);
        const uint32_t tempty0 = tc::mapa(tc::smem_u32(&bars->tempty[0]), 0);
        uint16_t *stg = reinterpret_cast<uint16_t *>(stage_out + (warp - 2) * R2_NBUF * RES_STG_BYTES);
        int lt = 0, sbuf = 0;
        bool ok = true;
        for (int64_t T = t0; T < total && ok; T += tstep) {
            Residue2Args a;
            const CUtensorMap *mT, *mR;
            const Residue2Unit U = job(T, a, mT, mR);
            (void)mT;
            const int row = U.row0 + (int)rank * 4 + quad;
            for (int jj = 0; jj < U.j1 - U.j0; jj++, lt++) {
                int n0, nn;
                col_tile(a, U, jj, n0, nn);
                const int b = lt & 1;
                if (!tc::mbar_wait(&bars->tfull[b], (lt >> 1) & 1)) { give_up(); ok = false; break; }
                tc::fence_after_sync();
                const int mi00 = (n0 + half * 128) >> 1;
                const int nch = max(0, min(4, (min(nn, a.ncols - n0) - half * 128 + 31) / 32));
                auto release = [&]() {
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive_cluster(tempty0 + 8u * b);
                };
                auto chunk = [&](int ch, const uint32_t(&v)[32]) {
                    const int mi0 = mi00 + 16 * ch;
                    f32x2 res[8];
                    residue_fold(v, mi0, true, res);
                    if (row >= a.rows) return;
                    if (lane == 0) tc::bulk_wait_read<R2_NBUF - 1>();
                    __syncwarp();
                    uint16_t *buf = stg + sbuf * (RES_STG_BYTES / 2);
#pragma unroll
                    for (int g = 0; g < 8; g++) {
                        f32x2 h2, l2;
                        bal_split2(res[g], h2, l2);
                        float h0, h1, x0, x1;
                        upk2(h2, h0, h1);
                        upk2(l2, x0, x1);
                        buf[(4 * g) * 32 + lane] = (uint16_t)(__float_as_uint(h0) >> 16);
                        buf[(4 * g + 1) * 32 + lane] = (uint16_t)(__float_as_uint(x0) >> 16);
                        buf[(4 * g + 2) * 32 + lane] = (uint16_t)(__float_as_uint(h1) >> 16);
                        buf[(4 * g + 3) * 32 + lane] = (uint16_t)(__float_as_uint(x1) >> 16);
                    }
                    tc::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        // planes past 2P and columns past kdim are clipped by the map
                        tc::tma_store_3d(mR, buf, U.k0, row, 2 * mi0);
                        tc::bulk_commit_group();
                    }
                    if (R2_NBUF > 1) sbuf ^= 1;
                };
                if (nch == 0) release();
#pragma unroll 1
                for (int ch = 0; ch < nch; ch++) {
                    uint32_t v[32];
                    tc::tmem_ld32(lb + (uint32_t)(256 * b + 32 * ch), v);
                    tc::tmem_ld_wait(v);
                    if (ch == nch - 1) release();
                    chunk(ch, v);
                }
            }
        }
        if (lane == 0) tc::bulk_wait_all();  // staging buffers stay live until the stores finish
        __syncwarp();
    } else {
        // converters: two threads per entry, 8 of a slot's 16 limbs each.  A's entries lie
        // along k (lane = k); B's along the plane row x, so its warps take 8 k by 4 x.
        const int ct = (warp - 2 - R2_EPI) * 32 + lane, part = ct >> 7;
        const uint32_t afull0 = tc::mapa(tc::smem_u32(&bars->afull[0]), 0);
        // All of a unit's limbs are loaded while the unit before it runs: its slots come free
        // only during that unit's last column tile, and then each has to be filled in a K
        // step's time (with a slot's loads issued one slot ahead, the GEMM waited for memory
        // most of the time: 677 us for both operands at 512 x 512 entries of 4096 bits).
        uint32_t sc = 0;
        uint32_t v[R2_SLOTS][8];
        int nk = 0, entry = 0;
        uint32_t flip = 0;
        auto fetch = [&](int64_t T) {
            Residue2Args a;
            const CUtensorMap *mT, *mR;
            const Residue2Unit U = job(T, a, mT, mR);
            (void)mT;
            int q, kk;
            if (a.sk == 1) {
                q = (ct & 127) >> 5;
                kk = lane;
            } else {
                q = lane >> 3;
                kk = (((ct & 127) >> 5) << 3) + (lane & 7);
            }
            entry = q * 32 + kk;
            int row = U.row0 + (int)rank * 4 + q;
            const int k = U.k0 + kk;
            const bool live = row < a.rows && k < a.kdim;
            int l0 = 0, nl = a.hrows ? a.hl : a.nlimbs;
            if (a.hrows && row >= a.hrows) {
                row -= a.hrows;
                l0 = a.hl;
                nl = a.nlimbs - a.hl;
            }
            const int64_t off = live ? row * a.srow + k * a.sk : 0;
            if (!live) nl = 0;
            flip = live && a.sizes[off] < 0 ? 0x80008000u : 0u;  // the digits carry the entry's sign
            nk = a.nk;
            const uint32_t *src = a.limbs + off + (int64_t)(l0 + 8 * part) * a.ld;
            nl -= 8 * part;
#pragma unroll
            for (int s = 0; s < R2_SLOTS; s++)
#pragma unroll
                for (int i = 0; i < 8; i++) v[s][i] = 16 * s + i < nl ? src[(int64_t)(16 * s + i) * a.ld] : 0u;
        };
        bool ok = true;
        if (t0 < total) fetch(t0);
        for (int64_t T = t0; T < total && ok; T += tstep) {
            uint8_t *drow = base + entry * 128;
#pragma unroll
            for (int s = 0; s < R2_SLOTS; s++) {
                if (s >= nk || !ok) continue;
                const uint32_t slot = sc % R2_SLOTS;
                if (sc >= R2_SLOTS && !tc::mbar_wait(&bars->aempty[slot], ((sc / R2_SLOTS) & 1) ^ 1)) {
                    give_up();
                    ok = false;
                    continue;
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t v0 = v[s][2 * c], v1 = v[s][2 * c + 1];
                    *reinterpret_cast<uint4 *>(drow + slot * R2_TILE + 16 * ((4 * part + c) ^ (entry & 7))) =
                        make_uint4(byte_pair_bf16(v0, 0) ^ flip, byte_pair_bf16(v0, 2) ^ flip, byte_pair_bf16(v1, 0) ^ flip,
                                   byte_pair_bf16(v1, 2) ^ flip);
                }
                tc::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive_cluster(afull0 + 8u * slot);
                sc++;
            }
            if (T + tstep < total) fetch(T + tstep);
        }
    }
    tc::grid_dep_launch();
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync_all();  // no CTA leaves while its peer may still signal it or write its TMEM
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc_pair(tmem, 512);
    }
}

// ======================================================================================
// 3. per-modulus product GEMM (persistent over (modulus, 128 x 64 output tiles);
//    TMEM double-buffered; 8 epilogue warps)
//
// With a = 256 a1 + a0 (residues of A as balanced digits) and u = 256 u1 + u0
// (residues of B, already multiplied by the CRT weight w = (Mod/p)^-1 mod p),
// the weighted product is
//     y = a b w = 65536 a1 u1 + 256 (a1 u0 + a0 u1) + a0 u0   (mod p).
// The epilogue takes 256 (256 d11 + d10 + d01) + d00 mod p on two columns at a time (packed
// FP32), three reductions for an entry.  With a short inner dimension it is what bounds the kernel:
// reads of tensor memory, staging and stores keep the load/store pipe two thirds busy and the warps wait
// for one another's data.  1024 x 64 x 1024 by 259 moduli 302 us, 380 with five scalar
// reductions; 512 x 512 x 512 by 516 moduli 350 us, 390 (the MMAs alone: 295).  Sixteen epilogue
// warps, 16 columns each or on alternate tiles, were no faster (321-350 and 306 us).
// Each K step issues two N = 128 MMAs against the stacked operand [U1; U0]:
// A1 into [a1 u1 | a1 u0] and A0 into [a0 u1 | a0 u0].  Each of the four 64-column
// accumulators sums k products of magnitude <= 2^14: at most 2^23 for k <= 512,
// and the middle pair adds to at most 2^24.
// ======================================================================================
struct ProductArgs {
    int32_t m, n, nk, P;
    int32_t npad;      // entry row pitch of Y: n rounded up to 16 (entry e = y * npad + x)
    int32_t nyt, nxt;
    int64_t ntiles;
    __nv_bfloat16 *Y;  // blocked [Ep/64][2Pp][64]: 64 entries per row, 2Pp rows per block
    int64_t yblk;      // elements per 64-entry block (2Pp * 64)
};
// One product of a grouped product launch.
struct ProductJob {
    CUtensorMap tmA, tmB;
    ProductArgs a;
};
constexpr int PBX = 64;  // output columns per product tile
constexpr int YPAD = 16;  // Y's entry rows are padded to a multiple of this (whole 32-byte runs)

// Staging of one epilogue warp's 32 rows x 32 columns of one plane of Y, and its store:
// four lanes write a row's 64 bytes, so a store instruction covers 8 rows in whole runs
// (from the rows' own lanes it touched 32 rows with 16 bytes each: every 16 bytes a request
// of its own to L2, 17 million for 512 x 512 entries by 259 moduli, which bounded
// products with a short inner dimension).  Rows of Y are padded to whole groups of
// 16 entries, so a 16-byte chunk of 8 lies inside one 64-entry block.
constexpr int PROD_STG_BYTES = 32 * 32 * 2;
__device__ __forceinline__ void store_plane(const ProductArgs &a, const uint4 *stg, int plane, int y0, int xh) {
    const int lane = threadIdx.x & 31, c = lane & 3;
    const int x = xh + 8 * c;
    uint8_t *yp = reinterpret_cast<uint8_t *>(a.Y) + (int64_t)plane * 128;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = 8 * i + (lane >> 2), y = y0 + row;
        const uint4 v = stg[row * 4 + (c ^ ((row >> 1) & 3))];
        const int64_t e = (int64_t)y * a.npad + x;
        if (y < a.m && x < a.npad)
            *reinterpret_cast<uint4 *>(yp + 2 * ((e >> 6) * a.yblk + (e & 63))) = v;
    }
}

// PAIR: a cluster of two CTAs shares one M = 256 tcgen05.mma.cta_group::2 per K
// slice (issued by the even CTA): each CTA stages its own 128 rows of A1 and A0,
// the even CTA U1's 64 rows and the odd CTA U0's, so per SM a K step moves 40 KB
// instead of 48 KB and the MMAs read 12 KB of shared memory instead of 16 KB.
template <int STAGES, bool PAIR, bool GRP>
__global__ void __launch_bounds__(CTA_THREADS8, 1)
    k_crt_product(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, ProductArgs a0,
                  Group<ProductJob> grp, uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = align1024(smem_raw);
    constexpr int NP = PAIR ? 2 : 1;
    // A1, A0 (128 rows each), then U1, U0 (64 rows each; one of them per CTA of a pair):
    // together the 128-row B operand [U1; U0]
    constexpr uint32_t A_BYTES = BM * 128, B_BYTES = PBX * 128, STAGE = 2 * A_BYTES + (3 - NP) * B_BYTES;
    Barriers *bars = reinterpret_cast<Barriers *>(base + STAGES * STAGE);
    uint8_t *stage_out = reinterpret_cast<uint8_t *>(bars) + SMEM_BARS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? tc::cluster_rank() : 0;
    const int64_t t0 = PAIR ? (blockIdx.x >> 1) : blockIdx.x, tstep = PAIR ? (gridDim.x >> 1) : gridDim.x;
    if (PAIR) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < STAGES; s++) {
                tc::mbar_init(&bars->full[s], 1);
                tc::mbar_init(&bars->empty[s], 1);
            }
            for (int b = 0; b < 2; b++) {
                tc::mbar_init(&bars->tfull[b], 1);
                tc::mbar_init(&bars->tempty[b], 16);  // the even CTA's: 8 epilogue warps of each CTA
            }
            bars->abort_flag = 0;
            tc::fence_mbar_init();
        }
        if (warp == 1) {
            tc::tmem_alloc_pair(&bars->tmem_base, 512);
            tc::tmem_relinquish_pair();
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
        tc::fence_after_sync();
    } else {
        cta_setup(bars, STAGES, 512, 1, 8);
    }
    tc::grid_dep_wait();  // the planes this launch reads are complete
    const uint32_t tmem = bars->tmem_base;
    const int64_t total = GRP ? grp.tile0[grp.njobs] : a0.ntiles;
    // global tile T -> its product's arguments and maps, and the tile within it
    GroupCursor cur;
    auto tile_job = [&](int64_t T, ProductArgs &a, const CUtensorMap *&mA, const CUtensorMap *&mB) -> int64_t {
        if (GRP) {
            cur.seek(grp, T);
            const ProductJob *J = grp.jobs + cur.j;
            a = J->a;
            mA = &J->tmA;
            mB = &J->tmB;
            return T - cur.beg;
        }
        a = a0;
        mA = &tmA;
        mB = &tmB;
        return T;
    };

    if (warp == 0) {
        if (tc::elect_one()) {
            if (!GRP) {
                tc::prefetch_tmap(&tmA);
                tc::prefetch_tmap(&tmB);
            }
            int it = 0;
            for (int64_t T = t0; T < total && !aborted(bars); T += tstep) {
                ProductArgs a;
                const CUtensorMap *mA, *mB;
                const int64_t t = tile_job(T, a, mA, mB);
                const int64_t per_mod = (int64_t)a.nyt * a.nxt;
                const int mi = (int)(t / per_mod), r = (int)(t % per_mod);
                const int y0 = (r / a.nxt) * (NP * BM) + (int)rank * BM, x0 = (r % a.nxt) * PBX;
                for (int s = 0; s < a.nk; s++, it++) {
                    const int st = it % STAGES;
                    if (it >= STAGES && !tc::mbar_wait(&bars->empty[st], ((it / STAGES) & 1) ^ 1)) {
                        set_abort(bars, err);
                        break;
                    }
                    uint8_t *sa = base + st * STAGE;
                    if (PAIR) {
                        const uint32_t full0 = tc::mapa(tc::smem_u32(&bars->full[st]), 0);
                        if (rank == 0) tc::mbar_arrive_expect_tx(&bars->full[st], 2 * STAGE);
                        tc::tma_load_2d_pair(sa, mA, full0, s * BK, (2 * mi) * a.m + y0);
                        tc::tma_load_2d_pair(sa + A_BYTES, mA, full0, s * BK, (2 * mi + 1) * a.m + y0);
                        tc::tma_load_2d_pair(sa + 2 * A_BYTES, mB, full0, s * BK, (2 * mi + (int)rank) * a.n + x0);
                    } else {
                        tc::mbar_arrive_expect_tx(&bars->full[st], STAGE);
                        tc::tma_load_2d(sa, mA, &bars->full[st], s * BK, (2 * mi) * a.m + y0);
                        tc::tma_load_2d(sa + A_BYTES, mA, &bars->full[st], s * BK, (2 * mi + 1) * a.m + y0);
                        tc::tma_load_2d(sa + 2 * A_BYTES, mB, &bars->full[st], s * BK, (2 * mi) * a.n + x0);
                        tc::tma_load_2d(sa + 2 * A_BYTES + B_BYTES, mB, &bars->full[st], s * BK,
                                        (2 * mi + 1) * a.n + x0);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && tc::elect_one()) {
            const uint32_t idesc = tc::idesc_bf16_f32(NP * BM, 2 * PBX, 0, 0);
            int it = 0, lt = 0;
            bool ok = true;
            for (int64_t T = t0; T < total && ok; T += tstep, lt++) {
                ProductArgs a;
                const CUtensorMap *mA, *mB;
                tile_job(T, a, mA, mB);
                (void)mA, (void)mB;
                const int b = lt & 1;
                if (lt >= 2 && !tc::mbar_wait(&bars->tempty[b], ((lt >> 1) & 1) ^ 1)) { set_abort(bars, err); break; }
                tc::fence_after_sync();
                const uint32_t d = tmem + 256u * b;
                for (int s = 0; s < a.nk; s++, it++) {
                    const int st = it % STAGES;
                    if (!tc::mbar_wait(&bars->full[st], (it / STAGES) & 1)) { set_abort(bars, err); ok = false; break; }
                    tc::fence_after_sync();
                    const uint32_t sa = tc::smem_u32(base + st * STAGE);
                    // three descriptors per K step; the K slices advance them by 32 bytes
                    const uint64_t a1d = tc::sdesc_kmajor(sa), a0d = tc::sdesc_kmajor(sa + A_BYTES),
                                   bd = tc::sdesc_kmajor(sa + 2 * A_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / UK; kk++) {
                        const uint64_t bdesc = tc::sdesc_advance(bd, kk * 32);
                        const uint64_t a1 = tc::sdesc_advance(a1d, kk * 32), a0 = tc::sdesc_advance(a0d, kk * 32);
                        const uint32_t acc = s != 0 || kk != 0;
                        if (PAIR) {
                            tc::mma_bf16_pair(d, a1, bdesc, idesc, acc);
                            tc::mma_bf16_pair(d + 2 * PBX, a0, bdesc, idesc, acc);
                        } else {
                            tc::mma_bf16(d, a1, bdesc, idesc, acc);
                            tc::mma_bf16(d + 2 * PBX, a0, bdesc, idesc, acc);
                        }
                    }
                    if (PAIR) tc::mma_commit_pair(&bars->empty[st], 0x3);
                    else tc::mma_commit(&bars->empty[st]);
                }
                if (ok) {
                    if (PAIR) tc::mma_commit_pair(&bars->tfull[b], 0x3);
                    else tc::mma_commit(&bars->tfull[b]);
                }
            }
        }
    } else {
        // warp (2..9) -> lane quadrant warp % 4, output columns 32 * ((warp - 2) / 4) + [0, 32).
        // All four accumulators' 32 columns are read first, so the buffer goes back to the
        // MMA before the arithmetic.
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t tempty0 = PAIR ? tc::mapa(tc::smem_u32(&bars->tempty[0]), 0) : 0;
        // this warp's staging: 32 rows of 32 entries of one plane, 16-byte chunks at positions
        // that keep both the row writes and the reads of whole rows conflict-free
        uint4 *stg = reinterpret_cast<uint4 *>(stage_out + (warp - 2) * PROD_STG_BYTES);
        const int swz = (lane >> 1) & 3;
        int lt = 0;
        for (int64_t T = t0; T < total; T += tstep, lt++) {
            ProductArgs a;
            const CUtensorMap *mA, *mB;
            const int64_t t = tile_job(T, a, mA, mB);
            (void)mA, (void)mB;
            const int64_t per_mod = (int64_t)a.nyt * a.nxt;
            const int b = lt & 1;
            const int mi = (int)(t / per_mod), r = (int)(t % per_mod);
            const int y0 = (r / a.nxt) * (NP * BM) + (int)rank * BM + quad * 32;  // the warp's first row
            const int xh = (r % a.nxt) * PBX + half * 32;  // this warp's 32 output columns
            if (!tc::mbar_wait(&bars->tfull[b], (lt >> 1) & 1)) { set_abort(bars, err); break; }
            tc::fence_after_sync();
            uint32_t D11[32], D10[32], D01[32], D00[32];
            const uint32_t col = 256u * b + half * 32;
            tc::tmem_ld32(lb + col, D11);
            tc::tmem_ld32(lb + col + PBX, D10);
            tc::tmem_ld32(lb + col + 2 * PBX, D01);
            tc::tmem_ld32(lb + col + 3 * PBX, D00);
            tc::tmem_ld_wait();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) tc::mbar_arrive_cluster(tempty0 + 8u * b);
                else tc::mbar_arrive(&bars->tempty[b]);
            }
            // p and fl(1/p) of modulus mi from the constant list (a broadcast: the warp's
            // lanes share mi); the same values as the moduli table's
            const float4 cmp = c_modpair[mi >> 1];
            const float pf = (mi & 1) ? cmp.y : cmp.x, ipf = (mi & 1) ? cmp.w : cmp.z;
            const f32x2 np = pk2(-pf, -pf), ip = pk2(ipf, ipf), np8 = pk2(-pf / 256.f, -pf / 256.f), ip8 = pk2(256.f * ipf, 256.f * ipf);
            // (256 x mod p) / 256, |256 x / p| < 2^17: the quotient is off by less than 0.01, and the
            // difference is a multiple of 1/256 below 2^16 / 256, so the FMA gives it exactly
            auto red8 = [&](f32x2 x) {
                const f32x2 q = add2(fma2(x, ip8, pk2(RND_MAGIC, RND_MAGIC)), pk2(-RND_MAGIC, -RND_MAGIC));
                return fma2(q, np8, x);
            };
            auto pair = [](const uint32_t(&v)[32], int j) { return pk2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])); };
            uint32_t plo[16];
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
                uint32_t phi[4];
#pragma unroll
                for (int j = c; j < c + 8; j += 2) {
                    // y = 256 (256 d11 + d10 + d01) + d00, each 256 x taken mod p.  |d10 + d01| <=
                    // 2^15 k, so with 256 d11 mod p added it stays below 2^24 up to k = 448
                    f32x2 mid = add2(pair(D10, j), pair(D01, j));
                    if (a.nk > 7) mid = red2(mid, np, ip);
                    const f32x2 w = red8(fma2(red8(pair(D11, j)), pk2(256.f, 256.f), mid));
                    f32x2 h2, l2;
                    bal_split2(red2(fma2(w, pk2(256.f, 256.f), pair(D00, j)), np, ip), h2, l2);
                    float h0, h1, l0, l1;
                    upk2(h2, h0, h1);
                    upk2(l2, l0, l1);
                    phi[(j - c) / 2] = __byte_perm(__float_as_uint(h0), __float_as_uint(h1), 0x7632);
                    plo[j / 2] = __byte_perm(__float_as_uint(l0), __float_as_uint(l1), 0x7632);
                }
                stg[lane * 4 + ((c >> 3) ^ swz)] = make_uint4(phi[0], phi[1], phi[2], phi[3]);
            }
            __syncwarp();
            store_plane(a, stg, 2 * mi, y0, xh);
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 4; c++)
                stg[lane * 4 + (c ^ swz)] = make_uint4(plo[4 * c], plo[4 * c + 1], plo[4 * c + 2], plo[4 * c + 3]);
            __syncwarp();
            store_plane(a, stg, 2 * mi + 1, y0, xh);
            __syncwarp();
        }
    }
    tc::grid_dep_launch();
    if (PAIR) {
        tc::fence_before_sync();
        __syncthreads();
        tc::cluster_sync_all();  // no CTA leaves while its peer may still signal it or write its TMEM
        if (warp == 1) {
            tc::fence_after_sync();
            tc::tmem_dealloc_pair(tmem, 512);
        }
    } else {
        cta_teardown(bars, 512);
    }
}

// ======================================================================================
// 4. reconstruction GEMM (persistent over tiles of 128 entries, or 256 entries
//    for a CTA pair; N tiles of 256 table rows; TMEM double-buffered across N
//    tiles; 16 epilogue warps per CTA, four per entry splitting the columns.  Base-128 table
//    digits keep one FP32 accumulation over all 2P rows exact, 2P * 128 * 64 < 2^24;
//    base-256 digits do wherever the table's column sums say so.)
//    Y arrives blocked, [E/64][2Pp][64], so each 64-entry x 64-row A box is one
//    contiguous 8 KB run.
//    PAIR: a cluster of two CTAs on two SMs runs one M = 256, N = 256
//    tcgen05.mma.cta_group::2 per K slice.  Each CTA stages its own 128 entries
//    and its own 128 of the 256 table rows, so per SM the K step moves 32 KB
//    through TMA and the MMA reads 8 KB of shared memory per 2^20 FLOP, against
//    48 KB and 12 KB for one CTA with N = 256: shared-memory bandwidth, which
//    bounds the single-SM tile, drops by a third.
// ======================================================================================
struct ReconArgs {
    int64_t mt0;     // first entry tile of this launch (tiles mt0 .. nmt-1)
    int64_t E;       // entries of Y: rows of C x padded row length
    int32_t ncols;   // padded row length of Y's entries (entry e -> row e / ncols, col e % ncols)
    int32_t ccols;   // columns of C: entries with col >= ccols are padding and not stored
    int32_t nk;      // K steps over 2Pp
    int32_t NT;      // N tiles of 256 table rows
    int32_t nlast;   // columns of the last one (a multiple of 32)
    int32_t Dout;    // output digit positions (base 2^DB)
    int32_t kpad;    // 2Pp: rows of one 64-entry block of Y
    int64_t nmt;     // entry tiles (128 entries, or 256 for a pair)
    const uint32_t *vtab;  // Mod's value per 32-digit chunk, 8 words: DB = 7: sum_u Mod_(32n+u) 128^u as 7
                           // two's-complement words + sign word; DB = 8: signed base-2^32 digits 8n .. 8n + 7
    uint32_t *climbs;
    int32_t *csizes;
    int64_t cld, crs;
    int32_t cnlimbs;
};
// One product of a grouped reconstruction launch (its tiles start at entry tile 0).
struct ReconJob {
    CUtensorMap tmY, tmT;
    ReconArgs a;
};
// Hand-offs between the four epilogue warps ("parts") of a TMEM lane quadrant, per entry.
// One token per quadrant goes round the parts, part 0 -> 1 -> 2 -> 3 -> 0 of the next N
// tile (also on to the next entry tile): the carry, the negation ripple, the highest nonzero
// limb and the dropped-limb flags so far.  A part writes the next part's slot only while
// it holds the token, so a slot or a barrier is never a round ahead of its reader.  Part 0's
// fixed-point results of entry tile i sit in slot and barrier i & 1: those of tile i + 2 are
// written after the token of tile i's last part came back, and every part reads its q before
// it passes the token on.
struct ReconXfer {
    uint64_t tokbar[4][4], qready[2][4];  // [part][quadrant], [tile parity][quadrant]
    int4 tok[4][128];                     // (carry, ripple, top, drop) for part p
    int2 q[2][128];                       // (q, sign and doubt bits)
};

// a * b + c with 32-bit factors (one wide multiply-add)
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

// Y's map is 3-D, [Ep/64 blocks][2P rows][64 entries]: the rows 2P .. 2Pp-1 of a
// block's last K step lie outside it and read as zeros.  GRP: a grouped launch;
// Mod's chunk values are then read from global memory (each product has its own),
// (the epilogue's token order holds for any sequence of N-tile counts).
// DB: bits of a table digit (build_tables chooses): 32 columns are DB limbs.
template <int STAGES, bool PAIR, bool GRP, int DB>
__global__ void __launch_bounds__(REC_THREADS, 1)
    k_crt_recon(const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmT, ReconArgs a0,
                Group<ReconJob> grp, uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = align1024(smem_raw);
    constexpr int NP = PAIR ? 2 : 1;
    constexpr int RBN = 256;                      // accumulator columns (table rows) per N tile
    constexpr int TROWS = RBN / NP;               // table rows this CTA stages per N tile
    constexpr uint32_t BOX = 64 * 128;            // one 64-entry x 64-row A box
    constexpr uint32_t A_BYTES = BM * 128, B_BYTES = TROWS * 128, STAGE = A_BYTES + B_BYTES;
    Barriers *bars = reinterpret_cast<Barriers *>(base + STAGES * STAGE);
    uint32_t *svtab = reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(bars) + SMEM_BARS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? tc::cluster_rank() : 0;
    const int64_t t0 = PAIR ? (blockIdx.x >> 1) : blockIdx.x, tstep = PAIR ? (gridDim.x >> 1) : gridDim.x;
    const int vwords = GRP ? 0 : (a0.Dout + 31) / 32 * 8;
    for (int i = threadIdx.x; i < vwords; i += blockDim.x) svtab[i] = a0.vtab[i];
    ReconXfer *xf = reinterpret_cast<ReconXfer *>(svtab + vwords);
    // entry tiles [tbeg, total) in global numbering; tile_job maps one to its
    // product's arguments and maps and to the entry tile within that product
    const int64_t tbeg = GRP ? 0 : a0.mt0, total = GRP ? grp.tile0[grp.njobs] : a0.nmt;
    GroupCursor cur;
    auto tile_job = [&](int64_t T, ReconArgs &a, const CUtensorMap *&mY, const CUtensorMap *&mT) -> int64_t {
        if (GRP) {
            cur.seek(grp, T);
            const ReconJob *J = grp.jobs + cur.j;
            a = J->a;
            mY = &J->tmY;
            mT = &J->tmT;
            return T - cur.beg;
        }
        a = a0;
        mY = &tmY;
        mT = &tmT;
        return T;
    };
    if (threadIdx.x == 0)
        for (int qd = 0; qd < 4; qd++) {
            for (int pt = 0; pt < 4; pt++) tc::mbar_init(&xf->tokbar[pt][qd], 1);
            for (int i = 0; i < 2; i++) tc::mbar_init(&xf->qready[i][qd], 1);
        }
    if (PAIR) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < STAGES; s++) {
                tc::mbar_init(&bars->full[s], 1);
                tc::mbar_init(&bars->empty[s], 1);
            }
            for (int b = 0; b < 2; b++) {
                tc::mbar_init(&bars->tfull[b], 1);
                tc::mbar_init(&bars->tempty[b], 2 * REC_EPI_WARPS);  // the even CTA's: every epilogue warp of both CTAs
            }
            bars->abort_flag = 0;
            tc::fence_mbar_init();
        }
        if (warp == 1) {
            tc::tmem_alloc_pair(&bars->tmem_base, 512);
            tc::tmem_relinquish_pair();
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
        tc::fence_after_sync();
    } else {
        cta_setup(bars, STAGES, 512, 1, REC_EPI_WARPS);
    }
    tc::grid_dep_wait();  // the planes this launch reads are complete
    const uint32_t tmem = bars->tmem_base;

    if (warp == 0) {
        if (tc::elect_one()) {
            if (!GRP) {
                tc::prefetch_tmap(&tmY);
                tc::prefetch_tmap(&tmT);
            }
            int it = 0;
            for (int64_t T = tbeg + t0; T < total && !aborted(bars); T += tstep) {
                ReconArgs a;
                const CUtensorMap *mY, *mT;
                const int64_t t = tile_job(T, a, mY, mT);
                const int blk0 = (int)(t * (2 * NP) + 2 * rank);  // this CTA's two 64-entry blocks
                for (int j = 0; j < a.NT && !aborted(bars); j++) {
                    for (int s = 0; s < a.nk; s++, it++) {
                        const int st = it % STAGES;
                        if (it >= STAGES && !tc::mbar_wait(&bars->empty[st], ((it / STAGES) & 1) ^ 1)) {
                            set_abort(bars, err);
                            break;
                        }
                        uint8_t *sa = base + st * STAGE;
                        // A (MN-major): two 64-entry blocks x 64 K-rows; blocks past the end of
                        // Y read as zeros and still count their full box bytes
                        if (PAIR) {
                            const uint32_t full0 = tc::mapa(tc::smem_u32(&bars->full[st]), 0);
                            if (rank == 0) tc::mbar_arrive_expect_tx(&bars->full[st], 2 * STAGE);
                            tc::tma_load_3d_pair(sa, mY, full0, 0, s * BK, blk0);
                            tc::tma_load_3d_pair(sa + BOX, mY, full0, 0, s * BK, blk0 + 1);
                            // the even CTA's rows are the tile's first half, also of a narrow last tile
                            tc::tma_load_2d_pair(sa + A_BYTES, mT, full0, s * BK,
                                                 j * RBN + (int)rank * (j + 1 < a.NT ? TROWS : a.nlast / 2));
                        } else {
                            tc::mbar_arrive_expect_tx(&bars->full[st], STAGE);
                            tc::tma_load_3d(sa, mY, &bars->full[st], 0, s * BK, blk0);
                            tc::tma_load_3d(sa + BOX, mY, &bars->full[st], 0, s * BK, blk0 + 1);
                            tc::tma_load_2d(sa + A_BYTES, mT, &bars->full[st], s * BK, j * RBN);
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && tc::elect_one()) {
            int it = 0, lt = 0;
            bool ok = true;
            for (int64_t T = tbeg + t0; T < total && ok; T += tstep) {
                ReconArgs a;
                const CUtensorMap *mY, *mT;
                tile_job(T, a, mY, mT);
                (void)mY, (void)mT;
                for (int j = 0; j < a.NT && ok; j++, lt++) {
                    // the last N tile's MMAs have only the columns it needs
                    const uint32_t idesc = tc::idesc_bf16_f32(NP * BM, j + 1 < a.NT ? RBN : a.nlast, 1, 0);
                    const int b = lt & 1;
                    if (lt >= 2 && !tc::mbar_wait(&bars->tempty[b], ((lt >> 1) & 1) ^ 1)) {
                        set_abort(bars, err);
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t d = tmem + 256u * b;
                    for (int s = 0; s < a.nk; s++, it++) {
                        const int st = it % STAGES;
                        if (!tc::mbar_wait(&bars->full[st], (it / STAGES) & 1)) { set_abort(bars, err); ok = false; break; }
                        tc::fence_after_sync();
                        const uint32_t sa = tc::smem_u32(base + st * STAGE);
                        const uint64_t ad = tc::sdesc_mnmajor(sa, BOX), bd = tc::sdesc_kmajor(sa + A_BYTES);
#pragma unroll
                        for (int kk = 0; kk < BK / UK; kk++) {
                            const uint64_t adesc = tc::sdesc_advance(ad, kk * 2048), bdesc = tc::sdesc_advance(bd, kk * 32);
                            const uint32_t acc = s != 0 || kk != 0;
                            if (PAIR) tc::mma_bf16_pair(d, adesc, bdesc, idesc, acc);
                            else tc::mma_bf16(d, adesc, bdesc, idesc, acc);
                        }
                        if (PAIR) tc::mma_commit_pair(&bars->empty[st], 0x3);
                        else tc::mma_commit(&bars->empty[st]);
                    }
                    if (ok) {
                        if (PAIR) tc::mma_commit_pair(&bars->tfull[b], 0x3);
                        else tc::mma_commit(&bars->tfull[b]);
                    }
                }
            }
        }
    } else {
        // 16 epilogue warps.  quad = warp % 4 owns TMEM lanes (entries) quad * 32 .. + 31 and
        // part = (warp - 2) / 4 owns accumulator columns part * 64 .. + 63 of every N tile.  An
        // entry's digits run through its carry chain part by part, N tile by N tile.  Each part
        // turns its two 32-column chunks into limbs starting from carry 0, then takes the
        // token (the carry and negation ripple so far), adds them, stores, and passes it on.
        // Waits are bounded.
        // What bounds it: dependent integer chains, not the issue slots (31 % used by two warps per
        // lane quadrant) and not HBM, hence four warps per quadrant:
        // 1024 x 1024 entries by 259 moduli 709 -> 518 us, 300 x 300 by 259 85 -> 65 us.  (Base-256 table
        // digits and one wide multiply-add per digit took the same launches from 921 to 738 us and
        // the 512 x 512 one by 516 moduli from 439 to 376 us.)
        const int quad = warp & 3, part = (warp - 2) >> 2, idx = quad * 32 + lane;
        const uint32_t lb = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * 64);
        const uint32_t tempty0 = PAIR ? tc::mapa(tc::smem_u32(&bars->tempty[0]), 0) : 0;
        int lt = 0, ntok = 0, et = 0;  // N tiles, tokens taken, entry tiles seen
        bool first = true, ok = true;
        for (int64_t T = tbeg + t0; T < total && ok; T += tstep, et++) {
            ReconArgs a;
            const CUtensorMap *mY, *mT;
            const int64_t t = tile_job(T, a, mY, mT);
            (void)mY, (void)mT;
            const int64_t e = t * (NP * BM) + rank * BM + quad * 32 + lane;
            const int64_t er = e / a.ncols, ec = e - er * a.ncols;
            const bool live = e < a.E && ec < a.ccols;
            const int64_t coff = live ? er * a.crs + ec : 0;
            // C = sum_u (acc_u - q Mod_u) 2^(DB u); the limbs written are |C| (negated on the
            // fly when the fixed-point sum says C < 0)
            int q = 0, sgn = 1, amb = 0, top = 0, c = 0;
            uint32_t nin = 0, drop = 2;  // dropped limbs: bit 0 any nonzero, bit 1 all ones
            for (int j = 0; j < a.NT; j++, lt++) {
                const int b = lt & 1;
                if (!tc::mbar_wait(&bars->tfull[b], (lt >> 1) & 1)) { set_abort(bars, err); ok = false; break; }
                tc::fence_after_sync();
                uint32_t g[32];
                tc::tmem_ld32(lb + (uint32_t)(256 * b), g);
                tc::tmem_ld_wait(g);
                if (j == 0) {
                    const int qb = et & 1;
                    if (part == 0) {
                        // fixed-point sum S = sum y_i 2^FIXB / p_i from the first SUSED columns
                        // (base 128): S = (q + C / Mod) 2^FIXB + err, |err| <= 128 P < 2^17, and
                        // |C / Mod| < 2^-18, so q = round(S / 2^FIXB) and the sign of
                        // frac = S - q 2^FIXB is the sign of C unless |C| < Mod 2^(20 - FIXB)
                        __int128 S = 0;
#pragma unroll
                        for (int u = SUSED - 1; u >= 0; u--) S = S * 128 + tc::acc_int(g[u]);
                        const __int128 halfw = (__int128)1 << (FIXB - 1);
                        const __int128 qq = (S + halfw) >> FIXB;
                        const __int128 frac = S - (qq << FIXB);
                        const __int128 tol = (__int128)1 << 20;
                        q = (int32_t)qq;
                        sgn = frac < -tol ? -1 : 1;
                        amb = frac <= tol && frac >= -tol;
                        xf->q[qb][idx] = make_int2(q, (sgn < 0 ? 1 : 0) | (amb ? 2 : 0));
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&xf->qready[qb][quad]);
                    } else {
                        if (!tc::mbar_wait(&xf->qready[qb][quad], (et >> 1) & 1)) { set_abort(bars, err); ok = false; break; }
                        const int2 v = xf->q[qb][idx];
                        q = v.x;
                        sgn = v.y & 1 ? -1 : 1;
                        amb = v.y >> 1;
                    }
                }
                // this part's limbs from carry 0: chunks ch, ch + 1 of 32 digits (DB limbs each, on
                // limb boundaries; the fixed-point columns are chunk -1)
                uint32_t L[2 * DB];
                c = 0;  // |carry| < 2^26
                const int ch = 8 * j + 2 * part - SROWS / 32;
                const int nq = -q;
                bool have[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (k == 1) {
                        tc::tmem_ld32(lb + (uint32_t)(256 * b + 32), g);
                        tc::tmem_ld_wait(g);
                        tc::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) {
                            if (PAIR) tc::mbar_arrive_cluster(tempty0 + 8u * b);
                            else tc::mbar_arrive(&bars->tempty[b]);
                        }
                    }
                    have[k] = live && ch + k >= 0 && (ch + k) * 32 < a.Dout;
                    if (!have[k]) continue;
                    const uint32_t *W = (GRP ? a.vtab : svtab) + (ch + k) * 8;
                    if constexpr (DB == 8) {
                        // four columns per limb: a0 + 2^8 a1 + 2^16 a2 + 2^24 a3 - q W_l + carry, |.| < 2^49
#pragma unroll
                        for (int l = 0; l < 8; l++) {
                            long long t = mad_wide(nq, (int)W[l], (long long)tc::acc_int(g[4 * l]));
                            t = mad_wide(tc::acc_int(g[4 * l + 1]), 1 << 8, t);
                            t = mad_wide(tc::acc_int(g[4 * l + 2]), 1 << 16, t);
                            t = mad_wide(tc::acc_int(g[4 * l + 3]), 1 << 24, t) + c;
                            L[8 * k + l] = (uint32_t)t;
                            c = (int)(t >> 32);
                        }
                    } else {
                        long long A[7];
                        A[0] = c;
#pragma unroll
                        for (int l = 1; l < 7; l++) A[l] = 0;
#pragma unroll
                        for (int u = 0; u < 32; u++)
                            A[(7 * u) >> 5] += (long long)tc::acc_int(g[u]) * (1LL << ((7 * u) & 31));
#pragma unroll
                        for (int l = 0; l < 7; l++) A[l] += (long long)nq * (long long)W[l];
#pragma unroll
                        for (int l = 0; l < 7; l++) {
                            if (l < 6) A[l + 1] += A[l] >> 32;
                            L[7 * k + l] = (uint32_t)A[l];
                        }
                        // the chunk's Mod value is sum W_l 2^(32 l) - s 2^224 (s = sign word)
                        c = (int)(A[6] >> 32) + (W[7] ? q : 0);
                    }
                }
                // the token: nothing to take at an entry's first columns but the turn
                int cin = 0;
                nin = sgn < 0;  // a non-negative value passes 0 on
                if (part > 0 || !first) {
                    if (!tc::mbar_wait(&xf->tokbar[part][quad], ntok & 1)) { set_abort(bars, err); ok = false; break; }
                    ntok++;
                    if (part > 0 || j > 0) {
                        const int4 v = xf->tok[part][idx];
                        cin = v.x;
                        nin = (uint32_t)v.y;
                        top = v.z;
                        drop = (uint32_t)v.w;
                    }
                }
                first = false;
                // add the carry in, negate when C < 0 (~limb + 1, the +1 rippling up), store
                const uint32_t mask = sgn < 0 ? 0xFFFFFFFFu : 0u;
                const int li0 = ch * DB, room = a.cnlimbs - li0;  // limbs of this part that C has planes for
                uint32_t *cp = a.climbs + (int64_t)li0 * a.cld + coff;
#pragma unroll
                for (int l = 0; l < 2 * DB; l++, cp += a.cld) {
                    if (!have[l / DB]) continue;
                    const uint32_t sum = L[l] + (uint32_t)cin;
                    cin = (cin >> 31) + (sum < L[l] ? 1 : 0);
                    const uint32_t limb = (sum ^ mask) + nin;
                    nin = limb == 0u ? nin : 0u;
                    if (l < room) {
                        *cp = limb;
                        if (limb) top = li0 + l + 1;
                    } else {
                        drop = (drop | (limb != 0u)) & (limb == 0xFFFFFFFFu ? 3u : 1u);
                    }
                }
                c += cin;
                // pass the token on (after the CTA's very last column nobody takes it)
                const int next = (part + 1) & 3;
                xf->tok[next][idx] = make_int4(c, (int)nin, top, (int)drop);
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&xf->tokbar[next][quad]);
            }
            if (!ok) break;
            if (part == 3 && live) {
                const bool drop_nz = drop & 1u, drop_ones = drop & 2u;
                const int nl = (a.Dout + 31) / 32 * DB;  // limbs produced
                const int written = nl < a.cnlimbs ? nl : a.cnlimbs;
                int neg = sgn < 0;
                // bits above the produced limbs of the written value: C's own, or -C's
                const long long carry = neg ? -(long long)c - 1 + (long long)nin : (long long)c;
                if (carry < 0) {
                    // only reachable on the ambiguous path: two's complement -> magnitude
                    if (!amb || carry != -1 || (nl > a.cnlimbs && !(drop_ones && top != 0)))
                        atomicOr(err, DEVERR_CAPACITY);
                    uint32_t cc = 1;
                    top = 0;
                    for (int l0 = 0; l0 < written; l0 += 8) {
                        uint32_t w[8];
#pragma unroll
                        for (int u = 0; u < 8; u++)
                            w[u] = l0 + u < written ? a.climbs[(int64_t)(l0 + u) * a.cld + coff] : 0u;
#pragma unroll
                        for (int u = 0; u < 8; u++) {
                            if (l0 + u >= written) break;
                            const uint64_t sum = (uint64_t)(~w[u]) + cc;
                            const uint32_t r = (uint32_t)sum;
                            cc = (uint32_t)(sum >> 32);
                            a.climbs[(int64_t)(l0 + u) * a.cld + coff] = r;
                            if (r) top = l0 + u + 1;
                        }
                    }
                    neg = 1;
                } else if (carry != 0 || drop_nz) {
                    atomicOr(err, DEVERR_CAPACITY);
                }
                for (int li = written; li < a.cnlimbs; li++) a.climbs[(int64_t)li * a.cld + coff] = 0u;
                a.csizes[coff] = top == 0 ? 0 : (neg ? -top : top);
            }
        }
    }
    tc::grid_dep_launch();
    if (PAIR) {
        tc::fence_before_sync();
        __syncthreads();
        tc::cluster_sync_all();  // no CTA leaves while its peer may still signal it or write its TMEM
        if (warp == 1) {
            tc::fence_after_sync();
            tc::tmem_dealloc_pair(tmem, 512);
        }
    } else {
        cta_teardown(bars, 512);
    }
}

// ======================================================================================
// tcgen05 GEMM self-test: D[M x N] (int32) = A * B^T with A K-major [M x K] or
// MN-major [K x M], B K-major [N x K]; used by tests to pin the descriptor
// layouts independently of the CRT arithmetic.
// ======================================================================================
struct TestArgs {
    int32_t M, N, nk, a_mn;
    int32_t *D;
    // failure-path test knobs: the producer leaves K step `skip_step` unloaded and
    // its stage barrier unarmed (-1: none), and every wait gives up after
    // `wait_limit` SM clocks
    int32_t skip_step;
    long long wait_limit;
};

template <int STAGES>
__global__ void __launch_bounds__(CTA_THREADS, 1)
    k_gemm_test(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, TestArgs a,
                uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = align1024(smem_raw);
    constexpr uint32_t A_BYTES = BM * 128, B_BYTES = BM * 128, STAGE = A_BYTES + B_BYTES;
    Barriers *bars = reinterpret_cast<Barriers *>(base + STAGES * STAGE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BM;
    cta_setup(bars, STAGES, 128, 1, 1);
    const uint32_t tmem = bars->tmem_base;
    const long long lim = a.wait_limit;
    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;  // K steps whose loads were issued: steps [0, issued) except skip_step
            for (int s = 0; s < a.nk; s++) {
                const int st = s % STAGES;
                if (s >= STAGES && !tc::mbar_wait(&bars->empty[st], ((s / STAGES) & 1) ^ 1, lim)) {
                    set_abort(bars, err);
                    break;
                }
                issued = s + 1;
                if (s == a.skip_step) continue;  // nothing arms this stage: its consumer's wait runs out
                uint8_t *sa = base + st * STAGE;
                tc::mbar_arrive_expect_tx(&bars->full[st], STAGE);
                if (a.a_mn) {
                    tc::tma_load_2d(sa, &tmA, &bars->full[st], m0, s * BK);
                    tc::tma_load_2d(sa + A_BYTES / 2, &tmA, &bars->full[st], m0 + 64, s * BK);
                } else {
                    tc::tma_load_2d(sa, &tmA, &bars->full[st], s * BK, m0);
                }
                tc::tma_load_2d(sa + A_BYTES, &tmB, &bars->full[st], s * BK, n0);
            }
            if (aborted(bars)) {
                // before the CTA's shared memory goes away: wait (bounded) until the
                // copies of the last stages issued have landed
                for (int s = issued - 1; s >= 0 && s >= issued - STAGES; s--)
                    if (s != a.skip_step) tc::mbar_wait(&bars->full[s % STAGES], (s / STAGES) & 1, lim);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_bf16_f32(BM, BM, a.a_mn, 0);
            bool ok = true;
            int mma_steps = 0;
            for (int s = 0; s < a.nk; s++) {
                const int st = s % STAGES;
                if (!tc::mbar_wait(&bars->full[st], (s / STAGES) & 1, lim)) { set_abort(bars, err); ok = false; break; }
                mma_steps++;
                tc::fence_after_sync();
                const uint32_t sa = tc::smem_u32(base + st * STAGE), sb = sa + A_BYTES;
#pragma unroll
                for (int kk = 0; kk < BK / UK; kk++) {
                    const uint64_t ad =
                        a.a_mn ? tc::sdesc_mnmajor(sa + kk * 2048, A_BYTES / 2) : tc::sdesc_kmajor(sa + kk * 32);
                    tc::mma_bf16(tmem, ad, tc::sdesc_kmajor(sb + kk * 32), idesc, s != 0 || kk != 0);
                }
                tc::mma_commit(&bars->empty[st]);
            }
            if (ok) tc::mma_commit(&bars->tfull[0]);
            else if (mma_steps > 0) {
                // MMAs already issued still write TMEM: wait (bounded) for them before teardown frees it
                tc::mma_commit(&bars->tfull[1]);
                tc::mbar_wait(&bars->tfull[1], 0, lim);
            }
        }
    } else {
        const int row = epi_row();
        bool ok = tc::mbar_wait(&bars->tfull[0], 0, lim);
        if (!ok) set_abort(bars, err);
        tc::fence_after_sync();
        const uint32_t lb = lane_base(tmem);
        for (int c0 = 0; c0 < BM && ok; c0 += 32) {
            uint32_t v[32];
            tc::tmem_ld32(lb + (uint32_t)c0, v);
            tc::tmem_ld_wait();
            const int m = m0 + row;
            if (m < a.M)
                for (int j = 0; j < 32; j++)
                    if (n0 + c0 + j < a.N) a.D[(int64_t)m * a.N + n0 + c0 + j] = tc::acc_int(v[j]);
        }
    }
    cta_teardown(bars, 128);
}

// ======================================================================================
// CTA-pair GEMM self-test: D[M x N] (int32) = A * B^T, A K-major [M x K], B
// K-major [N x K], one 256 x 256 tile per cluster of two CTAs.  The even CTA
// issues tcgen05.mma.cta_group::2 (M = 256, N = 256): each CTA holds its own 128
// rows of A and its own 128 rows of B at the same shared-memory offsets, and
// its TMEM receives its 128 rows of D.  Both CTAs' TMA loads complete on the
// even CTA's stage barrier; the MMA's commit arrives on both CTAs' barriers.
// ======================================================================================
constexpr uint32_t PAIR_TMEM_COLS = 256;
template <int STAGES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CTA_THREADS, 1)
    k_gemm_test_pair(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, TestArgs a,
                     uint32_t *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = align1024(smem_raw);
    constexpr uint32_t A_BYTES = BM * 128, B_BYTES = BM * 128, STAGE = A_BYTES + B_BYTES;
    Barriers *bars = reinterpret_cast<Barriers *>(base + STAGES * STAGE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();
    const int tile = blockIdx.x >> 1, tiles_x = (a.N + 255) / 256;
    const int ty = tile / tiles_x, tx = tile % tiles_x;
    const int m0 = ty * 256 + (int)rank * BM, n0 = tx * 256 + (int)rank * BM;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            tc::mbar_init(&bars->full[s], 1);
            tc::mbar_init(&bars->empty[s], 1);
        }
        tc::mbar_init(&bars->tfull[0], 1);
        bars->abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) {
        tc::tmem_alloc_pair(&bars->tmem_base, PAIR_TMEM_COLS);
        tc::tmem_relinquish_pair();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync_all();  // both CTAs' barriers exist before any cross-CTA signal
    tc::fence_after_sync();
    const uint32_t tmem = bars->tmem_base;
    if (threadIdx.x == 0 && rank == 1) {
        // the pair's MMA writes D at the even CTA's TMEM address: both must agree
        uint32_t lead;
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(lead) : "r"(tc::mapa(tc::smem_u32(&bars->tmem_base), 0)));
        if (lead != tmem) atomicOr(err, DEVERR_BADARG);
    }

    if (warp == 0) {
        if (lane == 0) {
            for (int s = 0; s < a.nk; s++) {
                const int st = s % STAGES;
                if (s >= STAGES && !tc::mbar_wait(&bars->empty[st], ((s / STAGES) & 1) ^ 1)) {
                    set_abort(bars, err);
                    break;
                }
                uint8_t *sa = base + st * STAGE;
                const uint32_t full_lead = tc::mapa(tc::smem_u32(&bars->full[st]), 0);
                if (rank == 0) tc::mbar_arrive_expect_tx(&bars->full[st], 2 * STAGE);
                tc::tma_load_2d_pair(sa, &tmA, full_lead, s * BK, m0);
                tc::tma_load_2d_pair(sa + A_BYTES, &tmB, full_lead, s * BK, n0);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = tc::idesc_bf16_f32(2 * BM, 2 * BM, 0, 0);
            bool ok = true;
            for (int s = 0; s < a.nk; s++) {
                const int st = s % STAGES;
                if (!tc::mbar_wait(&bars->full[st], (s / STAGES) & 1)) { set_abort(bars, err); ok = false; break; }
                tc::fence_after_sync();
                const uint32_t sa = tc::smem_u32(base + st * STAGE), sb = sa + A_BYTES;
#pragma unroll
                for (int kk = 0; kk < BK / UK; kk++)
                    tc::mma_bf16_pair(tmem, tc::sdesc_kmajor(sa + kk * 32), tc::sdesc_kmajor(sb + kk * 32), idesc,
                                      s != 0 || kk != 0);
                tc::mma_commit_pair(&bars->empty[st], 0x3);
            }
            if (ok) tc::mma_commit_pair(&bars->tfull[0], 0x3);
        }
    } else {
        const int row = (int)rank * BM + epi_row();
        const int m = ty * 256 + row;
        const uint32_t lb = lane_base(tmem);
        if (tc::mbar_wait(&bars->tfull[0], 0)) {
            tc::fence_after_sync();
            for (int c0 = 0; c0 < 256; c0 += 32) {
                uint32_t v[32];
                tc::tmem_ld32(lb + (uint32_t)c0, v);
                tc::tmem_ld_wait();
                if (m < a.M) {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (tx * 256 + c0 + j < a.N) a.D[(int64_t)m * a.N + tx * 256 + c0 + j] = tc::acc_int(v[j]);
                }
            }
        } else {
            set_abort(bars, err);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::cluster_sync_all();  // no CTA leaves while its peer may still signal it or write its TMEM
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc_pair(tmem, PAIR_TMEM_COLS);
    }
}

// ======================================================================================
// host side
// ======================================================================================
typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                     const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode() {
    static PFN_encodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(p);
    });
    return fn;
}

// 2-D bf16 tensor map: inner dimension `inner` (contiguous), `outer` rows with
// a pitch of `pitch_elems`; box = box_inner x box_outer, 128-byte swizzle.
gbmm_status make_map(CUtensorMap *m, const void *ptr, uint64_t inner, uint64_t outer, uint64_t pitch_elems,
                            uint32_t box_inner, uint32_t box_outer) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return set_error(GBMM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (pitch_elems * 2) % 16)
        return set_error(GBMM_ERR_INVALID, "tensor map base or pitch not 16-byte aligned");
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {pitch_elems * 2};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t es[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(GBMM_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return GBMM_OK;
}

// Residue planes [nplanes][rows][pitch] bf16 as a 3-D map for the residue epilogue's
// TMA stores: boxes of 32 entries x 1 row x 32 planes, no swizzle.
static gbmm_status make_map_planes(CUtensorMap *m, const void *ptr, uint64_t cols, uint64_t rows, uint64_t nplanes,
                                   uint64_t pitch_elems, uint64_t plane_elems) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return set_error(GBMM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (pitch_elems * 2) % 16 || (plane_elems * 2) % 16)
        return set_error(GBMM_ERR_INVALID, "tensor map base or pitch not 16-byte aligned");
    cuuint64_t dims[3] = {cols, rows, nplanes};
    cuuint64_t strides[2] = {pitch_elems * 2, plane_elems * 2};
    cuuint32_t box[3] = {32, 1, 32};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(GBMM_ERR_CUDA, "cuTensorMapEncodeTiled (planes) failed (%d)", (int)r);
    return GBMM_OK;
}

// ---- host big integers (tables only) ---------------------------------------------------------
typedef std::vector<uint32_t> big;  // little-endian 32-bit limbs
static void big_mul_small(big &x, uint32_t m) {
    uint64_t c = 0;
    for (auto &l : x) {
        uint64_t t = (uint64_t)l * m + c;
        l = (uint32_t)t;
        c = t >> 32;
    }
    if (c) x.push_back((uint32_t)c);
}
static big big_div_small(const big &x, uint32_t d, uint32_t *rem) {
    big q(x.size());
    uint64_t r = 0;
    for (size_t i = x.size(); i-- > 0;) {
        uint64_t cur = (r << 32) | x[i];
        q[i] = (uint32_t)(cur / d);
        r = cur % d;
    }
    while (!q.empty() && q.back() == 0) q.pop_back();
    if (rem) *rem = (uint32_t)r;
    return q;
}
static uint32_t big_mod_small(const big &x, uint32_t d) {
    uint64_t r = 0;
    for (size_t i = x.size(); i-- > 0;) r = ((r << 32) | x[i]) % d;
    return (uint32_t)r;
}
// balanced base-128 digits (each in [-64, 63]) of a nonnegative integer: digit t
// takes bits [7t, 7t + 7) plus the carry of the digit below.  32 digits span
// exactly 7 words, so each chunk of 32 reads its words once and extracts the
// digits with fixed shifts; the carry is one compare per digit.
static void balanced128(const big &x, int ndig, int *out) {
    const size_t nw = x.size();
    int c = 0;
    for (int t0 = 0; t0 < ndig; t0 += 32) {
        const size_t w0 = (size_t)(t0 / 32) * 7;
        uint64_t w[8];
        for (int k = 0; k < 8; k++) w[k] = w0 + k < nw ? x[w0 + k] : 0;
        const int lim = std::min(32, ndig - t0);
        for (int u = 0; u < 32; u++) {
            if (u >= lim) break;
            const int bit = 7 * u;
            const int b = (int)(((w[bit >> 5] | (w[(bit >> 5) + 1] << 32)) >> (bit & 31)) & 127u);
            const int v = b + c;
            c = v >= 64;
            out[t0 + u] = v - (c << 7);
        }
    }
}
// balanced base-256 digits (each in [-128, 127]): digit t takes byte t plus the carry of
// the digit below
static void balanced256(const big &x, int ndig, int *out) {
    int c = 0;
    for (int t = 0; t < ndig; t++) {
        const int b = (size_t)(t / 4) < x.size() ? (int)((x[t / 4] >> (8 * (t & 3))) & 255u) : 0;
        const int v = b + c;
        c = v >= 128;
        out[t] = v - (c << 8);
    }
}
static std::vector<int> balanced128(const big &x, int ndig) {
    std::vector<int> out(ndig, 0);
    balanced128(x, ndig, out.data());
    return out;
}
static uint32_t inv_mod(uint32_t a, uint32_t p) {
    int64_t t = 0, nt = 1, r = p, nr = a % p;
    while (nr) {
        int64_t q = r / nr;
        int64_t tmp = t - q * nt; t = nt; nt = tmp;
        tmp = r - q * nr; r = nr; nr = tmp;
    }
    if (t < 0) t += p;
    return (uint32_t)t;
}
static const std::vector<uint32_t> &primes_desc() {
    static std::vector<uint32_t> pr;
    static std::once_flag once;
    std::call_once(once, [] {
        std::vector<char> sieve(65536, 1);
        sieve[0] = sieve[1] = 0;
        for (int i = 2; i * i < 65536; i++)
            if (sieve[i])
                for (int j = i * i; j < 65536; j += i) sieve[j] = 0;
        for (int i = 65535; i >= 3; i--)
            if (sieve[i]) pr.push_back((uint32_t)i);
    });
    return pr;
}

static uint16_t bf16_bits(float f) {
    __nv_bfloat16 h = __float2bfloat16_rn(f);
    uint16_t b;
    memcpy(&b, &h, 2);
    return b;
}
// bf16 bits of the integers -256 .. 256 (every table digit lies in this range)
static uint16_t bf16_small(int v) {
    static const std::vector<uint16_t> lut = [] {
        std::vector<uint16_t> l(513);
        for (int i = -256; i <= 256; i++) l[i + 256] = bf16_bits((float)i);
        return l;
    }();
    return lut[v + 256];
}

struct crt_cache;
struct crt_tables {
    crt_cache *cache = nullptr;  // the cache that holds these tables (and the shared residue table)
    int P = 0, Pp = 0;   // moduli, padded 2P/2 (2Pp multiple of 64)
    int Dout = 0, NT = 0;
    int db = 7;          // bits of a digit of the reconstruction table
    __nv_bfloat16 *d_recon = nullptr;  // [NT * RTAB][2Pp]
    uint32_t *d_vtab = nullptr;        // [ceil(Dout / 32)][8]: Mod's digits per 32-digit chunk
    std::map<int, __nv_bfloat16 *> residue;  // 2 * dxp + weighted -> [2P rows][dxp]
    std::vector<ModConst> h_mods;
};

struct crt_cache {
    std::mutex mu;
    std::map<int, crt_tables *> by_p;
    // the unweighted residue table of every modulus (256^j mod p_i for all 1024
    // moduli and every digit position an operand can have): each product's
    // unweighted table is a view of it (its first moduli, its first dxp columns)
    __nv_bfloat16 *d_res_all = nullptr;
    ~crt_cache() {
        cudaFree(d_res_all);
        for (auto &kv : by_p) {
            crt_tables *t = kv.second;
            cudaFree(t->d_recon);
            cudaFree(t->d_vtab);
            for (auto &r : t->residue) cudaFree(r.second);
            delete t;
        }
    }
};

crt_cache *crt_cache_create() { return new crt_cache(); }
void crt_cache_destroy(crt_cache *c) { delete c; }

// number of moduli for a product bound of `bits` bits (plus margin)
static int moduli_for_bits(int64_t bits) {
    const auto &pr = primes_desc();
    double acc = 0;
    int n = 0;
    while (acc < (double)bits && n < (int)pr.size()) acc += std::log2((double)pr[n++]);
    return acc >= (double)bits ? n : -1;
}

// Host side of a table set: moduli constants, the reconstruction table, Mod's
// chunk values and the constant (p, 1/p) list.
struct crt_tables_host {
    int P = 0, Pp = 0, Dout = 0, NT = 0;
    int db = 7;                   // bits of a digit of the reconstruction table
    double bound = 0;             // largest magnitude an accumulator of its digit columns can reach
    std::vector<ModConst> mods;
    std::vector<uint16_t> recon;  // [NT * RTAB][2Pp] bf16 bits
    std::vector<uint32_t> vtab;   // [ceil(Dout / 32)][8]
    std::vector<float> cmod;      // 4 * CMOD_PAIRS
};

// Digits of the reconstruction table: base 128 is exact for every P up to 1023 (2P digits
// of Y of magnitude 128 against digits of at most 64: 2P * 2^13 < 2^24).  Base 256 digits
// reach 128, but a column's true bound is 128 times the sum of its digits' magnitudes,
// half as large on average: below 2^24 up to about 950 moduli (checked on each table as it
// is built).  They take an eighth fewer columns, and four of them are a limb.
static constexpr int RECON256_MAX_P = 940;

static void build_tables_host(int P, crt_tables_host &o, int db = 7) {
    const auto &pr = primes_desc();
    o.P = P;
    o.db = db;
    auto digits = [db](const big &x, int ndig, int *out) {
        if (db == 8) balanced256(x, ndig, out);
        else balanced128(x, ndig, out);
    };
    o.Pp = (2 * P + 63) / 64 * 32;
    big Mod{1};
    for (int i = 0; i < P; i++) big_mul_small(Mod, pr[i]);
    int modbits = (int)(32 * Mod.size());
    o.Dout = (modbits + db - 1) / db + 2;  // output digits
    o.NT = (SROWS + o.Dout + RTAB - 1) / RTAB;  // in units of RTAB rows
    const int rows = o.NT * RTAB, cols = 2 * o.Pp;
    o.recon.assign((size_t)rows * cols, bf16_bits(0.f));
    std::vector<uint16_t> &tab = o.recon;
    o.mods.resize(P);
    // the moduli are independent: contiguous ranges of them on up to 16 host threads
    // (each writes its own table columns)
    // The moduli are independent: blocks of MB on up to 16 host threads.  A block's
    // digits go to a small row-major buffer first and then into the table row by
    // row, 2 MB adjacent columns at a time (writing one column at a time would
    // touch a new cache line with every 2-byte store).
    constexpr int MB = 32;
    std::mutex sum_mu;
    std::vector<int64_t> colsum(o.Dout, 0);  // sum of the digits' magnitudes per column
    auto block = [&](int i0, int i1, std::vector<int8_t> &dig, std::vector<int> &tmp, std::vector<int64_t> &cs) {
        const int nb = i1 - i0;
        for (int q = 0; q < nb; q++) {
            const int i = i0 + q;
            const uint32_t p = pr[i];
            uint32_t rem = 0;
            big Mi = big_div_small(Mod, p, &rem);
            big Mi256 = Mi;
            big_mul_small(Mi256, 256);
            const uint32_t w = inv_mod(big_mod_small(Mi, p), p);
            ModConst mc;
            memset(&mc, 0, sizeof mc);
            mc.p = (int32_t)p;
            mc.inv_p = 1.0f / (float)p;
            mc.mu = (uint32_t)(((uint64_t)1 << 32) / p);
            mc.h16 = (uint32_t)((1u << 16) % p);
            mc.w = w;
            o.mods[i] = mc;
            // column 2i multiplies the high digit (x256), column 2i+1 the low digit
            digits(Mi256, o.Dout, tmp.data());
            for (int r = 0; r < o.Dout; r++) dig[(size_t)r * (2 * MB) + 2 * q] = (int8_t)tmp[r];
            digits(Mi, o.Dout, tmp.data());
            for (int r = 0; r < o.Dout; r++) dig[(size_t)r * (2 * MB) + 2 * q + 1] = (int8_t)tmp[r];
            // fixed-point weights: round(2^(FIXB+8) / p) for the high digit, round(2^FIXB / p) for the low digit
            const unsigned __int128 one = 1;
            const unsigned __int128 gh = ((one << (FIXB + 8)) + p / 2) / p;
            const unsigned __int128 gl = ((one << FIXB) + p / 2) / p;
            big bh, bl;
            for (int w2 = 0; w2 < 4; w2++) {
                bh.push_back((uint32_t)(gh >> (32 * w2)));
                bl.push_back((uint32_t)(gl >> (32 * w2)));
            }
            std::vector<int> sh = balanced128(bh, SUSED), sl = balanced128(bl, SUSED);
            for (int r = 0; r < SUSED; r++) {
                tab[(size_t)r * cols + 2 * i] = bf16_small(sh[r]);
                tab[(size_t)r * cols + 2 * i + 1] = bf16_small(sl[r]);
            }
        }
        for (int r = 0; r < o.Dout; r++) {
            uint16_t *row = &tab[(size_t)(SROWS + r) * cols + 2 * i0];
            const int8_t *src = &dig[(size_t)r * (2 * MB)];
            for (int c = 0; c < 2 * nb; c++) {
                row[c] = bf16_small(src[c]);
                cs[r] += std::abs((int)src[c]);
            }
        }
    };
    const int nblocks = (P + MB - 1) / MB;
    const int nthr = std::max(1, std::min<int>({16, (int)std::thread::hardware_concurrency(), nblocks}));
    auto range = [&](int th) {
        std::vector<int8_t> dig((size_t)o.Dout * 2 * MB);
        std::vector<int> tmp(o.Dout);
        std::vector<int64_t> cs(o.Dout, 0);
        for (int bk = th; bk < nblocks; bk += nthr) block(bk * MB, std::min(P, (bk + 1) * MB), dig, tmp, cs);
        std::lock_guard<std::mutex> lk(sum_mu);
        for (int r = 0; r < o.Dout; r++) colsum[r] += cs[r];
    };
    if (nthr == 1) {
        range(0);
    } else {
        std::vector<std::thread> pool;
        for (int th = 1; th < nthr; th++) pool.emplace_back(range, th);
        range(0);
        for (auto &th : pool) th.join();
    }
    o.bound = 128.0 * (double)*std::max_element(colsum.begin(), colsum.end());
    const int nch = (o.Dout + 31) / 32;
    o.vtab.assign((size_t)nch * 8, 0u);
    // the constant (p, 1/p) list: the same for every table, written with each
    o.cmod.resize(4 * CMOD_PAIRS);
    for (int q = 0; q < CMOD_PAIRS; q++) {
        o.cmod[4 * q] = (float)pr[2 * q];
        o.cmod[4 * q + 1] = (float)pr[2 * q + 1];
        o.cmod[4 * q + 2] = 1.0f / (float)pr[2 * q];
        o.cmod[4 * q + 3] = 1.0f / (float)pr[2 * q + 1];
    }
    if (db == 8) {
        // Mod in signed base-2^32 digits (each in [-2^31, 2^31)); Dout leaves a limb above Mod
        uint64_t c = 0;
        for (int l = 0; l < 8 * nch; l++) {
            const uint64_t v = ((size_t)l < Mod.size() ? (uint64_t)Mod[l] : 0ull) + c;
            o.vtab[l] = (uint32_t)v;
            c = (v + 0x80000000ull) >> 32;
        }
        return;
    }
    // Mod's balanced base-128 digits, summed per 32-digit chunk n into the 224-bit
    // value V_n = sum_u Mod_(32n+u) 128^u, kept as 8 words of a 256-bit two's
    // complement number (|V_n| < 2^223, so word 7 is the sign extension)
    std::vector<int> md = balanced128(Mod, o.Dout);
    for (int n = 0; n < nch; n++) {
        uint32_t *w = &o.vtab[(size_t)n * 8];
        for (int u = 0; u < 32; u++) {
            const int r = 32 * n + u;
            if (r >= o.Dout || md[r] == 0) continue;
            const int bit = 7 * u, k = bit / 32;
            const uint64_t v = (uint64_t)((int64_t)md[r] * ((int64_t)1 << (bit % 32)));  // two's complement
            uint32_t add[8];
            for (int kk = 0; kk < 8; kk++) add[kk] = md[r] < 0 ? 0xFFFFFFFFu : 0u;
            for (int kk = 0; kk < k; kk++) add[kk] = 0u;
            add[k] = (uint32_t)v;
            if (k + 1 < 8) add[k + 1] = (uint32_t)(v >> 32);
            uint64_t c = 0;
            for (int kk = 0; kk < 8; kk++) {
                const uint64_t sum = (uint64_t)w[kk] + add[kk] + c;
                w[kk] = (uint32_t)sum;
                c = sum >> 32;
            }
        }
    }
}

// Whether the columns of the top base-256 digits stay below the bound: the Mod / p share their
// leading digits, the moduli being close together, so these columns alone can pass it (36 of the
// moduli counts up to 940, all from 739 on).  Read off Mod's top 13 to 14 bytes before a table is
// built: building base 256, then base 128 took 9.9 ms at 922 moduli, base 128 alone 7.5.
static bool top_digits_fit(int P) {
    if (2 * P * 128 * 128 < (1 << 24)) return true;
    const auto &pr = primes_desc();
    unsigned __int128 mod = 1;  // Mod without its low bytes
    for (int i = 0; i < P; i++)
        for (mod *= pr[i]; mod >> 112;) mod >>= 8;
    int64_t sum[16] = {};
    for (int i = 0; i < P; i++) {
        unsigned __int128 q = mod / (unsigned)pr[i] >> 32;  // (the low bytes lack what was dropped)
        for (int t = 0, c = 0; t < 12; t++, q >>= 8) {
            const int v = (int)(q & 255u) + c;
            c = v >= 128;
            const int d = std::abs(v - (c << 8));
            sum[t] += d;      // the low digit's factor
            sum[t + 1] += d;  // the high digit's, 256 times it
        }
    }
    return 128 * *std::max_element(sum, sum + 16) < (1 << 24);
}

// The table of P moduli in the larger digits that its columns allow; returns the builds it took.
static int build_tables_fit(int P, crt_tables_host &o) {
    int builds = 0;
    if (P <= RECON256_MAX_P && top_digits_fit(P)) {
        build_tables_host(P, o, 8);
        builds++;
        if (o.bound < 16777216.0) return builds;
        o = crt_tables_host();
    }
    build_tables_host(P, o, 7);
    return builds + 1;
}

static gbmm_status build_tables(crt_tables *t, int P) {
    crt_tables_host o;
    build_tables_fit(P, o);
    t->db = o.db;
    t->P = o.P;
    t->Pp = o.Pp;
    t->Dout = o.Dout;
    t->NT = o.NT;
    t->h_mods = o.mods;
    // every upload has landed before the tables are used (kernels that use them may
    // run on any stream)
    {
        cudaStream_t cs = copy_stream();
        if (!cs) return set_error(GBMM_ERR_CUDA, "no copy stream");
        GBMM_CUDA_TRY(cudaMemcpyToSymbolAsync(c_modpair, o.cmod.data(), o.cmod.size() * sizeof(float), 0,
                                              cudaMemcpyHostToDevice, cs));
        GBMM_CUDA_TRY(cudaStreamSynchronize(cs));
    }
    GBMM_CUDA_TRY(cudaMalloc(&t->d_recon, o.recon.size() * 2));
    GBMM_TRY(upload_now(t->d_recon, o.recon.data(), o.recon.size() * 2));
    GBMM_CUDA_TRY(cudaMalloc(&t->d_vtab, o.vtab.size() * 4));
    GBMM_TRY(upload_now(t->d_vtab, o.vtab.data(), o.vtab.size() * 4));
    return GBMM_OK;
}

// Residue table [2P rows][dxp]: rows 2i / 2i+1 hold the low / high balanced
// byte of 256^j mod p_i (weighted = 0) or of w_i 256^j mod p_i (weighted = 1, the
// CRT weight w_i = (Mod/p_i)^-1 mod p_i folded into the B operand).
// GEMM columns of the residue table for P moduli: two per modulus, padded to whole pairs
static int residue_cols(int P) { return (2 * P + 3) / 4 * 4; }
// Digit positions an operand's rows can have: four groups of 15 K steps of 64.
constexpr int RES_DXMAX = 4 * RES_GROUP_STEPS_B * BK;
// Fills rows [2P padded][dxp] of a residue table (pitch `pitch`) for moduli 0..P-1.
static void residue_rows(const crt_tables *t, int P, int dxp, int pitch, int weighted, uint16_t *tab);
// The table of this product and operand: the unweighted one is a view of the
// cache's shared table (pitch RES_DXMAX), the weighted one is built per (P, dxp).
static gbmm_status residue_table(crt_tables *t, int dxp, int weighted, __nv_bfloat16 **out, int *pitch) {
    if (!weighted) {
        crt_cache *c = t->cache;
        if (!c->d_res_all) {
            const int rows = residue_cols(2 * CMOD_PAIRS);
            std::vector<uint16_t> tab((size_t)rows * RES_DXMAX, 0);
            residue_rows(t, 2 * CMOD_PAIRS, RES_DXMAX, RES_DXMAX, 0, tab.data());
            __nv_bfloat16 *d = nullptr;
            GBMM_CUDA_TRY(cudaMalloc(&d, tab.size() * 2));
            GBMM_TRY(upload_now(d, tab.data(), tab.size() * 2));
            c->d_res_all = d;
        }
        *out = c->d_res_all;
        *pitch = RES_DXMAX;
        return GBMM_OK;
    }
    *pitch = dxp;
    const int key = 2 * dxp + weighted;
    auto it = t->residue.find(key);
    if (it != t->residue.end()) { *out = it->second; return GBMM_OK; }
    std::vector<uint16_t> tab((size_t)residue_cols(t->P) * dxp, 0);
    residue_rows(t, t->P, dxp, dxp, 1, tab.data());
    __nv_bfloat16 *d = nullptr;
    GBMM_CUDA_TRY(cudaMalloc(&d, tab.size() * 2));
    GBMM_TRY(upload_now(d, tab.data(), tab.size() * 2));
    t->residue[key] = d;
    *out = d;
    return GBMM_OK;
}

// Rows (table columns of the GEMM) in groups of four per pair of moduli (i, i + 1):
// [lo_i, lo_i+1, hi_i, hi_i+1]; with P odd the last group's second slot stays zero.
// In the shared table every slot holds its modulus; a product with P odd then
// computes one residue past its moduli in the padding column of its last pair,
// bounded like the others and never stored.
static void residue_rows(const crt_tables *t, int P, int dxp, int pitch, int weighted, uint16_t *tab) {
    const auto &pr = primes_desc();
    auto range = [&](int i0, int i1) {
        for (int i = i0; i < i1; i++) {
            const uint32_t p = pr[i];
            const size_t r_lo = (size_t)4 * (i >> 1) + (i & 1), r_hi = r_lo + 2;
            uint32_t v = weighted ? t->h_mods[i].w : 1u;  // (w) 256^j mod p
            for (int j = 0; j < dxp; j++) {
                int32_t b = v > p / 2 ? (int32_t)v - (int32_t)p : (int32_t)v;
                int32_t d0 = ((b + 128) & 255) - 128;
                int32_t d1 = (b - d0) / 256;
                tab[r_lo * pitch + j] = bf16_small(d0);  // x1
                tab[r_hi * pitch + j] = bf16_small(d1);  // x256
                v = (uint32_t)(((uint64_t)v * 256) % p);
            }
        }
    };
    // the moduli's rows are independent: contiguous ranges on up to 16 host threads
    const int nthr = std::max(1, std::min<int>({16, (int)std::thread::hardware_concurrency(), (P * dxp) >> 16}));
    if (nthr == 1) {
        range(0, P);
    } else {
        std::vector<std::thread> pool;
        for (int th = 1; th < nthr; th++) pool.emplace_back(range, (int)((int64_t)P * th / nthr), (int)((int64_t)P * (th + 1) / nthr));
        range(0, P / nthr);
        for (auto &th : pool) th.join();
    }
}

static gbmm_status get_tables(crt_cache *c, int P, crt_tables **out) {
    std::lock_guard<std::mutex> lk(c->mu);
    auto it = c->by_p.find(P);
    if (it != c->by_p.end()) { *out = it->second; return GBMM_OK; }
    crt_tables *t = new crt_tables();
    t->cache = c;
    gbmm_status st = build_tables(t, P);
    if (st != GBMM_OK) { delete t; return st; }
    c->by_p[P] = t;
    *out = t;
    return GBMM_OK;
}

static constexpr int RES_STAGES = 4, PROD_STAGES = 4, REC_STAGES = 4, TEST_STAGES = 4;
static constexpr int REC_STAGES_PAIR = 6;  // a pair CTA stages 32 KB per K step
static constexpr int RES_STAGES_PAIR = 5;  // a pair CTA stages 32 KB per K step
static constexpr int PROD_STAGES_PAIR = 5;  // a pair CTA stages 40 KB per K step
static constexpr int PROD_PAIR_MIN_NK = 8;  // K steps (of 64) from which the product runs on CTA pairs
static int g_residue_mode = -1;  // residue GEMM form: -1 by the K loop's length, 0 one CTA, 1 CTA pairs
static constexpr int RES_PAIR_MIN_NK = 1 << 30;  // the pair form of the residue GEMM measured slower at every size
static bool residue_pair(int nk) { return g_residue_mode < 0 ? nk >= RES_PAIR_MIN_NK : g_residue_mode == 1; }

int num_sms() {
    static std::atomic<int> n{0};
    int v = n.load(std::memory_order_relaxed);
    if (v <= 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) return 148;
        n.store(v, std::memory_order_relaxed);
    }
    return v;
}
static size_t smem_bytes(int stages, size_t stage_bytes) { return stages * stage_bytes + SMEM_BARS + 1024 + 64; }

static gbmm_status set_smem(const void *fn, size_t bytes) {
    GBMM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return GBMM_OK;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Programmatic dependent launch: every kernel of the four CRT stages is launched
// with programmatic stream serialization, so its CTAs may be scheduled, set up
// their barriers and allocate TMEM while the kernel before it in the stream
// finishes its last tiles.  Each of them calls tc::grid_dep_wait() before its
// first global-memory access and tc::grid_dep_launch() when its work is issued.
// A kernel's dependences on other streams (events) stay full dependences.
static bool g_pdl = true;

static void set_pdl(cudaLaunchAttribute &at) {
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
}

// Launch of one of the four stages' kernels on plain CTAs.
template <typename... KArgs, typename... Args>
static gbmm_status launch_one(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t s,
                              Args &&...args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute attr[1];
    set_pdl(attr[0]);
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl ? 1 : 0;
    GBMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...));
    return GBMM_OK;
}

// Launch of a persistent kernel in clusters of two CTAs (one CTA per SM): the
// grid is as many pairs as can be resident at once (GPCs with an odd number of
// free SMs leave one SM without a partner), capped by the work.
template <typename... KArgs, typename... Args>
static gbmm_status launch_pairs(void (*kern)(KArgs...), int threads, int64_t work_pairs, size_t smem, cudaStream_t s,
                                Args &&...args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)(2 * std::max<int>(1, num_sms() / 2)));
    int resident = 0;
    GBMM_CUDA_TRY(cudaOccupancyMaxActiveClusters(&resident, (const void *)kern, &cfg));
    if (resident < 1) return set_error(GBMM_ERR_UNSUPPORTED, "no CTA pair of this kernel fits on the device");
    cfg.gridDim = dim3((unsigned)(2 * std::min<int64_t>(work_pairs, resident)));
    set_pdl(attr[1]);
    cfg.numAttrs = g_pdl ? 2 : 1;
    GBMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...));
    return GBMM_OK;
}

// ---- launch plans of the four stages (one product, or one record of a grouped launch) ----------

// digit-row length of an operand's entries: 4 digits per limb, padded to 64
static int operand_dxp(const gbmm_mat &X) { return (4 * std::max(X.nlimbs, 1) + 63) / 64 * 64; }
static size_t digits_bytes(const gbmm_mat &X) { return (size_t)X.rows * X.cols * operand_dxp(X) * 2 + 1024; }

// Digits + residues of one operand into planes [2P][rowsR][kp] (A: a1, a0 per
// modulus); B's table is weighted, so B's planes hold u = w b (u1, u0).  Only
// the first kdim columns of each plane row are written.
struct OperandPlan {
    DigitArgs da;
    dim3 dgrid;
    int balanced = 0, gsteps = 0;
    bool pair = false;
    CUtensorMap tmD, tmT, tmR;
    ResidueArgs ra;
    size_t smem = 0;
};
static gbmm_status plan_operand(crt_tables *t, const gbmm_mat &X, int transpose, int rowsR, int kdim, int kp, int weighted,
                                __nv_bfloat16 *R, __nv_bfloat16 *D, bool grouped, OperandPlan &op) {
    const int dxp = operand_dxp(X);
    const int64_t E = (int64_t)X.rows * X.cols;
    if (E > (int64_t)INT32_MAX - 4 * BM) return set_error(GBMM_ERR_UNSUPPORTED, "crt: more than 2^31 entries in one operand");
    const int nk = dxp / BK;
    // unsigned byte digits up to 512 per row; longer rows in balanced digits, whose
    // groups are nearly twice as long (fewer groups, wider table tiles)
    op.balanced = nk > RES_GROUP_STEPS_U;
    op.gsteps = op.balanced ? RES_GROUP_STEPS_B : RES_GROUP_STEPS_U;
    DigitArgs &a = op.da;
    memset(&a, 0, sizeof a);
    a.limbs = X.limbs; a.sizes = X.sizes; a.ld = X.ld; a.rs = X.rs; a.rows = X.rows; a.cols = X.cols;
    a.nlimbs = X.nlimbs; a.transpose = transpose; a.dxp = dxp; a.out = D;
    op.dgrid = dim3((unsigned)((X.cols + 31) / 32), (unsigned)((X.rows + 3) / 4), (unsigned)((dxp / 4 + 63) / 64));
    __nv_bfloat16 *T = nullptr;
    int tpitch = dxp;
    GBMM_TRY(residue_table(t, dxp, weighted, &T, &tpitch));
    const int G = (nk + op.gsteps - 1) / op.gsteps;
    int BN = 256;
    while (BN * G > 256) BN /= 2;
    if (BN < 64) return set_error(GBMM_ERR_UNSUPPORTED, "crt: entries longer than 30720 bits");
    op.pair = !grouped && residue_pair(nk);
    const int NP = op.pair ? 2 : 1;
    GBMM_TRY(make_map(&op.tmD, D, dxp, E, dxp, BK, BM));
    GBMM_TRY(make_map(&op.tmT, T, dxp, residue_cols(t->P), tpitch, BK, BN / NP));
    ResidueArgs &r = op.ra;
    memset(&r, 0, sizeof r);
    r.kdim = kdim; r.E = (int32_t)E; r.nk = nk;
    r.BN = BN; r.G = G; r.P = t->P; r.R = R; r.plane = (int64_t)rowsR * kp; r.kp = kp;
    r.ncols = residue_cols(t->P);
    r.n_ntiles = (r.ncols + BN - 1) / BN;
    r.ntiles = (int32_t)((int64_t)r.n_ntiles * ((E + NP * BM - 1) / (NP * BM)));
    // 32-entry boxes of one plane row: [32 planes][1 row][32 entries]
    r.tma_out = kdim % 32 == 0;
    if (r.tma_out) GBMM_TRY(make_map_planes(&op.tmR, R, kdim, rowsR, 2 * t->P, kp, r.plane));
    else op.tmR = op.tmD;  // unused
    // a grouped launch sizes every stage for 256 table columns
    const int bcols = grouped ? 256 : (op.pair ? BN / 2 : BN);
    op.smem = smem_bytes(op.pair ? RES_STAGES_PAIR : RES_STAGES, BM * 128 + (size_t)bcols * 128) +
              (size_t)RES_EPI_WARPS * (op.pair ? 2 : 1) * RES_STG_BYTES;
    return GBMM_OK;
}

// Digits of half hf of an operand given as two stacked limb halves: the stacked operand's
// digit rows straight from x's planes.  The high half's rows follow the low half's (A:
// rows m.., B: columns n..); both halves carry x's sign, and digits past a half's limbs
// read as zeros.
static DigitArgs half_digits(const OperandPlan &op, const crt_halves &hv, int hf, dim3 &grid) {
    const gbmm_mat &x = hv.x;
    DigitArgs a = op.da;
    a.limbs = x.limbs + (hf ? (int64_t)hv.hl * x.ld : 0);
    a.sizes = x.sizes;
    a.ld = x.ld;
    a.rs = x.rs;
    a.rows = x.rows;
    a.cols = x.cols;
    a.nlimbs = hf ? x.nlimbs - hv.hl : hv.hl;
    a.out = op.da.out + (hf ? (int64_t)x.rows * x.cols * op.da.dxp : 0);
    grid = dim3((unsigned)((x.cols + 31) / 32), (unsigned)((x.rows + 3) / 4), op.dgrid.z);
    return a;
}

static gbmm_status launch_operand(const OperandPlan &op, const crt_halves *halves, cudaStream_t s) {
    for (int hf = 0; hf < (halves ? 2 : 1); hf++) {
        dim3 grid = op.dgrid;
        const DigitArgs da = halves ? half_digits(op, *halves, hf, grid) : op.da;
        LaunchScope ls_("k_crt_digits", s);
        const Group<DigitJob> none{nullptr, nullptr, 0};
        if (op.balanced) GBMM_TRY(launch_one(k_crt_digits<true, false>, grid, 256, 0, s, da, none));
        else GBMM_TRY(launch_one(k_crt_digits<false, false>, grid, 256, 0, s, da, none));
        GBMM_CUDA_TRY(cudaGetLastError());
    }
    const Group<ResidueJob> none{nullptr, nullptr, 0};
    const size_t sm = op.smem;
    LaunchScope ls_("k_crt_residue", s);
#define RESIDUE_LAUNCH(GS_)                                                                                          \
    do {                                                                                                             \
        if (op.pair) {                                                                                       \
            GBMM_TRY(set_smem((const void *)k_crt_residue<RES_STAGES_PAIR, true, GS_, false>, sm));           \
            GBMM_TRY(launch_pairs(k_crt_residue<RES_STAGES_PAIR, true, GS_, false>, RES_THREADS,            \
                                  op.ra.ntiles, sm, s, op.tmD, op.tmT, op.tmR, op.ra, none, device_error_word()));   \
        } else {                                                                                                     \
            GBMM_TRY(set_smem((const void *)k_crt_residue<RES_STAGES, false, GS_, false>, sm));               \
            dim3 grid((unsigned)std::min<int64_t>(op.ra.ntiles, num_sms()));                                         \
            GBMM_TRY(launch_one(k_crt_residue<RES_STAGES, false, GS_, false>, grid, RES_THREADS, sm, s,      \
                                op.tmD, op.tmT, op.tmR, op.ra, none, device_error_word()));                          \
        }                                                                                                            \
    } while (0)
    if (op.gsteps == RES_GROUP_STEPS_B) RESIDUE_LAUNCH(RES_GROUP_STEPS_B);
    else RESIDUE_LAUNCH(RES_GROUP_STEPS_U);
#undef RESIDUE_LAUNCH
    GBMM_CUDA_TRY(cudaGetLastError());
    return GBMM_OK;
}

// The one-kernel form of the same (k_crt_residue2).  It takes rows of up to 512 digits,
// unless an operand is large and most of its 8 x 32 blocks padding.  Measured, digits and
// residues of both operands: 1024 x 16 x 1024 entries of 2048 bits 47 us, 61 in two kernels;
// 8192 x 8 x 16 of 4096 bits 228 and 255; 16384 x 6 x 16 of 2048 bits (5.3 times the entries)
// 222 and 267; 16384 x 4 x 16 of 4096 bits (8 times) 440 and 409; 65536 x 1 x 16 of 1024 bits 505 and
// 418.  Up to 64 K padded entries are three or four waves, and the second launch costs more.
static bool residue2_ok(const gbmm_mat &X, int rowsR, int kdim) {
    if (g_residue_mode >= 0 || operand_dxp(X) / BK > R2_SLOTS) return false;
    const int64_t padded = (int64_t)((kdim + 31) / 32 * 32) * ((rowsR + 7) / 8 * 8), E = (int64_t)rowsR * kdim;
    return padded <= 6 * E || padded <= 65536;
}
// 256-entry row blocks of an operand
static int64_t residue2_blocks(int rowsR, int kdim) { return (int64_t)((kdim + 31) / 32) * ((rowsR + 7) / 8); }
// Into how many CTA pairs the column tiles of a row block are split: few row blocks (of all
// the launch's operands together) leave pairs idle; each pair then converts the digits itself
// (about a third of a column tile's time).
static int residue2_split(int64_t blocks, int ncols) {
    const int64_t pairs = std::max(1, num_sms() / 2);
    const int nt = (ncols + 255) / 256;
    int best_g = 1;
    double best = 1e30;
    for (int g = 1; g <= nt; g++) {
        const double c = (double)((blocks * g + pairs - 1) / pairs) * (0.35 + (double)((nt + g - 1) / g));
        if (c < best) {
            best = c;
            best_g = g;
        }
    }
    return best_g;
}
static gbmm_status plan_residue2(crt_tables *t, const gbmm_mat &X, int transpose, int rowsR, int kdim, int kp, int weighted,
                                 __nv_bfloat16 *R, const crt_halves *halves, int ngr, Residue2Job &rp) {
    const int dxp = operand_dxp(X);
    __nv_bfloat16 *T = nullptr;
    int tpitch = dxp;
    GBMM_TRY(residue_table(t, dxp, weighted, &T, &tpitch));
    memset(&rp, 0, sizeof rp);
    Residue2Args &a = rp.a;
    const gbmm_mat &x = halves ? halves->x : X;
    a.limbs = x.limbs; a.sizes = x.sizes; a.ld = x.ld;
    a.srow = transpose ? 1 : x.rs;
    a.sk = transpose ? x.rs : 1;
    a.rows = rowsR; a.kdim = kdim; a.nlimbs = x.nlimbs;
    if (halves) {
        a.hrows = rowsR / 2;
        a.hl = halves->hl;
    }
    a.nk = dxp / BK;
    a.ncols = residue_cols(t->P);
    a.n_ntiles = (a.ncols + 255) / 256;
    a.nkb = (kdim + 31) / 32;
    const int64_t rb = residue2_blocks(rowsR, kdim);
    a.ngr = ngr;
    if (rb * a.ngr > INT32_MAX / 2) return set_error(GBMM_ERR_UNSUPPORTED, "crt: too many entries in one operand");
    a.units = (int32_t)(rb * a.ngr);
    // One tile per pair: the widest is the launch's time, so they are of about equal width
    // (both operands at 64 x 64 entries of 1024 bits: 28 us, 30 in tiles of 256).  Otherwise
    // full tiles and a narrow last one, whose MMAs cost less than the rounding of equal ones
    // to 32 columns (512 x 512 of 4096 bits: 526 us, 542 in equal tiles).
    a.BN = a.ngr == a.n_ntiles ? ((a.ncols + a.n_ntiles - 1) / a.n_ntiles + 31) / 32 * 32 : 256;
    GBMM_TRY(make_map(&rp.tmT, T, dxp, residue_cols(t->P), tpitch, BK, (uint32_t)a.BN / 2));
    GBMM_TRY(make_map_planes(&rp.tmR, R, kdim, rowsR, 2 * t->P, kp, (uint64_t)rowsR * kp));
    return GBMM_OK;
}
static constexpr size_t R2_SMEM =
    (size_t)(R2_SLOTS + R2_STAGES) * R2_TILE + (size_t)R2_EPI * R2_NBUF * RES_STG_BYTES + sizeof(Residue2Bars) + 1024 + 64;
static gbmm_status launch_residue2(const Residue2Two &two, cudaStream_t s) {
    auto kern = k_crt_residue2<false>;
    GBMM_TRY(set_smem((const void *)kern, R2_SMEM));
    LaunchScope ls_("k_crt_residue2", s);
    const Group<Residue2Job> none{nullptr, nullptr, 0};
    return launch_pairs(kern, R2_THREADS, (int64_t)two.j[0].a.units + two.j[1].a.units, R2_SMEM, s, two, none,
                        device_error_word());
}

// Product GEMM over residue planes RA [2P][m][kp] and RB [2P][n][kp].  The maps'
// inner extent is k, not kp: the columns k .. kp-1 of the last K step lie outside
// and read as zeros, so the planes need no cleared padding.
struct ProductPlan {
    CUtensorMap tmA, tmB;
    ProductArgs pa;
    bool pair = false;
    size_t smem = 0;
};
static gbmm_status plan_product(crt_tables *t, __nv_bfloat16 *RA, __nv_bfloat16 *RB, __nv_bfloat16 *Y, int m, int k, int n,
                                int kp, int npad, int tiles, bool grouped, ProductPlan &pp) {
    const int P = t->P;
    GBMM_TRY(make_map(&pp.tmA, RA, k, (uint64_t)2 * P * m, kp, BK, BM));
    GBMM_TRY(make_map(&pp.tmB, RB, k, (uint64_t)2 * P * n, kp, BK, PBX));
    ProductArgs &pa = pp.pa;
    memset(&pa, 0, sizeof pa);
    pa.m = m; pa.n = n; pa.npad = npad; pa.nk = kp / BK; pa.P = P; pa.Y = Y;
    pa.yblk = (int64_t)2 * t->Pp * 64;
    // CTA pairs pay off once the K loop is long enough to hide the pair's per-tile
    // synchronisation (measured: faster at k = 512, slower at k = 256); a plan may
    // fix the form (tiles: 1 one-CTA tiles, 2 CTA pairs); grouped launches use one-CTA tiles
    pp.pair = !grouped && (tiles == 0 ? pa.nk >= PROD_PAIR_MIN_NK : tiles == 2);
    const int NP = pp.pair ? 2 : 1;
    pa.nyt = (m + NP * BM - 1) / (NP * BM);
    pa.nxt = (n + PBX - 1) / PBX;
    pa.ntiles = (int64_t)P * pa.nyt * pa.nxt;
    pp.smem = (pp.pair ? smem_bytes(PROD_STAGES_PAIR, 2 * BM * 128 + PBX * 128)
                       : smem_bytes(PROD_STAGES, 2 * BM * 128 + 2 * PBX * 128)) + 8 * PROD_STG_BYTES;
    return GBMM_OK;
}

static gbmm_status launch_product(const ProductPlan &pp, cudaStream_t s) {
    const Group<ProductJob> none{nullptr, nullptr, 0};
    uint32_t *err = device_error_word();
    LaunchScope ls_("k_crt_product", s);
    if (pp.pair) {
        GBMM_TRY(set_smem((const void *)k_crt_product<PROD_STAGES_PAIR, true, false>, pp.smem));
        GBMM_TRY(launch_pairs(k_crt_product<PROD_STAGES_PAIR, true, false>, CTA_THREADS8, pp.pa.ntiles, pp.smem, s,
                              pp.tmA, pp.tmB, pp.pa, none, err));
    } else {
        GBMM_TRY(set_smem((const void *)k_crt_product<PROD_STAGES, false, false>, pp.smem));
        dim3 grid((unsigned)std::min<int64_t>(pp.pa.ntiles, num_sms()));
        GBMM_TRY(launch_one(k_crt_product<PROD_STAGES, false, false>, grid, CTA_THREADS8, pp.smem, s, pp.tmA, pp.tmB,
                            pp.pa, none, err));
    }
    GBMM_CUDA_TRY(cudaGetLastError());
    return GBMM_OK;
}

// Y as a 3-D map [Ep/64 blocks][2P rows][64 entries] with a block pitch of 2Pp
// rows: boxes of 64 entries x 64 rows; rows 2P .. 2Pp-1 read as zeros.
static gbmm_status make_map_yblocks(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t rows_pitch, uint64_t blocks) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return set_error(GBMM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    if (reinterpret_cast<uintptr_t>(ptr) & 15) return set_error(GBMM_ERR_INVALID, "tensor map base not 16-byte aligned");
    cuuint64_t dims[3] = {64, rows, blocks};
    cuuint64_t strides[2] = {64 * 2, rows_pitch * 64 * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)BK, 1};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(ptr), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(GBMM_ERR_CUDA, "cuTensorMapEncodeTiled (Y blocks) failed (%d)", (int)r);
    return GBMM_OK;
}

// Reconstruction of C (m x n, Y's entries in rows of npad) from Y.
struct ReconPlan {
    CUtensorMap tmY, tmT;
    ReconArgs ra;
    int db = 7;
    bool pair = false;
    size_t smem = 0;
};
static gbmm_status plan_recon(crt_tables *t, __nv_bfloat16 *Y, int m, int n, int npad, const gbmm_mat &c, int tiles,
                              bool grouped, ReconPlan &rp) {
    const int64_t E = (int64_t)m * npad, Ep = (E + 63) / 64 * 64;
    GBMM_TRY(make_map_yblocks(&rp.tmY, Y, (uint64_t)2 * t->P, (uint64_t)2 * t->Pp, (uint64_t)(Ep / 64)));
    // CTA pairs once the K loop over the 2Pp moduli digits is long enough (see the
    // product), unless the plan fixes the form; grouped launches use CTA pairs
    rp.pair = grouped || (tiles == 0 ? 2 * t->Pp / BK >= PROD_PAIR_MIN_NK : tiles == 2);
    const int NP = rp.pair ? 2 : 1, TROWS = 256 / NP;
    GBMM_TRY(make_map(&rp.tmT, t->d_recon, 2 * t->Pp, (uint64_t)t->NT * RTAB, 2 * t->Pp, BK, TROWS));
    ReconArgs &ra = rp.ra;
    memset(&ra, 0, sizeof ra);
    ra.E = E; ra.ncols = npad; ra.ccols = n; ra.nk = 2 * t->Pp / BK; ra.NT = (SROWS + t->Dout + 255) / 256;
    ra.nlast = (SROWS + t->Dout - 256 * (ra.NT - 1) + 31) / 32 * 32;
    rp.db = t->db;
    ra.Dout = t->Dout; ra.vtab = t->d_vtab; ra.climbs = c.limbs; ra.csizes = c.sizes; ra.cld = c.ld; ra.crs = c.rs;
    ra.cnlimbs = c.nlimbs; ra.kpad = 2 * t->Pp;
    ra.mt0 = 0;
    ra.nmt = (E + NP * BM - 1) / (NP * BM);
    // a grouped launch reads Mod's chunk values from global memory
    const size_t extra = (grouped ? 0 : (size_t)(t->Dout + 31) / 32 * 32) + sizeof(ReconXfer) + 64;
    rp.smem = smem_bytes(rp.pair ? REC_STAGES_PAIR : REC_STAGES, BM * 128 + TROWS * 128) + extra;
    return GBMM_OK;
}

int crt_moduli(int64_t bits_a, int64_t bits_b, int k) {
    int lg = 0;
    while ((1LL << lg) < std::max(k, 1)) lg++;
    return moduli_for_bits(bits_a + bits_b + lg + 2 + 16);
}

// device workspace (bytes) of one single-pass product: residue planes, Y, and
// digits (one operand's at a time, or both when `both_digits`)
static size_t crt_workspace(const gbmm_mat &a, const gbmm_mat &b, int64_t bits_a, int64_t bits_b, int nprimes,
                            bool both_digits) {
    const int m = a.rows, k = a.cols, n = b.cols;
    int P = nprimes > 0 ? nprimes : crt_moduli(bits_a, bits_b, k);
    if (P <= 0) return 0;
    const int Pp = (2 * P + 63) / 64 * 32;
    const int kp = (k + 63) / 64 * 64;
    const int64_t Ep = ((int64_t)m * ((n + YPAD - 1) / YPAD * YPAD) + 63) / 64 * 64;
    const size_t da = align256(digits_bytes(a)), db = align256(digits_bytes(b));
    return align256((size_t)2 * P * m * kp * 2) + align256((size_t)2 * P * n * kp * 2) + align256((size_t)2 * Pp * Ep * 2) +
           (both_digits ? da + db : std::max(da, db)) + 8192;
}

bool crt_feasible(int la, int lb, int k) {
    const int P = crt_moduli(32LL * la, 32LL * lb, std::min(k, PROD_MAX_K));
    // at most four residue accumulation groups: digit rows of up to 4 * 15 * 64 digits
    return P > 0 && P <= 1023 && 4 * std::max(la, lb) <= 4 * RES_GROUP_STEPS_B * BK;
}

static gbmm_mat shape_only(int rows, int cols, int nlimbs) {
    gbmm_mat x;
    memset(&x, 0, sizeof x);
    x.rows = rows; x.cols = cols; x.nlimbs = nlimbs;
    return x;
}

size_t crt_workspace_bytes(int la, int lb, int m, int k, int n, int cn) {
    const int kc = std::min(k, PROD_MAX_K);
    size_t ws = crt_workspace(shape_only(m, kc, la), shape_only(kc, n, lb), 32LL * la, 32LL * lb, 0, false);
    // an accumulating chunk adds a product-sized temporary
    if (k > kc) ws += align256((size_t)m * n * (std::max(cn, la + lb + 4) + 1) * 4) + 8192;
    return ws;
}

bool crt_single_pass(int k) { return k <= PROD_MAX_K; }

gbmm_status crt_matmul(gbmm_handle h, const gbmm_mat &c, const gbmm_mat &a, const gbmm_mat &b, int64_t bits_a,
                       int64_t bits_b, int nprimes, int accumulate, cudaStream_t s, const crt_halves *halves) {
    const int m = a.rows, k = a.cols, n = b.cols;
    // stage hooks apply to this product only; any branch but the single-pass one
    // waits for B at once and runs the reconstruction whole
    crt_stage_hooks *hk = h->stage;
    h->stage = nullptr;
    if (hk && (m == 0 || n == 0 || k == 0 || accumulate || k > PROD_MAX_K)) {
        if (hk->b_ready) GBMM_CUDA_TRY(cudaStreamWaitEvent(s, hk->b_ready, 0));
        hk = nullptr;
    }
    if (m == 0 || n == 0) return GBMM_OK;
    if (k == 0) return accumulate ? GBMM_OK : launch_mat_zero(c, s);
    if (halves && (accumulate || k > PROD_MAX_K))
        return set_error(GBMM_ERR_UNSUPPORTED, "crt: stacked halves need a single-pass product");
    if (accumulate) {
        // C += A*B: product into a workspace matrix, then one elementwise add
        size_t mark = arena_mark(h);
        const int cn = std::max(c.nlimbs, (int)((bits_a + bits_b + 64) / 32) + 2);
        size_t need = align256((size_t)m * n * cn * 4) + align256((size_t)m * n * 4) + 4096;
        GBMM_TRY(arena_reserve(h, need + crt_workspace(a, b, bits_a, bits_b, nprimes, false)));
        gbmm_mat T;
        T.rows = m; T.cols = n; T.nlimbs = cn; T.pad_ = 0; T.rs = n; T.ld = (int64_t)m * n;
        T.limbs = (uint32_t *)arena_alloc(h, (size_t)m * n * cn * 4);
        T.sizes = (int32_t *)arena_alloc(h, (size_t)m * n * 4);
        if (!T.limbs || !T.sizes) return set_error(GBMM_ERR_NOMEM, "crt: accumulate workspace");
        gbmm_status st = crt_matmul(h, T, a, b, bits_a, bits_b, nprimes, 0, s);
        if (st == GBMM_OK) st = launch_mat_addsub(c, c, T, 0, s);
        arena_release(h, mark);
        return st;
    }
    if (k > PROD_MAX_K) {
        // inner dimension in chunks of 512: C = A_0 B_0, then C += A_j B_j
        for (int k0 = 0; k0 < k; k0 += PROD_MAX_K) {
            const int kc = std::min(PROD_MAX_K, k - k0);
            gbmm_mat ac = sub_view(a, 0, k0, m, kc), bc = sub_view(b, k0, 0, kc, n);
            GBMM_TRY(crt_matmul(h, c, ac, bc, bits_a, bits_b, nprimes, k0 > 0, s));
        }
        return GBMM_OK;
    }
    int P = nprimes > 0 ? nprimes : crt_moduli(bits_a, bits_b, k);
    // one exact FP32 accumulation in the reconstruction covers 2P * 2^13 < 2^24
    if (P <= 0 || P > 1023)
        return set_error(GBMM_ERR_UNSUPPORTED, "crt: product bound needs %d moduli (at most 1023)", P);
    crt_tables *t = nullptr;
    GBMM_TRY(get_tables(h->crt, P, &t));
    if (!get_encode()) return set_error(GBMM_ERR_CUDA, "crt: no tensor-map encoder");

    const int kp = (k + 63) / 64 * 64;  // residue-plane row pitch (TMA needs 16-byte pitches)
    // Y's entries: rows of C times n padded to whole groups of 16 (the product
    // GEMM's epilogue then stores only whole 32-byte runs)
    const int npad = (n + YPAD - 1) / YPAD * YPAD;
    const int64_t E = (int64_t)m * npad;
    const int64_t Ep = (E + 63) / 64 * 64;
    GBMM_TRY(arena_reserve(h, crt_workspace(a, b, bits_a, bits_b, P, false)));
    size_t mark = arena_mark(h);
    __nv_bfloat16 *RA = (__nv_bfloat16 *)arena_alloc(h, (size_t)2 * P * m * kp * 2);
    __nv_bfloat16 *RB = (__nv_bfloat16 *)arena_alloc(h, (size_t)2 * P * n * kp * 2);
    __nv_bfloat16 *Y = (__nv_bfloat16 *)arena_alloc(h, (size_t)2 * t->Pp * Ep * 2);
    if (!RA || !RB || !Y) return set_error(GBMM_ERR_NOMEM, "crt: workspace");
    // Nothing is cleared: the product reads RA / RB through maps k columns wide and
    // Y through a map 2P rows deep per 64-entry block, and the padding entries
    // E .. Ep-1 of Y only reach accumulator rows that are never stored.
    // Both operands in one launch where they take the one-kernel form, unless B is still on
    // its way: small operands then fill the chip together and large ones share a last wave.
    // Two launches and one, us for both operands: 64 x 64 entries of 1024 bits 31.9 and 16.1,
    // 256 x 256 of 2048 bits 93 and 75, 512 x 512 of 4096 bits 515 and 484.
    const bool both = residue2_ok(a, m, k) && residue2_ok(b, n, k) && !(hk && hk->b_ready);
    if (both) {
        const int split = residue2_split(residue2_blocks(m, k) + residue2_blocks(n, k), residue_cols(P));
        Residue2Two two;
        for (int side = 0; side < 2; side++) {
            // the operand with the longer rows first
            const int slot = operand_dxp(b) > operand_dxp(a) ? 1 - side : side;
            GBMM_TRY(plan_residue2(t, side ? b : a, side, side ? n : m, k, kp, side, side ? RB : RA,
                                   halves && halves->side == side ? halves : nullptr, split, two.j[slot]));
        }
        GBMM_TRY(launch_residue2(two, s));
    } else {
        for (int side = 0; side < 2; side++) {
            const gbmm_mat &x = side ? b : a;
            __nv_bfloat16 *R = side ? RB : RA;
            const int rows = side ? n : m;
            const crt_halves *hv = halves && halves->side == side ? halves : nullptr;
            if (side == 1 && hk && hk->b_ready) GBMM_CUDA_TRY(cudaStreamWaitEvent(s, hk->b_ready, 0));
            if (residue2_ok(x, rows, k)) {
                Residue2Two two;
                memset(&two, 0, sizeof two);
                const int split = residue2_split(residue2_blocks(rows, k), residue_cols(P));
                GBMM_TRY(plan_residue2(t, x, side, rows, k, kp, side, R, hv, split, two.j[0]));
                GBMM_TRY(launch_residue2(two, s));
                continue;
            }
            size_t mk = arena_mark(h);
            OperandPlan op;
            __nv_bfloat16 *D = (__nv_bfloat16 *)arena_alloc(h, digits_bytes(x));
            if (!D) return set_error(GBMM_ERR_NOMEM, "crt: workspace for digits");
            GBMM_TRY(plan_operand(t, x, side, rows, k, kp, side, R, D, false, op));
            GBMM_TRY(launch_operand(op, hv, s));
            arena_release(h, mk);
        }
    }
    {
        ProductPlan pp;
        GBMM_TRY(plan_product(t, RA, RB, Y, m, k, n, kp, npad, h->crt_tiles, false, pp));
        GBMM_TRY(launch_product(pp, s));
    }
    {
        ReconPlan rp;
        GBMM_TRY(plan_recon(t, Y, m, n, npad, c, h->crt_tiles, false, rp));
        ReconArgs ra = rp.ra;
        const int64_t nmt = ra.nmt;
        const Group<ReconJob> none{nullptr, nullptr, 0};
        uint32_t *err = device_error_word();
        auto kpair = rp.db == 8 ? k_crt_recon<REC_STAGES_PAIR, true, false, 8> : k_crt_recon<REC_STAGES_PAIR, true, false, 7>;
        auto kone = rp.db == 8 ? k_crt_recon<REC_STAGES, false, false, 8> : k_crt_recon<REC_STAGES, false, false, 7>;
        GBMM_TRY(set_smem(rp.pair ? (const void *)kpair : (const void *)kone, rp.smem));
        const int NP = rp.pair ? 2 : 1;
        // one launch, or (stage hooks) entry ranges each followed by an event
        const int parts = hk ? (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)hk->parts, (int64_t)CRT_MAX_PARTS, nmt})) : 1;
        for (int pi = 0; pi < parts; pi++) {
            ra.mt0 = nmt * pi / parts;
            ra.nmt = nmt * (pi + 1) / parts;
            LaunchScope ls_("k_crt_recon", s);
            if (rp.pair) {
                GBMM_TRY(launch_pairs(kpair, REC_THREADS, ra.nmt - ra.mt0, rp.smem, s,
                                      rp.tmY, rp.tmT, ra, none, err));
            } else {
                dim3 grid((unsigned)std::min<int64_t>(ra.nmt - ra.mt0, num_sms()));
                GBMM_TRY(launch_one(kone, grid, REC_THREADS, rp.smem, s, rp.tmY,
                                    rp.tmT, ra, none, err));
            }
            GBMM_CUDA_TRY(cudaGetLastError());
            if (hk && parts > 1) {
                GBMM_CUDA_TRY(cudaEventRecord(hk->part_ev[pi], s));
                // entries of C (dense, row-major) done after this part: Y's entries below
                // ra.nmt * NP * BM, mapped back through the padded row length
                const int64_t ye = std::min<int64_t>(E, ra.nmt * NP * BM);
                hk->part_end[pi] = std::min<int64_t>((int64_t)m * n, (ye / npad) * n + std::min<int64_t>(ye % npad, n));
            }
        }
        if (hk && parts > 1) hk->parts_done = parts;
    }
    arena_release(h, mark);
    return GBMM_OK;
}

// ---- grouped launches -------------------------------------------------------------------------
// The CRT products of a batch, collected without launching: every product's
// workspace is carved at once, its stage records go into per-stage lists, and
// each stage then runs as ONE persistent launch per kernel form over the tiles of
// all products (digits and residues by digit form, products on one-CTA tiles,
// reconstructions on CTA pairs).  Records are ordered by the cost of one tile,
// largest first, so that the long tiles start in the first wave.
struct crt_group {
    struct Rec {
        std::vector<char> bytes;  // one record
        int64_t tiles = 0;
        double cost = 0;  // per tile
    };
    // dig by digit form (unsigned, balanced); res by accumulation groups: unsigned
    // digits (one group), balanced with one group (256-column table tiles), balanced
    // with several (table tiles of 128 or 64 columns, a deeper ring of smaller
    // stages); rec[2 f + d]: reconstructions of products with (f = 1) and without a post
    // step, by table digits (d = 1: base 256)
    std::vector<Rec> dig[2], res[3], res2, prod, rec[4];  // res2: operands whose digits and residues are one kernel
    std::vector<std::function<gbmm_status(cudaStream_t)>> post;
    struct Sect {
        size_t jobs_off = 0, tile0_off = 0;
        int n = 0;
        int64_t total = 0;
    };
    Sect sdig[2], sres[3], sres2, sprod, srec[4];
    size_t smem_prod = 0, smem_rec = 0;
    std::vector<char> blob;
};

crt_group *crt_group_create() { return new crt_group(); }
void crt_group_destroy(crt_group *g) { delete g; }
bool crt_group_empty(const crt_group *g) { return g->prod.empty() && g->post.empty(); }
void crt_group_post(crt_group *g, std::function<gbmm_status(cudaStream_t)> f) { g->post.push_back(std::move(f)); }

size_t crt_group_ws(int la, int lb, int m, int k, int n) {
    return crt_workspace(shape_only(m, k, la), shape_only(k, n, lb), 32LL * la, 32LL * lb, 0, true) + 2048;
}

template <typename J>
static crt_group::Rec make_rec(const J &j, int64_t tiles, double cost) {
    crt_group::Rec r;
    r.bytes.resize(sizeof(J));
    memcpy(r.bytes.data(), &j, sizeof(J));
    r.tiles = tiles;
    r.cost = cost;
    return r;
}

gbmm_status crt_group_add(gbmm_handle h, crt_group *g, const gbmm_mat &c, const gbmm_mat &a, const gbmm_mat &b,
                          int64_t bits_a, int64_t bits_b, int nprimes, const crt_halves *halves) {
    const int m = a.rows, k = a.cols, n = b.cols;
    if (m == 0 || n == 0 || k == 0 || k > PROD_MAX_K)
        return set_error(GBMM_ERR_UNSUPPORTED, "crt group: needs a nonempty single-pass product");
    const int P = nprimes > 0 ? nprimes : crt_moduli(bits_a, bits_b, k);
    if (P <= 0 || P > 1023)
        return set_error(GBMM_ERR_UNSUPPORTED, "crt: product bound needs %d moduli (at most 1023)", P);
    crt_tables *t = nullptr;
    GBMM_TRY(get_tables(h->crt, P, &t));
    if (!get_encode()) return set_error(GBMM_ERR_CUDA, "crt: no tensor-map encoder");
    const int kp = (k + 63) / 64 * 64;
    const int npad = (n + YPAD - 1) / YPAD * YPAD;
    const int64_t Ep = ((int64_t)m * npad + 63) / 64 * 64;
    __nv_bfloat16 *RA = (__nv_bfloat16 *)arena_alloc(h, (size_t)2 * P * m * kp * 2);
    __nv_bfloat16 *RB = (__nv_bfloat16 *)arena_alloc(h, (size_t)2 * P * n * kp * 2);
    __nv_bfloat16 *Y = (__nv_bfloat16 *)arena_alloc(h, (size_t)2 * t->Pp * Ep * 2);
    if (!RA || !RB || !Y) return set_error(GBMM_ERR_NOMEM, "crt group: workspace");
    for (int side = 0; side < 2; side++) {
        const gbmm_mat &xs = side ? b : a;
        __nv_bfloat16 *R = side ? RB : RA;
        const int rows = side ? n : m;
        const crt_halves *hv = halves && halves->side == side ? halves : nullptr;
        if (residue2_ok(xs, rows, k)) {
            Residue2Job j2;  // not split: the batch's other products fill the chip
            GBMM_TRY(plan_residue2(t, xs, side, rows, k, kp, side, R, hv, 1, j2));
            g->res2.push_back(make_rec(j2, j2.a.units, (double)j2.a.nk * j2.a.n_ntiles));
            continue;
        }
        __nv_bfloat16 *D = (__nv_bfloat16 *)arena_alloc(h, digits_bytes(xs));
        if (!D) return set_error(GBMM_ERR_NOMEM, "crt group: workspace");
        OperandPlan op;
        GBMM_TRY(plan_operand(t, xs, side, rows, k, kp, side, R, D, true, op));
        if (hv) {
            for (int hf = 0; hf < 2; hf++) {
                DigitJob dj;
                memset(&dj, 0, sizeof dj);
                dim3 grid;
                dj.a = half_digits(op, *hv, hf, grid);
                dj.nbx = (int32_t)grid.x;
                dj.nby = (int32_t)grid.y;
                g->dig[op.balanced].push_back(make_rec(dj, (int64_t)grid.x * grid.y * grid.z, 1.0));
            }
        } else {
            DigitJob dj;
            memset(&dj, 0, sizeof dj);
            dj.a = op.da;
            dj.nbx = (int32_t)op.dgrid.x;
            dj.nby = (int32_t)op.dgrid.y;
            g->dig[op.balanced].push_back(make_rec(dj, (int64_t)op.dgrid.x * op.dgrid.y * op.dgrid.z, 1.0));
        }
        ResidueJob rj;
        memset(&rj, 0, sizeof rj);
        rj.tmD = op.tmD; rj.tmT = op.tmT; rj.tmR = op.tmR; rj.a = op.ra;
        const int rf = op.gsteps == RES_GROUP_STEPS_U ? 0 : (op.ra.BN > 128 ? 1 : 2);
        g->res[rf].push_back(make_rec(rj, op.ra.ntiles, (double)op.ra.nk * op.ra.BN));
    }
    ProductPlan pp;
    GBMM_TRY(plan_product(t, RA, RB, Y, m, k, n, kp, npad, 0, true, pp));
    ProductJob pj;
    memset(&pj, 0, sizeof pj);
    pj.tmA = pp.tmA; pj.tmB = pp.tmB; pj.a = pp.pa;
    g->prod.push_back(make_rec(pj, pp.pa.ntiles, (double)pp.pa.nk));
    g->smem_prod = std::max(g->smem_prod, pp.smem);
    ReconPlan rp;
    GBMM_TRY(plan_recon(t, Y, m, n, npad, c, 0, true, rp));
    ReconJob rj;
    memset(&rj, 0, sizeof rj);
    rj.tmY = rp.tmY; rj.tmT = rp.tmT; rj.a = rp.ra;
    g->rec[(halves ? 2 : 0) + (rp.db == 8)].push_back(make_rec(rj, rp.ra.nmt, (double)rp.ra.NT * rp.ra.nk));
    g->smem_rec = std::max(g->smem_rec, rp.smem);
    return GBMM_OK;
}

// One stage's records, largest tile cost first, then their tile offsets.
static void pack_section(std::vector<char> &blob, std::vector<crt_group::Rec> &recs, crt_group::Sect &sec) {
    std::stable_sort(recs.begin(), recs.end(),
                     [](const crt_group::Rec &x, const crt_group::Rec &y) { return x.cost > y.cost; });
    sec.n = (int)recs.size();
    sec.total = 0;
    if (recs.empty()) return;
    blob.resize((blob.size() + 127) & ~(size_t)127);
    sec.jobs_off = blob.size();
    for (const auto &r : recs) blob.insert(blob.end(), r.bytes.begin(), r.bytes.end());
    blob.resize((blob.size() + 127) & ~(size_t)127);
    sec.tile0_off = blob.size();
    std::vector<int64_t> t0(recs.size() + 1, 0);
    for (size_t i = 0; i < recs.size(); i++) t0[i + 1] = t0[i] + recs[i].tiles;
    sec.total = t0.back();
    const char *p = reinterpret_cast<const char *>(t0.data());
    blob.insert(blob.end(), p, p + t0.size() * sizeof(int64_t));
}

const std::vector<char> &crt_group_blob(crt_group *g) {
    g->blob.clear();
    for (int f = 0; f < 2; f++) pack_section(g->blob, g->dig[f], g->sdig[f]);
    for (int f = 0; f < 3; f++) pack_section(g->blob, g->res[f], g->sres[f]);
    pack_section(g->blob, g->res2, g->sres2);
    pack_section(g->blob, g->prod, g->sprod);
    for (int f = 0; f < 4; f++) pack_section(g->blob, g->rec[f], g->srec[f]);
    return g->blob;
}

template <typename J>
static Group<J> group_at(const char *d_blob, const crt_group::Sect &sec) {
    return Group<J>{reinterpret_cast<const J *>(d_blob + sec.jobs_off),
                    reinterpret_cast<const int64_t *>(d_blob + sec.tile0_off), sec.n};
}

gbmm_status crt_group_launch(crt_group *g, const char *d_blob, cudaStream_t s, cudaStream_t s2, cudaEvent_t ev) {
    if (reinterpret_cast<uintptr_t>(d_blob) & 127) return set_error(GBMM_ERR_INVALID, "crt group: blob not 128-byte aligned");
    uint32_t *err = device_error_word();
    static const CUtensorMap zmap = {};
    for (int f = 0; f < 2; f++) {
        const crt_group::Sect &sec = g->sdig[f];
        if (!sec.n) continue;
        if (sec.total > INT32_MAX) return set_error(GBMM_ERR_UNSUPPORTED, "crt group: too many digit blocks");
        DigitArgs none;
        memset(&none, 0, sizeof none);
        LaunchScope ls_("k_crt_digits", s);
        const dim3 grid((unsigned)sec.total);
        if (f) GBMM_TRY(launch_one(k_crt_digits<true, true>, grid, 256, 0, s, none, group_at<DigitJob>(d_blob, sec)));
        else GBMM_TRY(launch_one(k_crt_digits<false, true>, grid, 256, 0, s, none, group_at<DigitJob>(d_blob, sec)));
        GBMM_CUDA_TRY(cudaGetLastError());
    }
    // residue GEMMs: 4 stages of 48 KB for 256-column table tiles, 6 of 32 KB for
    // operands whose several accumulation groups narrow the tiles to 128 columns
    static constexpr int RES_STAGES_NARROW = 6;
    for (int f = 0; f < 3; f++) {
        const crt_group::Sect &sec = g->sres[f];
        if (!sec.n) continue;
        ResidueArgs none;
        memset(&none, 0, sizeof none);
        const dim3 grid((unsigned)std::min<int64_t>(sec.total, num_sms()));
        const size_t stg = (size_t)RES_EPI_WARPS * RES_STG_BYTES;
        LaunchScope ls_("k_crt_residue", s);
        if (f == 0) {
            auto kern = k_crt_residue<RES_STAGES, false, RES_GROUP_STEPS_U, true, 256>;
            const size_t sm = smem_bytes(RES_STAGES, BM * 128 + 256 * 128) + stg;
            GBMM_TRY(set_smem((const void *)kern, sm));
            GBMM_TRY(launch_one(kern, grid, RES_THREADS, sm, s, zmap, zmap, zmap, none,
                                group_at<ResidueJob>(d_blob, sec), err));
        } else if (f == 1) {
            auto kern = k_crt_residue<RES_STAGES, false, RES_GROUP_STEPS_B, true, 256>;
            const size_t sm = smem_bytes(RES_STAGES, BM * 128 + 256 * 128) + stg;
            GBMM_TRY(set_smem((const void *)kern, sm));
            GBMM_TRY(launch_one(kern, grid, RES_THREADS, sm, s, zmap, zmap, zmap, none,
                                group_at<ResidueJob>(d_blob, sec), err));
        } else {
            auto kern = k_crt_residue<RES_STAGES_NARROW, false, RES_GROUP_STEPS_B, true, 128>;
            const size_t sm = smem_bytes(RES_STAGES_NARROW, BM * 128 + 128 * 128) + stg;
            GBMM_TRY(set_smem((const void *)kern, sm));
            GBMM_TRY(launch_one(kern, grid, RES_THREADS, sm, s, zmap, zmap, zmap, none,
                                group_at<ResidueJob>(d_blob, sec), err));
        }
        GBMM_CUDA_TRY(cudaGetLastError());
    }
    if (g->sres2.n) {
        Residue2Two none;
        memset(&none, 0, sizeof none);
        auto kern = k_crt_residue2<true>;
        GBMM_TRY(set_smem((const void *)kern, R2_SMEM));
        LaunchScope ls_("k_crt_residue2", s);
        GBMM_TRY(launch_pairs(kern, R2_THREADS, g->sres2.total, R2_SMEM, s, none,
                              group_at<Residue2Job>(d_blob, g->sres2), err));
    }
    if (g->sprod.n) {
        ProductArgs none;
        memset(&none, 0, sizeof none);
        auto kern = k_crt_product<PROD_STAGES, false, true>;
        GBMM_TRY(set_smem((const void *)kern, g->smem_prod));
        const dim3 grid((unsigned)std::min<int64_t>(g->sprod.total, num_sms()));
        LaunchScope ls_("k_crt_product", s);
        GBMM_TRY(launch_one(kern, grid, CTA_THREADS8, g->smem_prod, s, zmap, zmap, none,
                            group_at<ProductJob>(d_blob, g->sprod), err));
        GBMM_CUDA_TRY(cudaGetLastError());
    }
    // The products with post steps first: their shifted adds then run on s2 while
    // the other reconstructions do.  With s2 the two table forms run side by side too: an entry's N
    // tiles follow one another, so on few entries a launch takes as long as the longest entry
    // however little it has to do (9 products of up to 36 rows and 13489 bits, us: 288 one after the
    // other, 233 side by side; 24 of up to 150 rows and 15092 bits 808 and 692).
    const bool side = s2 && ev;
    if (side && (g->srec[0].n || g->srec[2].n) && (g->srec[1].n || g->srec[3].n)) {
        GBMM_CUDA_TRY(cudaEventRecord(ev, s));
        GBMM_CUDA_TRY(cudaStreamWaitEvent(s2, ev, 0));
    }
    auto recon = [&](int f, int d, cudaStream_t rs) -> gbmm_status {
        const crt_group::Sect &sec = g->srec[2 * f + d];
        if (!sec.n) return GBMM_OK;
        ReconArgs none;
        memset(&none, 0, sizeof none);
        auto kern = d ? k_crt_recon<REC_STAGES_PAIR, true, true, 8> : k_crt_recon<REC_STAGES_PAIR, true, true, 7>;
        GBMM_TRY(set_smem((const void *)kern, g->smem_rec));
        LaunchScope ls_("k_crt_recon", rs);
        return launch_pairs(kern, REC_THREADS, sec.total, g->smem_rec, rs, zmap, zmap, none, group_at<ReconJob>(d_blob, sec),
                            err);
    };
    // base-128 tables beside base-256 ones, on s2 (where there are both)
    const cudaStream_t s7 = side && (g->srec[1].n || g->srec[3].n) ? s2 : s;
    GBMM_TRY(recon(1, 1, s));
    GBMM_TRY(recon(1, 0, s7));
    if (side && !g->post.empty()) GBMM_CUDA_TRY(cudaEventRecord(ev, s));
    GBMM_TRY(recon(0, 0, s7));
    if (!g->post.empty()) {
        if (side) GBMM_CUDA_TRY(cudaStreamWaitEvent(s2, ev, 0));
        for (auto &fn : g->post) GBMM_TRY(fn(side ? s2 : s));
    }
    GBMM_TRY(recon(0, 1, s));
    return GBMM_OK;
}

}  // namespace gbmm

using namespace gbmm;

// Internal test hook (not part of the public ABI): D = A * B^T through the
// tcgen05 pipeline.  A: bf16 [M x K] (a_mn = 0) or [K x M] (a_mn = 1), B: bf16
// [N x K]; K a multiple of 64, M and N multiples of 128 ... any (padded by TMA).
extern "C" gbmm_status gbmmx_test_gemm(const void *A, const void *B, int32_t *D, int32_t M, int32_t N, int32_t K,
                                       int32_t a_mn, void *stream) {
    cudaStream_t s = as_stream(stream);
    if (K % 64 || M % 8 || N % 8) return set_error(GBMM_ERR_INVALID, "test gemm: K % 64, M % 8, N % 8 required");
    CUtensorMap tmA, tmB;
    if (a_mn) GBMM_TRY(make_map(&tmA, A, M, K, M, 64, BK));
    else GBMM_TRY(make_map(&tmA, A, K, M, K, BK, BM));
    GBMM_TRY(make_map(&tmB, B, K, N, K, BK, BM));
    TestArgs ta;
    ta.M = M; ta.N = N; ta.nk = K / BK; ta.a_mn = a_mn; ta.D = D;
    ta.skip_step = -1;
    ta.wait_limit = tc::WAIT_LIMIT_CLOCKS;
    const size_t sm = smem_bytes(TEST_STAGES, 2 * BM * 128);
    GBMM_TRY(set_smem((const void *)k_gemm_test<TEST_STAGES>, sm));
    dim3 grid((unsigned)((N + BM - 1) / BM), (unsigned)((M + BM - 1) / BM));
    LaunchScope ls_("k_gemm_test", s);
    k_gemm_test<TEST_STAGES><<<grid, CTA_THREADS, sm, s>>>(tmA, tmB, ta, device_error_word());
    GBMM_CUDA_TRY(cudaGetLastError());
    return check_device_error(s);
}

// Internal test hook for the failure path: the same single-CTA pipeline (M = N =
// 128, one CTA) with K step `skip_step` never loaded (its stage barrier is never
// armed, so the MMA issuer's wait for it cannot complete) and every wait bounded
// by `wait_limit_clocks`.  Each role gives up when its wait runs out, records
// DEVERR_TIMEOUT, lets its in-flight copies and MMAs finish (bounded waits), and
// the CTA frees its TMEM and exits; the status comes back as GBMM_ERR_TIMEOUT.
extern "C" gbmm_status gbmmx_test_gemm_timeout(const void *A, const void *B, int32_t *D, int32_t K, int32_t skip_step,
                                               int64_t wait_limit_clocks, void *stream) {
    cudaStream_t s = as_stream(stream);
    if (K % 64 || K < 64 || skip_step < 0 || skip_step >= K / BK || wait_limit_clocks < 1000 ||
        wait_limit_clocks > tc::WAIT_LIMIT_CLOCKS)
        return set_error(GBMM_ERR_INVALID, "test gemm timeout: bad arguments");
    CUtensorMap tmA, tmB;
    GBMM_TRY(make_map(&tmA, A, K, BM, K, BK, BM));
    GBMM_TRY(make_map(&tmB, B, K, BM, K, BK, BM));
    TestArgs ta;
    ta.M = BM; ta.N = BM; ta.nk = K / BK; ta.a_mn = 0; ta.D = D;
    ta.skip_step = skip_step;
    ta.wait_limit = wait_limit_clocks;
    const size_t sm = smem_bytes(TEST_STAGES, 2 * BM * 128);
    GBMM_TRY(set_smem((const void *)k_gemm_test<TEST_STAGES>, sm));
    LaunchScope ls_("k_gemm_test", s);
    k_gemm_test<TEST_STAGES><<<dim3(1, 1), CTA_THREADS, sm, s>>>(tmA, tmB, ta, device_error_word());
    GBMM_CUDA_TRY(cudaGetLastError());
    return check_device_error(s);
}

// Internal test hook: the same product through the CTA-pair kernel (A and B
// K-major only).
extern "C" gbmm_status gbmmx_test_gemm_pair(const void *A, const void *B, int32_t *D, int32_t M, int32_t N, int32_t K,
                                            void *stream) {
    cudaStream_t s = as_stream(stream);
    if (K % 64 || M % 8 || N % 8) return set_error(GBMM_ERR_INVALID, "test gemm: K % 64, M % 8, N % 8 required");
    CUtensorMap tmA, tmB;
    GBMM_TRY(make_map(&tmA, A, K, M, K, BK, BM));
    GBMM_TRY(make_map(&tmB, B, K, N, K, BK, BM));
    TestArgs ta;
    ta.M = M; ta.N = N; ta.nk = K / BK; ta.a_mn = 0; ta.D = D;
    ta.skip_step = -1;
    ta.wait_limit = tc::WAIT_LIMIT_CLOCKS;
    const size_t sm = smem_bytes(TEST_STAGES, 2 * BM * 128);
    GBMM_TRY(set_smem((const void *)k_gemm_test_pair<TEST_STAGES>, sm));
    const unsigned tiles = (unsigned)(((M + 255) / 256) * ((N + 255) / 256));
    LaunchScope ls_("k_gemm_test_pair", s);
    k_gemm_test_pair<TEST_STAGES><<<2 * tiles, CTA_THREADS, sm, s>>>(tmA, tmB, ta, device_error_word());
    GBMM_CUDA_TRY(cudaGetLastError());
    return check_device_error(s);
}

extern "C" gbmm_status gbmmx_crt_params(int64_t bits_a, int64_t bits_b, int32_t k, int32_t *nmoduli) {
    if (!nmoduli) return set_error(GBMM_ERR_INVALID, "null pointer");
    *nmoduli = crt_moduli(bits_a, bits_b, k);
    return GBMM_OK;
}

// Internal hook: builds the host side of the table set for P moduli (no device
// work) and returns an FNV-1a checksum of its contents; *ms gets the build time.
extern "C" uint64_t gbmmx_table_build(int32_t P, double *ms) {
    if (P < 1 || P > 2 * CMOD_PAIRS) return 0;
    const auto t0 = std::chrono::steady_clock::now();
    crt_tables_host o;
    build_tables_host(P, o);
    const auto t1 = std::chrono::steady_clock::now();
    if (ms) *ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
    uint64_t h = 1469598103934665603ull;
    auto mix = [&](const void *p, size_t n) {
        const unsigned char *c = (const unsigned char *)p;
        for (size_t i = 0; i < n; i++) h = (h ^ c[i]) * 1099511628211ull;
    };
    mix(o.recon.data(), o.recon.size() * 2);
    mix(o.vtab.data(), o.vtab.size() * 4);
    mix(o.mods.data(), o.mods.size() * sizeof(ModConst));
    return h;
}

// Test hook: bits of a digit of the table that P moduli get, and the builds that took.
extern "C" int32_t gbmmx_table_digits(int32_t P, int32_t *builds) {
    if (P < 1 || P > 2 * CMOD_PAIRS) return 0;
    crt_tables_host o;
    const int n = build_tables_fit(P, o);
    if (builds) *builds = n;
    return o.db;
}

// Test hook: launch the four stages' kernels with programmatic stream
// serialization (1, the default) or as plain stream-ordered launches (0); returns
// the previous setting.
extern "C" int32_t gbmmx_launch_pdl(int32_t enable) {
    const int32_t old = g_pdl ? 1 : 0;
    g_pdl = enable != 0;
    return old;
}

// Test hook: the residue GEMM's form (-1 by the K loop's length, 0 single CTAs,
// 1 or more CTA pairs); returns the previous setting.
extern "C" int32_t gbmmx_residue_mode(int32_t mode) {
    const int32_t old = g_residue_mode;
    g_residue_mode = mode < 0 ? -1 : (mode > 1 ? 1 : mode);
    return old;
}
