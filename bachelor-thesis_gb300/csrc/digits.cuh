// Limb planes -> rows of byte digits in bf16: the operands of the exact tensor-core
// GEMMs (the residue stage of the CRT form, the digit-column products of the limb form).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace gbmm {

// bf16 bit patterns of two small integers (|v| <= 256 has at most 9 significant
// bits, so the low 16 bits of its FP32 encoding are zero and truncation is exact):
// a in the low half, b in the high half
__device__ __forceinline__ uint32_t bf16x2_bits(float a, float b) {
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// bf16 bits of bytes k and k+1 of w, byte k in the low half (unsigned digits).
// Each byte b becomes the FP32 value 2^23 + b (bits 0x4B000000 | b, built by one
// byte permute) minus 2^23, which is exact; b has at most 8 significant bits, so
// the top half of its FP32 encoding is its bf16 encoding.
__device__ __forceinline__ uint32_t byte_pair_bf16(uint32_t w, int k) {
    const float lo = __fadd_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u + k)), -8388608.0f);
    const float hi = __fadd_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7541u + k)), -8388608.0f);
    return bf16x2_bits(lo, hi);
}

// Balanced byte digits of limb w: byte b_i becomes d_i = b_i + c_i - 256 m_i with
// m_i its top bit and c_i the top bit of the byte below (cin for byte 0), so
// sum d_i 256^i = sum b_i 256^i with every d_i in [-128, 128].  The carry needs no
// propagation: c_i depends on the byte below only.  The last digit of a row
// (last, byte 3) keeps its carry and is not reduced: it lies in [0, 256].
// Computed as e_i = (b_i ^ 128) + c_i = d_i + 128 in [0, 256]: two byte permutes
// and an integer add build the FP32 bits of 2^23 + e_i, and one exact FADD of
// -(2^23 + 128) leaves d_i.  With at most 9 significant bits the top half of the
// FP32 encoding is the bf16 encoding.  No int->float conversion instructions.
__device__ __forceinline__ void limb_digits_bal(uint32_t w, uint32_t cin, bool last, float (&d)[4]) {
    const uint32_t x = w ^ 0x80808080u;                          // b_i ^ 128 per byte
    const uint32_t c = ((w & 0x80808080u) >> 7 << 8) | cin;      // c_i in bit 0 of byte i
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t bits = __byte_perm(x, 0x4B000000u, 0x7650u + i) + __byte_perm(c, 0u, 0x4440u + i);
        d[i] = __fadd_rn(__uint_as_float(bits), -8388736.0f);  // (2^23 + e_i) - (2^23 + 128)
    }
    if (last) {
        // the row's last digit unreduced: b_3 + c_3 (the reduced form subtracted 256 when m_3 = 1)
        d[3] = (w >> 31) ? __fadd_rn(d[3], 256.0f) : d[3];
    }
}

// The digits carry the entry's sign (a negative entry's digits are negated), so
// the residue GEMM yields signed residues directly.
struct DigitArgs {
    const uint32_t *limbs;
    const int32_t *sizes;  // sizes[r * rs + c]: the entry's sign
    int64_t ld, rs;
    int32_t rows, cols, nlimbs;
    int32_t transpose;  // 0: out row r*cols + c ; 1: out row c*rows + r
    int32_t dxp;        // digits per out row (multiple of 64)
    __nv_bfloat16 *out;
};

// BAL: balanced digits.  s[entry][li - LO] holds limb l0 + li for li >= LO; with
// balanced digits LO = -1, so slot 0 holds limb l0 - 1 (its top byte carries into the
// chunk's first digit).  Rows of 65 and 67 words keep the column loads conflict-free.
// Digit rows of the 4 x 32 entries at block (bx, by), 64-limb chunk bz, by 256 threads.
template <bool BAL>
__device__ __forceinline__ void digits_block(const DigitArgs &a, int bx, int by, int bz) {
    __shared__ uint32_t s[128][BAL ? 67 : 65];
    __shared__ uint32_t sflip[128];  // 0x80008000 for a negative entry: flips both bf16 signs of a word
    const int tr = 4, tcn = 32;
    const int r0 = by * tr, c0 = bx * tcn;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < 128) {
        const int r = r0 + (threadIdx.x >> 5), c = c0 + (threadIdx.x & 31);
        sflip[threadIdx.x] = (r < a.rows && c < a.cols && a.sizes[(int64_t)r * a.rs + c] < 0) ? 0x80008000u : 0u;
    }
    {
        // one chunk of 64 limbs per block (blockIdx.z): more, shorter blocks keep the
        // last wave of the grid small
        const int l0 = bz * 64;
        // load limbs [l0 - 1, l0 + 64) of the 4 x 32 entries, coalesced along c: slot
        // 1 + li holds limb l0 + li, slot 0 limb l0 - 1 (its top byte carries into the
        // chunk's first digit)
        constexpr int LO = BAL ? -1 : 0;  // first limb loaded, relative to l0
        for (int q = threadIdx.x; q < (64 - LO) * 128; q += 256) {
            int cc = q & 31, rr = (q >> 5) & 3, li = (q >> 7) + LO;
            int r = r0 + rr, c = c0 + cc, l = l0 + li;
            uint32_t v = 0;
            if (r < a.rows && c < a.cols && l >= 0 && l < a.nlimbs) v = a.limbs[(int64_t)l * a.ld + (int64_t)r * a.rs + c];
            s[rr * 32 + cc][li - LO] = v;
        }
        __syncthreads();
        // each warp writes whole digit rows: lane j -> limbs l0+2j, l0+2j+1 (8 digits, 16 bytes)
        for (int ent = warp; ent < 128; ent += 8) {
            int rr = ent >> 5, cc = ent & 31;
            int r = r0 + rr, c = c0 + cc;
            if (r >= a.rows || c >= a.cols) continue;
            int64_t row = a.transpose ? (int64_t)c * a.rows + r : (int64_t)r * a.cols + c;
            int dg = 4 * (l0 + 2 * lane);
            if (dg >= a.dxp) continue;
            const uint32_t flip = sflip[ent];
            uint4 pk;
            if (BAL) {
                const uint32_t vp = s[ent][2 * lane], v0 = s[ent][2 * lane + 1], v1 = s[ent][2 * lane + 2];
                float d0[4], d1[4];
                limb_digits_bal(v0, vp >> 31, false, d0);
                limb_digits_bal(v1, v0 >> 31, dg + 8 == a.dxp, d1);
                pk.x = bf16x2_bits(d0[0], d0[1]) ^ flip;
                pk.y = bf16x2_bits(d0[2], d0[3]) ^ flip;
                pk.z = bf16x2_bits(d1[0], d1[1]) ^ flip;
                pk.w = bf16x2_bits(d1[2], d1[3]) ^ flip;
            } else {
                const uint32_t v0 = s[ent][2 * lane], v1 = s[ent][2 * lane + 1];
                pk.x = byte_pair_bf16(v0, 0) ^ flip;
                pk.y = byte_pair_bf16(v0, 2) ^ flip;
                pk.z = byte_pair_bf16(v1, 0) ^ flip;
                pk.w = byte_pair_bf16(v1, 2) ^ flip;
            }
            *reinterpret_cast<uint4 *>(a.out + row * a.dxp + dg) = pk;
        }
    }
}

}  // namespace gbmm
