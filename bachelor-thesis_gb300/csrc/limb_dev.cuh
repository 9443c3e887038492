// Device-side matrix views shared by the limb-form kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "gbmm_internal.h"

namespace gbmm {

__device__ __forceinline__ int iabs_d(int x) { return x < 0 ? -x : x; }

struct MatArgs {
    uint32_t *limbs;
    int32_t *sizes;
    int64_t rs, ld;
    int32_t rows, cols, nlimbs;
};
__host__ __device__ static inline MatArgs margs(const gbmm_mat &m) {
    MatArgs a;
    a.limbs = m.limbs; a.sizes = m.sizes; a.rs = m.rs; a.ld = m.ld;
    a.rows = m.rows; a.cols = m.cols; a.nlimbs = m.nlimbs;
    return a;
}

// Views of Winograd's breadth-first tree (its layout: limb.cu).
__device__ __forceinline__ MatArgs wt_quad(MatArgs m, int qr, int qc, int h) {
    const int64_t off = (int64_t)qr * h * m.rs + (int64_t)qc * h;
    m.limbs += off;
    m.sizes += off;
    m.rows = h;
    m.cols = h;
    return m;
}
__device__ __forceinline__ MatArgs wt_dense(uint32_t *limbs, int32_t *sizes, int64_t q, int h, int cap) {
    MatArgs m;
    const int64_t e = (int64_t)h * h;
    m.limbs = limbs + q * e * cap;
    m.sizes = sizes + q * e;
    m.rs = h;
    m.ld = e;
    m.rows = h;
    m.cols = h;
    m.nlimbs = cap;
    return m;
}
// Operand `which` (0: A, 1: B) of node `node` at level d.
__device__ __forceinline__ MatArgs wt_operand(const WinoTree &t, int which, int d, int64_t node) {
    MatArgs v = margs(which ? t.B : t.A);
    int h = t.N;
    int64_t pw = 1;
    for (int l = 1; l < d; l++) pw *= 7;
    for (int l = 1; l <= d; l++) {
        const int64_t self = node / pw;  // this node's ancestor at level l
        const int j = (int)(self % 7);
        const int64_t parent = self / 7;
        h >>= 1;
        int s = -1;
        if (which == 0) {
            if (j == 0) v = wt_quad(v, 0, 0, h);
            else if (j == 1) v = wt_quad(v, 0, 1, h);
            else if (j == 3) v = wt_quad(v, 1, 1, h);
            else s = j == 2 ? 3 : j - 4;
        } else {
            if (j == 0) v = wt_quad(v, 0, 0, h);
            else if (j == 1) v = wt_quad(v, 1, 0, h);
            else if (j == 2) v = wt_quad(v, 1, 1, h);
            else s = j == 3 ? 3 : j - 4;
        }
        if (s >= 0)
            v = which ? wt_dense(t.sb_limbs[l], t.sb_sizes[l], 4 * parent + s, h, t.capSB)
                      : wt_dense(t.sa_limbs[l], t.sa_sizes[l], 4 * parent + s, h, t.capSA);
        pw /= 7;
    }
    return v;
}

}  // namespace gbmm
