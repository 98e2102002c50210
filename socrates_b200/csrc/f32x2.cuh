// Two-wide float32 arithmetic (retention and selective scan; gemm_f32.cu and linear_recurrence.cu have their own forms) and the
// register-tile steps of the retention kernels.
#pragma once

#include <stdint.h>

namespace sb {

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pair(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ unsigned long long twice(float x) { return pair(x, x); }
__device__ __forceinline__ float low(unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float high(unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }

// acc += x y^T for one step of the contraction: 8 rows (x[0..3] and x[32..35], as 4 pairs) by 4 NC columns (y[64 h + 0..3]).
// PAIR0: the first pair of rows that takes part (2: the second four rows alone).
template <int NC, int PAIR0>
__device__ __forceinline__ void tile_step(unsigned long long (&acc)[4][4 * NC], const float* x, const float* y) {
    unsigned long long xs[4];
    if (PAIR0 == 0) *reinterpret_cast<ulonglong2*>(xs) = *reinterpret_cast<const ulonglong2*>(x);
    *reinterpret_cast<ulonglong2*>(xs + 2) = *reinterpret_cast<const ulonglong2*>(x + 32);
#pragma unroll
    for (int h = 0; h < NC; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(y + 64 * h);
        const float ys[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned long long yy = twice(ys[j]);
#pragma unroll
            for (int p = PAIR0; p < 4; ++p) fma2(acc[p][4 * h + j], xs[p], yy);
        }
    }
}

// tile_step for a y that rows `from` and later of a group of four take: of the first group (PAIR0 0, the second takes it whole) or
// of the second (PAIR0 2).  The others, whose x is zero, get a zero for it, whatever y is.
template <int NC, int PAIR0>
__device__ __forceinline__ void tile_step_from(unsigned long long (&acc)[4][4 * NC], const float* x, const float* y, int from) {
    unsigned long long xs[4];
    if (PAIR0 == 0) *reinterpret_cast<ulonglong2*>(xs) = *reinterpret_cast<const ulonglong2*>(x);
    *reinterpret_cast<ulonglong2*>(xs + 2) = *reinterpret_cast<const ulonglong2*>(x + 32);
#pragma unroll
    for (int h = 0; h < NC; ++h) {
        const float4 v = *reinterpret_cast<const float4*>(y + 64 * h);
        const float ys[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned long long yy = twice(ys[j]);
            fma2(acc[PAIR0][4 * h + j], xs[PAIR0], pair(from <= 0 ? ys[j] : 0.f, from <= 1 ? ys[j] : 0.f));
            fma2(acc[PAIR0 + 1][4 * h + j], xs[PAIR0 + 1], pair(from <= 2 ? ys[j] : 0.f, from <= 3 ? ys[j] : 0.f));
#pragma unroll
            for (int p = PAIR0 + 2; p < 4; ++p) fma2(acc[p][4 * h + j], xs[p], yy);
        }
    }
}

}  // namespace sb
