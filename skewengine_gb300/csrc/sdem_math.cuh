// Arithmetic shared by the total-viewshed sweeps (k_sweep.cu, k_sdem.cu).
#pragma once

#include "f32x2.cuh"
#include "kernels.h"

namespace ske {

constexpr int kFastMaxRow = 4096;  // step table entries; exact ring sums up to rows of this length

// Division.  The quotient (S[k]-h)/d must be the correctly rounded one, because
// visibility compares it strictly against the running maximum: q0 = RN(a*y),
// r = fma(q0, -d, a), q = fma(r, y, q0) with y = RN(1/d) (Markstein's correction
// step, P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. R&D 34(1), 1990).  It is applied only to rows
// whose values lie in a range where it is exact for every d <= 4095 (checked
// exhaustively against IEEE division by ske_selftest_division); other rows take
// the IEEE-division path.

// Values for which the Markstein quotient is exact: zero, or finite with
// magnitude in [2^-80, 2^90].  If S[k] and h both qualify, a = S[k]-h is zero or
// has magnitude in [2^-103, 2^91].
__device__ __forceinline__ bool div_safe(float v) {
    const float m = fabsf(v);
    return v == 0.0f || (m >= 8.271806125530277e-25f && m <= 1.2379400392853803e27f);
}

__device__ __forceinline__ float div_fast(float a, float negd, float y) {
    const float q0 = __fmul_rn(a, y);
    const float r = __fmaf_rn(q0, negd, a);
    return __fmaf_rn(r, y, q0);
}

// Both halves of a/d correctly rounded (div_fast on each half).
__device__ __forceinline__ f2 div2(f2 a, f2 negd, f2 y) {
    const f2 q0 = mul2(a, y);
    return fma2(fma2(q0, negd, a), y, q0);
}

struct Item {
    int slot, row, chunk;
};

__device__ __forceinline__ Item decode(uint64_t it) {
    Item r;
    r.slot = (int)(it >> 48);
    r.row = (int)((it >> 16) & 0xffffffffu);
    r.chunk = (int)(it & 0xffffu);
    return r;
}

// Reference-order path (kernelSDEM.h:180-218 step for step): IEEE division,
// std::max horizon update, cv accumulated in float forward then backward.
static __device__ float scan_reference(const float* __restrict__ A, int x, int L, float povh) {
    const float h = __fadd_rn(A[x], povh);
    float cv = 0.0f;
    for (int dir = 1; dir >= -1; dir -= 2) {
        float mx = -2000.0f, opened = 0.0f;
        bool vis = true;
        const int n = dir > 0 ? L - 1 - x : x;
        for (int s = 1; s <= n; s++) {
            const float d = (float)s;
            const float sl = __fdiv_rn(__fsub_rn(A[x + dir * s], h), d);
            const bool above = sl > mx;
            const bool opening = above && !vis;
            const bool closing = !above && vis;
            vis = above;
            mx = (sl < mx) ? mx : sl;
            if (opening) opened = d;
            if (closing) cv = __fadd_rn(cv, __fsub_rn(__fmul_rn(d, d), __fmul_rn(opened, opened)));
        }
    }
    return cv;
}

}  // namespace ske
