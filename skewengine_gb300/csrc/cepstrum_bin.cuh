// The cepstrum of a 64-sample window in float with a bound on its error, and from
// it the 1000-wide bin of the reference's output (lineCepstrum,
// src/kernelBLUR.h:153-228 -> getBlurParameter2 :88-110) where that is proven.
//
//  * Windows with all 64 cells inside the row lose their centre cell's value
//    first: only X_0 depends on the mean, and a smaller window makes every bound
//    smaller.
//  * X is off, as a vector, by at most 240 u |window| (u = 2^-24, Euclidean
//    norms): the transform is sqrt(32) times a unitary one, and its stages are
//    off by u (two stages of plain additions), 5.8 u (three of fused
//    butterflies), 8 u (the real-input split) and u (the subtraction) of their
//    norm, 29 u together; X_0 takes another sqrt(2).
//  * log |X_n|^2 is off by at most 2.2 |dX_n| / |X_n| while that is below 0.05,
//    the sum over n by Cauchy's inequality by 2.2 |dX| (sum of 1 / |X_n|^2)^1/2;
//    the logarithm itself by 2^-22 max(1, |log2|); log |X_n|^2 + log |X_{32-n}|^2
//    is the logarithm of the product, 17 logarithms instead of 32.
//  * Scaling X by a constant only moves c_0, which nothing reads.
//  * c_4 .. c_15 are cosine sums folded over n, 16 - n and 8 - n: 62
//    multiply-adds; their roundings stay below 14 u times the sum of the logs.
//  * The search is repeated for every sample that could be the first ascent;
//    the cell is decided when all of them land in one bin with the bound to
//    spare.
//  * cepstrum_f32, the float32 mode's own evaluation, is off by as much from the
//    window with its mean (kPlain): 30 u sqrt(32) |window| for its transform, whose
//    butterflies round three times (5 u a stage), and 24 u times the sum of its
//    logarithms for logf, the sums' additions and coefficients.  A bin that leaves
//    room for both errors is the bin it arrives at.
#pragma once

#include "kernels.h"

namespace ske {

// cos(2 pi k / 64) for any k, folded to a compile-time constant.
__device__ __forceinline__ constexpr float cos64(int k) {
    constexpr float c[17] = {1.0f, 0.995184727f, 0.98078528f, 0.956940336f, 0.923879533f, 0.881921264f, 0.831469612f, 0.773010453f, 0.707106781f, 0.634393284f, 0.555570233f, 0.471396737f, 0.382683432f, 0.290284677f, 0.195090322f, 0.0980171403f, 0.0f};
    k &= 63;
    k = k > 32 ? 64 - k : k;
    return k > 16 ? -c[32 - k] : c[k];
}
__device__ __forceinline__ constexpr float sin64(int k) { return cos64(k - 16); }

__device__ __forceinline__ constexpr int brev5(int v) {
    return ((v & 1) << 4) | ((v & 2) << 2) | (v & 4) | ((v & 8) >> 2) | ((v & 16) >> 4);
}

// 32-point complex FFT in registers, radix-2 decimation in time: input in
// bit-reversed order, output in natural order.  A butterfly's sum takes four
// fused operations and its difference 2a - sum two.
__device__ __forceinline__ void fft32_fused(float (&re)[32], float (&im)[32]) {
#pragma unroll
    for (int span = 1; span < 32; span <<= 1) {
#pragma unroll
        for (int start = 0; start < 32; start += 2 * span) {
#pragma unroll
            for (int k = 0; k < span; k++) {
                const int a = start + k, b = a + span;
                const float ar = re[a], ai = im[a], br = re[b], bi = im[b];
                if (k == 0) {
                    re[a] = __fadd_rn(ar, br);
                    im[a] = __fadd_rn(ai, bi);
                    re[b] = __fsub_rn(ar, br);
                    im[b] = __fsub_rn(ai, bi);
                } else if (2 * k == span) {  // twiddle -i
                    re[a] = __fadd_rn(ar, bi);
                    im[a] = __fsub_rn(ai, br);
                    re[b] = __fsub_rn(ar, bi);
                    im[b] = __fadd_rn(ai, br);
                } else {
                    const float c = cos64(k * (32 / span)), s = sin64(k * (32 / span));  // twiddle c - i s
                    re[a] = __fmaf_rn(br, c, __fmaf_rn(bi, s, ar));
                    im[a] = __fmaf_rn(bi, c, __fmaf_rn(br, -s, ai));
                    re[b] = __fmaf_rn(2.0f, ar, -re[a]);
                    im[b] = __fmaf_rn(2.0f, ai, -im[a]);
                }
            }
        }
    }
}

__device__ __forceinline__ float lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The bin of the 64-sample window w[0..63], or -1 where float leaves it open.
// mean: the window's centre sample where every sample lies inside the row, else 0.
// kPlain: the bin cepstrum_f32 (k_cepstrum_f32.cu) arrives at, not the reference's.
template <bool kPlain>
__device__ __forceinline__ float cepstrum_bin(const float* __restrict__ w, float mean) {
    constexpr float u = 5.9604644775390625e-8f;  // 2^-24
    float re[32], im[32], l2 = 0.0f;
#pragma unroll
    for (int n = 0; n < 32; n++) {  // z_n = w[2n] + i w[2n+1], stored bit-reversed
        const float a = __fsub_rn(w[2 * n], mean), c = __fsub_rn(w[2 * n + 1], mean);
        re[brev5(n)] = a;
        im[brev5(n)] = c;
        l2 = __fmaf_rn(a, a, l2);
        l2 = __fmaf_rn(c, c, l2);
    }
    fft32_fused(re, im);
    // 2 X_k = E + W64^k O, E = Z_k + conj Z_{32-k}, O = -i (Z_k - conj Z_{32-k});
    // 2 X_{32-k} = conj(E - W64^k O).  e[n] = log2 |2 X_n|^2 |2 X_{32-n}|^2, inv =
    // sum of 1 / |2 X_n|^2, all: of the logs' magnitudes.
    float e[17], inv = 0.0f, all = 0.0f;
    {
        const float x0 = __fmaf_rn(128.0f, mean, __fmul_rn(2.0f, __fadd_rn(re[0], im[0])));
        const float p0 = __fmul_rn(x0, x0);
        const float p16 = __fmul_rn(4.0f, __fmaf_rn(re[16], re[16], __fmul_rn(im[16], im[16])));
        e[0] = lg2(p0);
        e[16] = lg2(p16);
        inv = rcp(p0) + rcp(p16);
        all = fabsf(e[0]) + fabsf(e[16]);
    }
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const int m = 32 - k;
        const float er = __fadd_rn(re[k], re[m]), ei = __fsub_rn(im[k], im[m]);
        const float orr = __fadd_rn(im[k], im[m]), oi = __fsub_rn(re[m], re[k]);
        const float c = cos64(k), s = sin64(k);
        const float ur = __fmaf_rn(orr, c, __fmaf_rn(oi, s, er)), ui = __fmaf_rn(oi, c, __fmaf_rn(orr, -s, ei));
        const float vr = __fmaf_rn(2.0f, er, -ur), vi = __fmaf_rn(2.0f, ei, -ui);
        const float pk = __fmaf_rn(ur, ur, __fmul_rn(ui, ui)), pm = __fmaf_rn(vr, vr, __fmul_rn(vi, vi));
        e[k] = lg2(__fmul_rn(pk, pm));
        inv += rcp(pk);
        inv += rcp(pm);
        all += fabsf(e[k]);
    }
    // T_k = e_0 + (-1)^k e_16 + sum over 0 < n < 16 of e_n cos(2 pi k n / 32); c_k = T_k ln 2 / sqrt(32).
    constexpr float kScale = 0.12253274f;
    float c[16];
    float f[8], o[8];
#pragma unroll
    for (int n = 1; n < 8; n++) {
        f[n] = __fadd_rn(e[n], e[16 - n]);
        o[n] = __fsub_rn(e[n], e[16 - n]);
    }
    const float odd = __fsub_rn(e[0], e[16]), sum = __fadd_rn(e[0], e[16]);
    const float ev = __fadd_rn(sum, e[8]), eo = __fsub_rn(sum, e[8]);
#pragma unroll
    for (int k = 5; k < 16; k += 2) {
        float acc = odd;
#pragma unroll
        for (int n = 1; n < 8; n++) acc = __fmaf_rn(o[n], cos64(2 * k * n), acc);
        c[k] = acc;
    }
    float g[4], h[4];
#pragma unroll
    for (int n = 1; n < 4; n++) {
        g[n] = __fadd_rn(f[n], f[8 - n]);
        h[n] = __fsub_rn(f[n], f[8 - n]);
    }
#pragma unroll
    for (int k = 6; k < 16; k += 4) {
        float acc = eo;
#pragma unroll
        for (int n = 1; n < 4; n++) acc = __fmaf_rn(h[n], cos64(2 * k * n), acc);
        c[k] = acc;
    }
#pragma unroll
    for (int k = 4; k < 16; k += 4) {
        float acc = k == 8 ? __fadd_rn(ev, f[4]) : __fsub_rn(ev, f[4]);
#pragma unroll
        for (int n = 1; n < 4; n++) acc = __fmaf_rn(g[n], cos64(2 * k * n), acc);
        c[k] = acc;
    }
    // The bound of every c_k: 0.17678 = 1 / sqrt(32); 2 X is off by 480 u |window|.
    const float dx = 481.0f * u * sqrtf(l2 * inv);
    float err = 0.17678f * (2.2f * dx + 0.7f * (4.0f * u * (17.0f + all) + 14.0f * u * all)) + 100.0f * u;
    float far = dx;
    if (kPlain) {
        const float norm = sqrtf(l2) + 8.0f * fabsf(mean);  // of the window as it is, at most
        far = 481.0f * u * norm * sqrtf(inv);
        // Every |2 X_n|^2 lies between 1 / inv and 256 norm^2; the other's logarithms are of |X_n / 8|^2.
        const float logs = fmaxf(fabsf(lg2(256.0f * norm * norm)), fabsf(lg2(inv))) + 9.0f;
        err += 0.17678f * (2.2f * far + 24.0f * u * 32.0f * 0.7f * logs) + 100.0f * u;
    }
    float s[16], top = 0.0f;
#pragma unroll
    for (int k = 15; k >= 4; k--) {
        c[k] = __fmul_rn(c[k], kScale);
        s[k] = fmaxf(-c[k], 0.0f);
    }
    // Samples after i: top.  Every sample i that may be the first ascent gives
    // the result max(s_{i-1}, top_i); lo and hi span those up to the first that
    // must be one (going down: a sure ascent discards what lies after it).
    float lo = 0.0f, hi = 0.0f;  // no ascent at all
#pragma unroll
    for (int i = 15; i >= 5; i--) {
        const float rise = s[i] - s[i - 1];
        const float best = fmaxf(s[i - 1], top);
        const bool may = rise > -2.0f * err && !(c[i] > err), must = rise > 2.0f * err;
        lo = may ? (must ? best : fminf(lo, best)) : lo;
        hi = may ? (must ? best : fmaxf(hi, best)) : hi;
        top = fmaxf(top, s[i]);
    }
    const float slack = err + 8.0f * u * hi;
    const float b0 = floorf(10.0f * fmaxf(lo - slack, 0.0f)), b1 = floorf(10.0f * (hi + slack));
    const bool sure = b0 == b1 && far < 0.05f && all < 1e4f && l2 > 1e-20f && l2 < 1e24f;
    return sure ? b0 : -1.0f;
}

}  // namespace ske
