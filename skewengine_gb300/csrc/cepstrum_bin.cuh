// The cepstrum of a 64-sample window in float with a bound on its error, and from
// it the 1000-wide bin of the reference's output (lineCepstrum,
// src/kernelBLUR.h:153-228 -> getBlurParameter2 :88-110) where that is proven.
//
//  * Windows with all 64 cells inside the row lose their centre cell's value
//    first: only X_0 depends on the mean, and a smaller window makes every bound
//    smaller.
//  * X is off, as a vector, by at most 162 u |window| (u = 2^-24, Euclidean
//    norms): the transform is sqrt(32) times a unitary one, and each stage is off
//    by a share of its norm.  The subtraction and two stages of plain additions:
//    u each.  A fused butterfly of a and b, n = (|a|^2 + |b|^2)^1/2: its inner
//    operations u (|a| + |b|), its constant u |b|, the outer one u |sum|, and the
//    difference 2a - sum all of that and u |difference|; over both outputs, of norm
//    sqrt(2) n, 5^1/2 u from the first two and ((3 + 5^1/2) / 2)^1/2 u from the
//    roundings of the outputs, 3.86 u (three stages).  The real-input split: the
//    same and sqrt(2) u for its two sums, 5.27 u.  Together 19.9 u, 20.3 u with the
//    terms in u^2; X_0 takes another sqrt(2).
//  * log |X_n|^2 is off by at most 2.1 |dX_n| / |X_n| while that is below 0.05,
//    the sum over n by Cauchy's inequality by 2.1 |dX| (sum of 1 / |X_n|^2)^1/2;
//    the logarithm itself by 2^-22 max(1, |log2|); log |X_n|^2 + log |X_{32-n}|^2
//    is the logarithm of the product, 17 logarithms instead of 32.
//  * Scaling X by a constant only moves c_0, which nothing reads.
//  * 1 / |X_n|^2 + 1 / |X_{32-n}|^2 is their sum times the reciprocal of their
//    product, whose logarithm is formed anyway; |window|^2 comes from the spectrum
//    (Parseval), off by 10^-5 of itself against the 3 10^-3 the bound has to spare.
//  * A thread evaluates two windows in the halves of f32x2 registers, from samples
//    staged as such pairs: the transform and the sums take the instructions of one
//    (a 512 x 512 texture, 180 angles: 2.2 ms with one window a thread, 1.86 with two).
//    What is left to the FMA pipe is the same, and it is the bound now (f32x2 occupies
//    it for two cycles).
//  * c_4 .. c_15 are cosine sums folded over n, 16 - n and 8 - n: 62
//    multiply-adds; their roundings stay below 14 u times the sum of the logs, at most 17
//    times the largest.
//  * The search is repeated for every sample that could be the first ascent;
//    the cell is decided when all of them land in one bin with the bound to
//    spare.
//  * cepstrum_f32, the float32 mode's own evaluation, is off by as much from the
//    window with its mean (kPlain): 172 u |window| for its transform, whose
//    butterflies are off by 5^1/2 u |b| in the product, u |b| in its constant and u
//    in each sum, 4.25 u a stage (the second stage 2 u), whose split is off by 5.36
//    u in the same way, 21.1 u together, 21.5 u with the rest; and 24 u times the sum of its
//    logarithms for logf, the sums' additions and coefficients.  A bin that leaves
//    room for both errors is the bin it arrives at.
#pragma once

#include "f32x2.cuh"
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

// The same constant in both halves.
__device__ __forceinline__ f2 both(float c) { return pk(c, c); }

// A packed pair stored as itself or as its negative (neg, known at compile time
// once the loops are unrolled): f32x2 operations take no negated operands, and a
// sign that only moves on to the next constant or from an addition to a
// subtraction costs nothing.
struct Signed {
    f2 v;
    bool neg;
};
__device__ __forceinline__ Signed operator-(Signed a) { return {a.v, !a.neg}; }
__device__ __forceinline__ Signed operator+(Signed a, Signed b) {
    if (a.neg == b.neg) return {add2(a.v, b.v), a.neg};
    return a.neg ? Signed{sub2(b.v, a.v), false} : Signed{sub2(a.v, b.v), false};
}
__device__ __forceinline__ Signed operator-(Signed a, Signed b) { return a + -b; }
// acc + x * c.
__device__ __forceinline__ Signed mad(Signed x, float c, Signed acc) {
    return {fma2(x.v, both(x.neg == acc.neg ? c : -c), acc.v), acc.neg};
}

// 32-point complex FFT in registers of two windows at a time, radix-2 decimation
// in time: input in bit-reversed order, output in natural order.  A butterfly's
// sum takes four fused operations and its difference 2a - sum two.
__device__ __forceinline__ void fft32_fused(Signed (&re)[32], Signed (&im)[32]) {
#pragma unroll
    for (int span = 1; span < 32; span <<= 1) {
#pragma unroll
        for (int start = 0; start < 32; start += 2 * span) {
#pragma unroll
            for (int k = 0; k < span; k++) {
                const int a = start + k, b = a + span;
                const Signed ar = re[a], ai = im[a], br = re[b], bi = im[b];
                if (k == 0) {
                    re[a] = ar + br;
                    im[a] = ai + bi;
                    re[b] = ar - br;
                    im[b] = ai - bi;
                } else if (2 * k == span) {  // twiddle -i
                    re[a] = ar + bi;
                    im[a] = ai - br;
                    re[b] = ar - bi;
                    im[b] = ai + br;
                } else {
                    const float c = cos64(k * (32 / span)), s = sin64(k * (32 / span));  // twiddle c - i s
                    re[a] = mad(br, c, mad(bi, s, ar));
                    im[a] = mad(bi, c, mad(br, -s, ai));
                    re[b] = -mad(ar, -2.0f, re[a]);
                    im[b] = -mad(ai, -2.0f, im[a]);
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

// The search for one window: its bin, or -1 where float leaves it open.
// c: its c_4 .. c_15.  l2, inv, emax: |window|^2, the sum of 1 / |2 X_n|^2 and the
// largest of the logarithms' magnitudes.
template <bool kPlain>
__device__ __forceinline__ float cepstrum_decide(const float (&c)[16], float l2, float inv, float emax, float mean) {
    constexpr float u = 5.9604644775390625e-8f;  // 2^-24
    // The bound of every c_k: 0.17678 = 1 / sqrt(32); 2 X is off by 324 u |window|.
    const float all = 17.0f * emax;  // bounds the sum of the logs' magnitudes
    const float dx = 325.0f * u * sqrtf(l2 * inv);
    float err = 0.17678f * (2.1f * dx + 0.7f * (4.0f * u * (17.0f + all) + 14.0f * u * all)) + 100.0f * u;
    float far = dx;
    if (kPlain) {
        const float norm = sqrtf(l2) + 8.0f * fabsf(mean);  // of the window as it is, at most
        far = 345.0f * u * norm * sqrtf(inv);
        // Every |2 X_n|^2 lies between 1 / inv and 256 norm^2; the other's logarithms are of |X_n / 8|^2.
        const float logs = fmaxf(fabsf(lg2(256.0f * norm * norm)), fabsf(lg2(inv))) + 9.0f;
        err += 0.17678f * (2.1f * far + 24.0f * u * 32.0f * 0.7f * logs) + 100.0f * u;
    }
    float s[16], top = 0.0f;
#pragma unroll
    for (int k = 15; k >= 4; k--) s[k] = fmaxf(-c[k], 0.0f);
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
    // Logarithms below 126: no product |2 X_n|^2 |2 X_{32-n}|^2 and no reciprocal left the float range.
    const bool sure = b0 == b1 && far < 0.05f && emax < 126.0f && l2 > 1e-20f && l2 < 1e24f;
    return sure ? b0 : -1.0f;
}

// The bins of two 64-sample windows, the halves of w[0..63], or -1 where float
// leaves one open.  mean: each window's centre sample where all of its samples lie
// inside its row, else 0.
// kPlain: the bin cepstrum_f32 (k_cepstrum_f32.cu) arrives at, not the reference's.
template <bool kPlain>
__device__ __forceinline__ float2 cepstrum_bin(const f2* __restrict__ w, f2 mean) {
    Signed re[32], im[32];
#pragma unroll
    for (int n = 0; n < 32; n++) {  // z_n = w[2n] + i w[2n+1], stored bit-reversed
        re[brev5(n)] = {sub2(w[2 * n], mean), false};
        im[brev5(n)] = {sub2(w[2 * n + 1], mean), false};
    }
    fft32_fused(re, im);
    // 2 X_k = E + W64^k O, E = Z_k + conj Z_{32-k}, O = -i (Z_k - conj Z_{32-k});
    // 2 X_{32-k} = conj(E - W64^k O).  e[n] = log2 |2 X_n|^2 |2 X_{32-n}|^2, inv =
    // sum of 1 / |2 X_n|^2, e_max: the largest of the logs' magnitudes.
    // Parseval: 256 |window|^2 = |2 X_0|^2 + |2 X_32|^2 + 2 sum over 0 < n < 32 of |2 X_n|^2, X_0 without the mean.
    f2 e[17], inv, pw;
    float e_max0, e_max1;
    const f2 two = both(2.0f), four = both(4.0f);
    {
        const Signed z0 = re[0] + im[0];
        const f2 y0 = mul2(both(z0.neg ? -2.0f : 2.0f), z0.v), y32 = mul2(two, (re[0] - im[0]).v);
        const f2 x0 = fma2(both(128.0f), mean, y0);
        const f2 p0 = mul2(x0, x0);
        const f2 p16 = mul2(four, fma2(re[16].v, re[16].v, mul2(im[16].v, im[16].v)));
        float a, b, c, d;
        upk(p0, a, b);
        upk(p16, c, d);
        inv = pk(rcp(a) + rcp(c), rcp(b) + rcp(d));
        a = lg2(a), b = lg2(b), c = lg2(c), d = lg2(d);
        e[0] = pk(a, b);
        e[16] = pk(c, d);
        e_max0 = fmaxf(fabsf(a), fabsf(c));
        e_max1 = fmaxf(fabsf(b), fabsf(d));
        pw = fma2(two, p16, fma2(y0, y0, mul2(y32, y32)));
    }
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const int m = 32 - k;
        const Signed er = re[k] + re[m], ei = im[k] - im[m], orr = im[k] + im[m], oi = re[m] - re[k];
        const float c = cos64(k), s = sin64(k);
        const Signed ur = mad(orr, c, mad(oi, s, er)), ui = mad(oi, c, mad(orr, -s, ei));
        const f2 vr = mad(er, -2.0f, ur).v, vi = mad(ei, -2.0f, ui).v;
        const f2 pu = fma2(ur.v, ur.v, mul2(ui.v, ui.v)), pv = fma2(vr, vr, mul2(vi, vi));
        const f2 prod = mul2(pu, pv), sum = add2(pu, pv);
        float a, b;
        upk(prod, a, b);
        inv = fma2(sum, pk(rcp(a), rcp(b)), inv);  // 1 / pu + 1 / pv
        a = lg2(a), b = lg2(b);
        e[k] = pk(a, b);
        e_max0 = fmaxf(e_max0, fabsf(a));
        e_max1 = fmaxf(e_max1, fabsf(b));
        pw = fma2(two, sum, pw);
    }
    // T_k = e_0 + (-1)^k e_16 + sum over 0 < n < 16 of e_n cos(2 pi k n / 32); c_k = T_k ln 2 / sqrt(32).
    constexpr float kScale = 0.12253274f;
    f2 c[16];
    f2 f[8], o[8];
#pragma unroll
    for (int n = 1; n < 8; n++) {
        f[n] = add2(e[n], e[16 - n]);
        o[n] = sub2(e[n], e[16 - n]);
    }
    const f2 odd = sub2(e[0], e[16]), sum = add2(e[0], e[16]);
    const f2 ev = add2(sum, e[8]), eo = sub2(sum, e[8]);
#pragma unroll
    for (int k = 5; k < 16; k += 2) {
        f2 acc = odd;
#pragma unroll
        for (int n = 1; n < 8; n++) acc = fma2(o[n], both(cos64(2 * k * n)), acc);
        c[k] = acc;
    }
    f2 g[4], h[4];
#pragma unroll
    for (int n = 1; n < 4; n++) {
        g[n] = add2(f[n], f[8 - n]);
        h[n] = sub2(f[n], f[8 - n]);
    }
#pragma unroll
    for (int k = 6; k < 16; k += 4) {
        f2 acc = eo;
#pragma unroll
        for (int n = 1; n < 4; n++) acc = fma2(h[n], both(cos64(2 * k * n)), acc);
        c[k] = acc;
    }
#pragma unroll
    for (int k = 4; k < 16; k += 4) {
        f2 acc = k == 8 ? add2(ev, f[4]) : sub2(ev, f[4]);
#pragma unroll
        for (int n = 1; n < 4; n++) acc = fma2(g[n], both(cos64(2 * k * n)), acc);
        c[k] = acc;
    }
    float c0[16], c1[16];
#pragma unroll
    for (int k = 4; k < 16; k++) upk(mul2(c[k], both(kScale)), c0[k], c1[k]);
    const f2 l2 = mul2(pw, both(1.0f / 256.0f));
    float l20, l21, inv0, inv1, m0, m1;
    upk(l2, l20, l21);
    upk(inv, inv0, inv1);
    upk(mean, m0, m1);
    return make_float2(cepstrum_decide<kPlain>(c0, l20, inv0, e_max0, m0),
                       cepstrum_decide<kPlain>(c1, l21, inv1, e_max1, m1));
}

}  // namespace ske
