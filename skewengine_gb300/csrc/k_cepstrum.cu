// Cepstrum motion-blur estimation (kernelBLUR, src/kernelBLUR.h:267-302 ->
// lineCepstrum :153-228 -> select_subarray :69-85, getBlurParameter2 :88-110).
//
// For every valid skewed cell j of row r: a 64-cell window of the row centred at
// j (cells outside [first, last) are zero; the effective window is 64 because
// kernelRADN.h:19 wins the shared KERNELCOMMONS guard), X = FFT(window)/8,
// c = FFT(log|X_k|^2, k < 32)/sqrt(32), s_k = -min(0, Re c_k) for k < 16, and
// the output is (float)(10000 * peak(s)).
//
// Exact values (k_cepstrum): one warp per cell: the window lives in shared memory as complex doubles and
// each lane performs one butterfly per stage of the reference radix-2
// decimation-in-frequency FFT (helper.h:59-106) with the reference's twiddle
// sequence, in binary64 without fused operations; cells whose FFT input is
// finite use warp_fft_real (same values up to the sign of zeros, which the
// outputs cannot see).  The logarithm is CUDA's double-precision log().
//
// Bins (k_cepstrum_bins): a whole run only ever deskews the values with the
// reference's max+angle encoding, angle + 1000*(int)(v/1000) (skewEngine.cuh:
// 774-785), which sees the 1000-wide bin of a value and nothing else of it.
// GB300 does 1/64 as many binary64 as float operations, and the exact kernel
// held a 512 x 512 image at the FP64 pipe's rate (353 ms for 180 angles, that
// pipe 84% busy).  So the cepstrum is formed in float with a bound on its error
// (one thread per cell, the window in registers), and only the cells whose bin
// that leaves open run the exact kernel.  The whole run of a 512 x 512 texture
// (180 angles): 353.3 ms with every cell in binary64, 3.20 ms so (the float
// kernel 2.2, the open cells 0.6).
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
#include "kernels.h"

namespace ske {

namespace {

constexpr int kWin = kBlurWindow;  // 64
constexpr int kWarpsPerBlock = 8;
constexpr float kOpen = -1.0f;  // left in SO by k_cepstrum_bins for k_cepstrum (no value is negative)

// kMarked: only the cells that hold kOpen, looked for 32 at a time.
template <bool kMarked>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, 6)
    k_cepstrum(DevGeometry g, Batch b, const float* __restrict__ SI, float* __restrict__ SO, int64_t stride,
               int64_t len, const double* __restrict__ tw64, const double* __restrict__ tw32) {
    __shared__ cd xs[kWarpsPerBlock][kWin];
    __shared__ double twa[2 * (kWin - 1)], twb[2 * (kWin / 2 - 1)];
    for (int i = threadIdx.x; i < 2 * (kWin - 1); i += blockDim.x) twa[i] = tw64[i];
    for (int i = threadIdx.x; i < 2 * (kWin / 2 - 1); i += blockDim.x) twb[i] = tw32[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cd* x = xs[warp];
    const int slot = blockIdx.y;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    const float* in = SI + slot * stride;
    float* out = SO + slot * stride;
    const double norm64 = __ddiv_rn(1.0, __dsqrt_rn(64.0));
    const double norm32 = __ddiv_rn(1.0, __dsqrt_rn(32.0));
    const int64_t warps = (int64_t)gridDim.x * kWarpsPerBlock;
    constexpr int kStep = kMarked ? 32 : 1;
    for (int64_t q0 = ((int64_t)blockIdx.x * kWarpsPerBlock + warp) * kStep; q0 < len; q0 += warps * kStep) {
        unsigned todo = 1u;
        if (kMarked) todo = __ballot_sync(0xffffffffu, q0 + lane < len && out[q0 + lane] == kOpen);
        for (; todo; todo &= todo - 1) {
            const int64_t p = q0 + __ffs(todo) - 1;
            const int r = owner_row(d, first, last, p);  // warp-uniform
            if (r < 0) {
                if (lane == 0) out[p] = 0.0f;
                continue;
            }
            const int64_t base = (int64_t)r * d.dim_i;
            const int j = (int)(p - base);
            const int f = first[r], l = last[r];
            bool fin = true, empty = true;
            for (int m = lane; m < kWin; m += 32) {
                const int idx = j - kWin / 2 + m;
                x[m] = (idx < f || idx >= l) ? cd{0.0, 0.0} : cd{(double)in[base + idx], 0.0};
                fin = fin && isfinite(x[m].re);
                empty = empty && x[m].re == 0.0;
            }
            // An empty window (image borders, cells of overrunning rows: float always
            // leaves it open): every log is -inf, so every c_k but the first is NaN
            // and no sample ascends: 0.
            if (kMarked && __all_sync(0xffffffffu, empty)) {
                if (lane == 0) out[p] = 0.0f;
                continue;
            }
            __syncwarp();
            // Finite real input: the reduced-work FFT gives the same values up to the
            // sign of zeros, which neither |X|^2 nor -min(0, c) can see.
            if (__all_sync(0xffffffffu, fin)) warp_fft_real<kKeepLow>(x, kWin, twa, lane);  // X_k, k < 32
            else warp_fft(x, kWin, twa, lane);
            // |X_k|^2 of the 1/sqrt(64)-scaled spectrum, k < 32, then its log.
            {
                const cd v = x[lane];
                const double re = __dmul_rn(v.re, norm64), im = __dmul_rn(v.im, norm64);
                const double ps = __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
                __syncwarp();
                x[lane] = {log(ps), 0.0};
            }
            __syncwarp();
            // A zero power gives log = -inf: such cells keep the exact FFT.
            if (__all_sync(0xffffffffu, isfinite(x[lane].re)))
                warp_fft_real<kKeepLowRe>(x, kWin / 2, twb, lane);  // Re c_k, k < 16
            else warp_fft(x, kWin / 2, twb, lane);
            // s_k = -min(0, c_k) for k < 16 (lane k), then getBlurParameter2: from
            // index 5 skip the non-ascending head; the result is the sample before
            // the first ascent or any larger sample after the ascending one.  The
            // samples are -0 or positive (never +0 or NaN), so the reference's
            // sequential `s > best` scan and a max reduction give the same value.
            const int k = lane & (kWin / 4 - 1);
            const double c = __dmul_rn(x[k].re, norm32);
            const double sk = -((c < 0.0) ? c : 0.0);  // -std::min(0.0, c)
            const double prev = __shfl_up_sync(0xffffffffu, sk, 1);
            const unsigned asc = __ballot_sync(0xffffffffu, lane >= 5 && lane < kWin / 4 && sk > prev);
            double best = 0.0;
            if (asc) {
                const int i = __ffs(asc) - 1;  // first ascent
                double m = (lane == i - 1 || (lane > i && lane < kWin / 4)) ? sk : -0.0;
                for (int o = 16; o > 0; o >>= 1) {
                    const double t = __shfl_xor_sync(0xffffffffu, m, o);
                    m = t > m ? t : m;
                }
                best = m;
            }
            if (lane == 0) out[p] = __double2float_rn(__dmul_rn(best, 10000.0));
            __syncwarp();
        }
    }
}

// ---- bins in float -------------------------------------------------------------

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
// full: every sample lies inside the row (mean: the window's centre sample).
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
    const float err = 0.17678f * (2.2f * dx + 0.7f * (4.0f * u * (17.0f + all) + 14.0f * u * all)) + 100.0f * u;
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
    const bool sure = b0 == b1 && dx < 0.05f && all < 1e4f && l2 > 1e-20f && l2 < 1e24f;
    return sure ? b0 : -1.0f;
}

// One warp per 32 consecutive valid cells of a skewed row.
__global__ void __launch_bounds__(kWarpsPerBlock * 32, 2)
    k_cepstrum_bins(DevGeometry g, Batch b, const float* __restrict__ SI, float* __restrict__ SO, int64_t stride,
                    int col_blocks) {
    __shared__ float seg[kWarpsPerBlock][32 + kWin];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    const int unit = blockIdx.x * kWarpsPerBlock + warp;
    const int r = unit / col_blocks;
    if (r >= d.H) return;
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    const int f = first[r], l = last[r];
    const int j0 = f + (unit % col_blocks) * 32;
    if (j0 >= l) return;  // warp-uniform
    const int64_t base = (int64_t)r * d.dim_i;
    const float* in = SI + slot * stride + base;
    float* sw = seg[warp];
#pragma unroll
    for (int t = 0; t < 3; t++) {
        const int x = j0 - kWin / 2 + lane + 32 * t;
        sw[lane + 32 * t] = x >= f && x < l ? in[x] : 0.0f;
    }
    __syncwarp();
    const int j = j0 + lane;
    if (j >= l || (j >= d.dim_i && owner_row(d, first, last, base + j) != r)) return;
    const bool full = j - kWin / 2 >= f && j + kWin / 2 <= l;
    const float bin = cepstrum_bin(sw + lane, full ? sw[lane + kWin / 2] : 0.0f);
    SO[slot * stride + base + j] = bin >= 0.0f ? __fmaf_rn(1000.0f, bin, 500.0f) : kOpen;
}

}  // namespace

cudaError_t launch_cepstrum(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                            int64_t len, const double* tw64, const double* tw32, cudaStream_t st) {
    int64_t blocks = (len + kWarpsPerBlock - 1) / kWarpsPerBlock;
    if (blocks > 8192) blocks = 8192;
    k_cepstrum<false><<<dim3((unsigned)blocks, b.count), kWarpsPerBlock * 32, 0, st>>>(g, b, SI, SO, stride, len, tw64,
                                                                                        tw32);
    return cudaGetLastError();
}

cudaError_t launch_cepstrum_bins(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                                 int64_t len, int max_H, int max_cols, const double* tw64, const double* tw32,
                                 cudaStream_t st) {
    const int col_blocks = (max_cols + 31) / 32;
    const int64_t units = (int64_t)max_H * col_blocks;
    k_cepstrum_bins<<<dim3((unsigned)((units + kWarpsPerBlock - 1) / kWarpsPerBlock), b.count), kWarpsPerBlock * 32, 0,
                      st>>>(g, b, SI, SO, stride, col_blocks);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    int64_t blocks = (len + kWarpsPerBlock * 32 - 1) / (kWarpsPerBlock * 32);
    if (blocks > 1024) blocks = 1024;
    k_cepstrum<true><<<dim3((unsigned)blocks, b.count), kWarpsPerBlock * 32, 0, st>>>(g, b, SI, SO, stride, len, tw64,
                                                                                       tw32);
    return cudaGetLastError();
}

}  // namespace ske
