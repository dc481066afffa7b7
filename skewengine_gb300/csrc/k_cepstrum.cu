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
// (a thread per two cells, the windows in registers), and only the cells whose bin
// that leaves open run the exact kernel.  The whole run of a 512 x 512 texture
// (180 angles): 353.3 ms with every cell in binary64, 2.57 ms so (the float
// kernel 1.86, the open cells 0.40).
// cepstrum_bin.cuh has the evaluation and its bounds.
#include "cepstrum_bin.cuh"

namespace ske {

namespace {

constexpr int kWin = kBlurWindow;  // 64
constexpr int kWarpsPerBlock = 8;
constexpr float kOpen = -1.0f;  // left in SO by k_cepstrum_bins for k_cepstrum (no value is negative)

// kMarked: only the cells that hold kOpen (MarkScan).
template <bool kMarked>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, 6)
    k_cepstrum(DevGeometry g, Batch b, const float* __restrict__ SI, float* __restrict__ SO, int64_t stride,
               int64_t len, MarkShape shape, const double* __restrict__ tw64, const double* __restrict__ tw32) {
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
    const int step = kMarked ? shape.step : 1, groups = kMarked ? shape.groups : 1;
    const int64_t far = warps * step;
    for (int64_t q0 = ((int64_t)blockIdx.x * kWarpsPerBlock + warp) * step; q0 < len; q0 += far * groups) {
        MarkScan marks;
        if (kMarked) marks.read(out, q0, far, len, shape, kOpen, lane);
        int64_t p = q0;
        for (bool some = kMarked ? marks.next(q0, far, p) : true; some; some = kMarked && marks.next(q0, far, p)) {
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

// Four CTAs of four warps, 128 registers: 1.86 ms; three, without the few spills,
// 1.91.
constexpr int kBinWarps = 4;

// One warp per 32 columns of two skewed rows, the upper and lower half of the pair
// that a lane holds.
__global__ void __launch_bounds__(kBinWarps * 32, 4)
    k_cepstrum_bins(DevGeometry g, Batch b, const float* __restrict__ SI, float* __restrict__ SO, int64_t stride,
                    int col_blocks) {
    __shared__ f2 seg[kBinWarps][32 + kWin];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    const int unit = blockIdx.x * kBinWarps + warp;
    const int r = 2 * (unit / col_blocks);
    if (r >= d.H) return;
    const bool two = r + 1 < d.H;
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    const int f0 = first[r], l0 = last[r];
    const int f1 = two ? first[r + 1] : f0, l1 = two ? last[r + 1] : f0;
    const int64_t base = (int64_t)r * d.dim_i;
    const float* in = SI + slot * stride + base;
    f2* sw = seg[warp];
    // (Two rows together may span more columns than the longest one.)
    for (int j0 = min(f0, f1) + (unit % col_blocks) * 32; j0 < max(l0, l1); j0 += col_blocks * 32) {
        __syncwarp();
#pragma unroll
        for (int t = 0; t < 3; t++) {
            const int x = j0 - kWin / 2 + lane + 32 * t;
            sw[lane + 32 * t] = pk(x >= f0 && x < l0 ? in[x] : 0.0f, x >= f1 && x < l1 ? in[x + d.dim_i] : 0.0f);
        }
        __syncwarp();
        const int j = j0 + lane;
        const bool own0 = j >= f0 && j < l0 && (j < d.dim_i || owner_row(d, first, last, base + j) == r);
        const bool own1 =
            j >= f1 && j < l1 && (j < d.dim_i || owner_row(d, first, last, base + d.dim_i + j) == r + 1);
        if (!own0 && !own1) continue;
        float m0, m1;
        upk(sw[lane + kWin / 2], m0, m1);
        const f2 mean = pk(j - kWin / 2 >= f0 && j + kWin / 2 <= l0 ? m0 : 0.0f,
                           j - kWin / 2 >= f1 && j + kWin / 2 <= l1 ? m1 : 0.0f);
        const float2 bin = cepstrum_bin<false>(sw + lane, mean);
        float* out = SO + slot * stride + base + j;
        if (own0) out[0] = bin.x >= 0.0f ? __fmaf_rn(1000.0f, bin.x, 500.0f) : kOpen;
        if (own1) out[d.dim_i] = bin.y >= 0.0f ? __fmaf_rn(1000.0f, bin.y, 500.0f) : kOpen;
    }
}

}  // namespace

cudaError_t launch_cepstrum(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                            int64_t len, const double* tw64, const double* tw32, cudaStream_t st) {
    int64_t blocks = (len + kWarpsPerBlock - 1) / kWarpsPerBlock;
    if (blocks > 8192) blocks = 8192;
    k_cepstrum<false><<<dim3((unsigned)blocks, b.count), kWarpsPerBlock * 32, 0, st>>>(g, b, SI, SO, stride, len,
                                                                                        MarkShape(), tw64, tw32);
    return cudaGetLastError();
}

cudaError_t launch_cepstrum_bins(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                                 int64_t len, int max_H, int max_cols, const double* tw64, const double* tw32,
                                 cudaStream_t st) {
    const int col_blocks = (max_cols + 31) / 32;
    const int64_t units = (int64_t)((max_H + 1) / 2) * col_blocks;
    k_cepstrum_bins<<<dim3((unsigned)((units + kBinWarps - 1) / kBinWarps), b.count), kBinWarps * 32, 0, st>>>(
        g, b, SI, SO, stride, col_blocks);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const MarkShape shape = mark_shape(len, kWarpsPerBlock, b.count);
    k_cepstrum<true><<<dim3(shape.blocks, b.count), kWarpsPerBlock * 32, 0, st>>>(g, b, SI, SO, stride, len, shape, tw64,
                                                                                  tw32);
    return cudaGetLastError();
}

}  // namespace ske
