// Local Radon transform in float32 (SKE_FLAG_LOCAL_RADON_F32): the same
// quantity as k_lradon (pointRadon, src/kernelRADN.h:114-182), computed on the
// FP32 pipes instead of the reference's binary64 FFTs.
//
// For every valid skewed cell (i, j) of a sector:
//   W(k, j) = sum of the 65 staged cells l = j-32 .. j+32 of row k (float32, in
//             increasing l; cells outside a row's valid range are 0)
//   x[m]    = W(i-32+m, j) * gauss[m]                      m = 0..63
//   Y[k]    = taper[k] * (sum_m x[m] cos(2 pi k m / 64)) / 8      k = 0..25
//             (the real part of the 64-point transform of the real x, scaled
//             by 1/sqrt(64) as the reference's (0.125, 0) product)
//   Z[m]    = (sum_k Y[k] e^(-2 pi i k m / 64)) / 8               m = 4..31
//   out     = |Z[m-1]|^2 for the first m >= 5 with |Z[m]|^2 > |Z[m-1]|^2, else 0.
// Only the transform bins the reference reads are formed, as direct sums: the
// 64 x 26 cosine products of Y and the 26 x 28 complex products of Z.  The
// twiddles (cosines and sines of 2 pi (k m mod 64) / 64, rounded to float on
// the host) sit in shared memory as one row per m, read by every thread at the
// same address (broadcast, 16 bytes per load), with the 26 bins unrolled in
// registers.  Two cells per thread (a twiddle row serves both), their bins in
// packed f32x2 operations; the second transform stops at the bin where both have
// ascended.  A CTA of 256 threads owns a 128 x 32 tile of cells (32 x 32 where those
// are few), stages the skewed rows it needs (191 rows x 96 columns) and forms each W
// once.  Bound by the FP32 pipe: 1.4e9 packed multiply-adds per 512 x 512 image
// (32-row tiles and all 28 bins of every cell: 9.4 ms; 3.8 so).
// The order of the float32 sums differs from the reference's binary64 FFT, so
// values differ in their last bits, and where two successive |Z|^2 nearly tie
// the first ascent can fall on another bin: the rate of output cells that
// differ by more than a relative 1e-3 from the reference is measured and
// stated (tests/test_local_radon.py).  Ownership of cells past a row's span
// follows owner_row as in k_lradon.
#include <cmath>

#include "f32x2.cuh"
#include "kernels.h"

namespace ske {

namespace {

constexpr int kW = kLocalRadonWindow;  // 64
constexpr int kHalf = kW / 2;          // 32
constexpr int kKeep = kLocalRadonKeep;  // 26
constexpr int kTJ = 32;              // columns of a tile
template <int kTI>
constexpr int kRowsOf = kTI + kW - 1;  // W rows a tile of kTI rows needs
constexpr int kCols = kTJ + kW;      // 96 staged columns
constexpr int kThreads = 256;
// Rows of a tile.  Tall ones form each W fewer times; but a dozen to an SM or fewer of
// them leave it waiting for the longest (us of a run, 32 against 128 rows: one
// sector of 300 x 200 117 and 198, of 512 x 512 116 and 141, empty 137 and 203;
// 15 sectors of 512 x 512, 1920 tall tiles, 435 and 436; 30 of them 784 and 759).
constexpr int kTallTile = 128, kLowTile = 32;
constexpr int64_t kFewTiles = 12 * 152;
constexpr int kZ0 = 4, kZ1 = 32;  // |Z_m|^2 formed for m = kZ0 .. kZ1 - 1
constexpr int kZn = kZ1 - kZ0;
constexpr int kKP = 28;  // twiddle row pitch (kKeep padded to 16 bytes)

// Row m of the first transform: cos(2 pi k m / 64); rows m = kZ0.. of the
// second: cos and sin of 2 pi k m / 64; k < kKeep, zero padding.
// (Global arrays: the lanes of a warp copy different entries to shared memory,
// which a constant bank would serve one at a time.)
__device__ float g_tx[kW * kKP];
__device__ float2 g_tz[kZn * kKeep];  // {cos, sin}

template <int kTI>
struct SmemF {
    static constexpr int kRows = kRowsOf<kTI>;
    int2 range[kRows];  // {first, last} of the staged rows ({0, 0} outside the grid)
    int2 pad;
    float s[kRows][kCols];
    float w[kRows][kTJ];
    float gauss[kW];
    float taper[kKP];
    float tx[kW][kKP];
    float2 tz[kZn][kKeep];  // {cos, sin}
};

template <int kTI>
__global__ void __launch_bounds__(kThreads)
    k_lradon_f32(DevGeometry g, Batch b, const float* __restrict__ SI, float* __restrict__ SO, int64_t stride,
                 int tiles_j, const double* __restrict__ gauss_all, const double* __restrict__ taper) {
    constexpr int kRows = kRowsOf<kTI>;
    extern __shared__ __align__(16) float smem_f[];
    SmemF<kTI>& sm = *reinterpret_cast<SmemF<kTI>*>(smem_f);
    const int slot = blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    const int i0 = (blockIdx.x / tiles_j) * kTI, j0 = (blockIdx.x % tiles_j) * kTJ;
    if (i0 >= d.H) return;
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int any = 0;
    for (int r = threadIdx.x; r < kRows; r += blockDim.x) {
        const int k = i0 - kHalf + r;
        const int2 fl = k >= 0 && k < d.H ? make_int2(first[k], last[k]) : make_int2(0, 0);
        sm.range[r] = fl;
        if (r >= kHalf && r < kHalf + kTI && fl.x < j0 + kTJ && fl.y > j0 && fl.x < fl.y) any = 1;
    }
    if (!__syncthreads_or(any)) return;

    // Staged rows: a warp per row, three columns per lane, four rows in flight.
    const float* in = SI + slot * stride;
#pragma unroll 4
    for (int r = warp; r < kRows; r += kThreads / 32) {
        const int2 fl = sm.range[r];
        const float* row = in + (int64_t)(i0 - kHalf + r) * d.dim_i;
#pragma unroll
        for (int t = 0; t < kCols / 32; t++) {
            const int l = j0 - kHalf + lane + 32 * t;
            sm.s[r][lane + 32 * t] = l >= fl.x && l < fl.y ? row[l] : 0.0f;
        }
    }
    for (int t = threadIdx.x; t < kW; t += blockDim.x) sm.gauss[t] = (float)gauss_all[(int64_t)b.angle[slot] * kW + t];
    for (int t = threadIdx.x; t < kKeep; t += blockDim.x) sm.taper[t] = (float)taper[t];
    for (int t = threadIdx.x; t < kW * kKP; t += blockDim.x) (&sm.tx[0][0])[t] = g_tx[t];
    for (int t = threadIdx.x; t < kZn * kKeep; t += blockDim.x) (&sm.tz[0][0])[t] = g_tz[t];
    __syncthreads();
    // Window sums, 65 sequential adds each: four columns of a row per thread, so
    // a 16-byte load serves up to 16 of them.
    for (int t = threadIdx.x; t < kRows * (kTJ / 4); t += kThreads) {
        const int r = t / (kTJ / 4), c = 4 * (t % (kTJ / 4));
        const float4* src = reinterpret_cast<const float4*>(&sm.s[r][c]);
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i <= kW / 4; i++) {
            const float4 v4 = src[i];
            const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (4 * i + e >= k && 4 * i + e - k <= kW) acc[k] = __fadd_rn(acc[k], v[e]);
        }
        *reinterpret_cast<float4*>(&sm.w[r][c]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    __syncthreads();

    // Two cells per thread, rows ca and ca + 1 of the tile: every twiddle row and
    // window weight read from shared memory serves both.
    float* out = SO + slot * stride;
    for (int ca = 2 * warp; ca < kTI; ca += 2 * (kThreads / 32)) {
        const int cj = lane, j = j0 + cj;
        int64_t p[2];
        bool valid[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = i0 + ca + u;
            const int2 fl = sm.range[kHalf + ca + u];
            valid[u] = j >= fl.x && j < fl.y;
            p[u] = (int64_t)i * d.dim_i + j;
            if (valid[u] && j >= d.dim_i && owner_row(d, first, last, p[u]) != i) valid[u] = false;
        }
        const unsigned act = __ballot_sync(0xffffffffu, valid[0] || valid[1]);
        if (!valid[0] && !valid[1]) continue;
        // Bins k and k + 1 of a cell in one pair.
        f2 acc[2][kKeep / 2];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int k = 0; k < kKeep / 2; k++) acc[u][k] = 0;
#pragma unroll 16  // fewer moves of the accumulators: 4.4 ms at 2, 3.7 at 8, 3.56 at 16
        for (int m = 0; m < kW; m++) {
            const float gm = sm.gauss[m];
            const float x0 = __fmul_rn(sm.w[ca + m][cj], gm);
            const float x1 = __fmul_rn(sm.w[ca + 1 + m][cj], gm);
            const f2 x0p = pk(x0, x0), x1p = pk(x1, x1);
            const float4* t4 = reinterpret_cast<const float4*>(sm.tx[m]);
#pragma unroll
            for (int q = 0; q < kKP / 4; q++) {
                const float4 t = t4[q];
                const f2 tv[2] = {pk(t.x, t.y), pk(t.z, t.w)};
#pragma unroll
                for (int e = 0; e < 2; e++)
                    if (2 * q + e < kKeep / 2) {
                        acc[0][2 * q + e] = fma2(x0p, tv[e], acc[0][2 * q + e]);
                        acc[1][2 * q + e] = fma2(x1p, tv[e], acc[1][2 * q + e]);
                    }
            }
        }
        float re[2][kKeep];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int k = 0; k < kKeep; k += 2) {
                upk(acc[u][k / 2], re[u][k], re[u][k + 1]);
                re[u][k] = __fmul_rn(sm.taper[k], __fmul_rn(re[u][k], 0.125f));
                re[u][k + 1] = __fmul_rn(sm.taper[k + 1], __fmul_rn(re[u][k + 1], 0.125f));
            }
        // m goes on only while a cell of the warp has seen no ascent: m = 6 or 7
        // on textures, not 31.
        float prev[2] = {0.0f, 0.0f}, found[2] = {0.0f, 0.0f};
        bool done[2] = {!valid[0], !valid[1]};
        for (int m = kZ0; m < kZ1; m++) {
            if (__all_sync(act, done[0] && done[1])) break;
            f2 z[2] = {0, 0};  // {re, im}
            const float4* t4 = reinterpret_cast<const float4*>(sm.tz[m - kZ0]);
#pragma unroll
            for (int q = 0; q < kKeep / 2; q++) {
                const float4 t = t4[q];
                const f2 ta = pk(t.x, t.y), tb = pk(t.z, t.w);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    z[u] = fma2(pk(re[u][2 * q], re[u][2 * q]), ta, z[u]);
                    z[u] = fma2(pk(re[u][2 * q + 1], re[u][2 * q + 1]), tb, z[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                float zr, zi;
                upk(z[u], zr, zi);
                const float a = __fmul_rn(zr, 0.125f), bq = __fmul_rn(zi, 0.125f);
                const float nm = __fadd_rn(__fmul_rn(a, a), __fmul_rn(bq, bq));
                if (m > kZ0 && !done[u] && nm > prev[u]) {
                    found[u] = prev[u];
                    done[u] = true;
                }
                prev[u] = nm;
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++)
            if (valid[u]) out[p[u]] = found[u];
    }
}

}  // namespace

int lradon_f32_init_tables() {
    static float tx[kW * kKP];
    static float2 tz[kZn * kKeep];
    for (int m = 0; m < kW; m++)
        for (int k = 0; k < kKP; k++)
            tx[m * kKP + k] = k < kKeep ? (float)std::cos(2.0 * M_PI * ((k * m) % kW) / kW) : 0.0f;
    for (int m = kZ0; m < kZ1; m++)
        for (int k = 0; k < kKeep; k++) {
            const double a = 2.0 * M_PI * ((k * m) % kW) / kW;
            tz[(m - kZ0) * kKeep + k] = make_float2((float)std::cos(a), (float)std::sin(a));
        }
    if (cudaMemcpyToSymbol(g_tx, tx, sizeof(tx)) != cudaSuccess) return -1;
    if (cudaMemcpyToSymbol(g_tz, tz, sizeof(tz)) != cudaSuccess) return -1;
    return 0;
}

template <int kTI>
static cudaError_t launch_tiles(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                                int max_H, int max_cols, const double* gauss, const double* taper, cudaStream_t st) {
    const int tiles_i = (max_H + kTI - 1) / kTI, tiles_j = (max_cols + kTJ - 1) / kTJ;
    const size_t smem = sizeof(SmemF<kTI>);
    cudaError_t e = cudaFuncSetAttribute(k_lradon_f32<kTI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_lradon_f32<kTI><<<dim3((unsigned)(tiles_i * tiles_j), b.count), kThreads, smem, st>>>(g, b, SI, SO, stride,
                                                                                          tiles_j, gauss, taper);
    return cudaGetLastError();
}

cudaError_t launch_local_radon_f32(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                                   int max_H, int max_cols, const double* gauss, const double* taper,
                                   cudaStream_t st) {
    if (b.count == 0) return cudaSuccess;
    const int64_t tiles = (int64_t)((max_H + kTallTile - 1) / kTallTile) * ((max_cols + kTJ - 1) / kTJ) * b.count;
    auto launch = tiles <= kFewTiles ? launch_tiles<kLowTile> : launch_tiles<kTallTile>;
    return launch(g, b, SI, SO, stride, max_H, max_cols, gauss, taper, st);
}

}  // namespace ske
