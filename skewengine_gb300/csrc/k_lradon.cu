// Local Radon transform (pointRadon, src/kernelRADN.h:114-182), the reference's
// Radon operator with its LRT switch set (kernelRADN.h:212-220).
//
// For every valid skewed cell (i, j) of a sector:
//   W(k, j) = sum over l = j-32 .. j+32 of S[k, l]   (binary64, in increasing l;
//             columns outside row k's valid range and rows outside the grid add 0)
//   x[m]    = W(i-32+m, j) * gauss[m],  m < 64,  gauss from the sector's scale
//   X       = FFT(x) / 8;  Y[k] = taper[k] * Re X[k] for k <= 25, else 0
//   Z       = FFT(Y) / 8;  out = getParameter(Z): from m = 5 the first
//             |Z_m|^2 > |Z_{m-1}|^2 gives |Z_{m-1}|^2 (none: 0), stored as float.
//
// The output is the reference's, bit for bit, but most cells never run its two
// binary64 transforms.  GB300 does 1/64 as many binary64 as float operations,
// and the transforms alone held the operator at the FP64 pipe's rate (279 ms
// per 512 x 512 image at all 180 angles, that pipe 83% busy).  Every value the
// output depends on is a comparison or one rounding to float, so a cheaper
// evaluation with a proven error decides it unless it falls within that error
// of a tie (the whole run of that image: 278.7 ms before, 3.34 ms so, of it 0.25 ms
// in step 1, 2.4 in step 2 and 0.35 in step 3):
//  1. k_lradon_sums: W of every row, once per column (the tile-by-tile form
//     recomputed each about three times), as exact 64-bit integer prefix sums
//     where the reference's sequential binary64 sums make no rounding.
//  2. k_lradon_cells, two cells per thread.  Both transforms and the weights
//     compose into Z_m = sum over q of (W(i-q, j) + W(i+q, j)) F_m[q], q = 0..32
//     (gauss and the kept bins' cosines are even around row i), so one Z_m is
//     66 multiply-adds, and m runs from 4 only until the first ascent (m = 6 or
//     7 on textures).  Float decides the ascent; the one Z_{m-1} the output
//     needs is then formed from 28-bit integers, whose products add up without
//     rounding in 64 bits, and float corrections, and rounded.
//  3. k_lradon_exact: the cells neither step could decide (about one in a
//     thousand of a texture's) run the reference's transforms, one warp per cell.
//
// W of a column of a tile is hi + lo in units of g, the largest |W| of the column
// being 2^26 .. 2^27 of them: hi an integer, |lo| <= 1/2.  F is an integer of
// 2^-33 units (|F| < 1/4) plus a rest.  Error bounds in g (u = 2^-24, maxW = the largest |W|
// of the cell's rows, SF_m = sum over q of |F_m[q]| times the W it multiplies):
//  * float Z_m: lo left out, SF_m / 2; rounding of hi, of the pair's sum, of F_m
//    and of the last sum, u each; and u for every addition from q's own to the
//    end of its chain, q/2 + 1 of them since the chains run from q = 32 down to
//    0, towards the large F: together u maxW SW_m, SW_m = sum of (q/2 + 5) times
//    |F_m[q]|, formed per sector (LrTable).
//  * integer Z_m: each component takes two float chains of 33 corrections, of lo
//    (partial sums below sum of |F_m[q]| < 0.46) and of the rest of F (33 times
//    2^28 2^-34 = 0.52): 33 u 0.98 = 1.9e-6, and 1.1e-6 for the inputs' own
//    roundings and joining the parts; together below 5e-6 for the complex value.
//    F_m itself is good to 2^-46 maxW.
//  * the reference's own binary64 result differs from the exact one by the
//    rounding of its 12 stages and its iterated twiddles (up to 15 * 2^-53 off
//    the unit circle in a stage of 64 points, 61 over a transform's stages): at
//    most 45 * 2^-53 S = 5e-15 S, S = sum of |W| gauss <= maxW sum gauss.
#include <algorithm>
#include <climits>
#include <cmath>

#include "f32x2.cuh"
#include "kernels.h"

namespace ske {

namespace {

constexpr int kW = kLocalRadonWindow;  // 64
constexpr int kHalf = kW / 2;          // 32
constexpr int kWarps = 8;

// ---- window sums -------------------------------------------------------------
// One warp per (row, 128 columns): the 192 cells the windows cover are staged,
// every float is an integer multiple of 2^(e - 150), and when the cells'
// exponents span at most 28 binades and the sum of their magnitudes in units of
// the smallest 2^e stays below 2^53, every partial sum of the reference's
// sequential binary64 loop is exact, so each window sum is a difference of two
// 64-bit integer prefix sums.  Other blocks (or a non-finite cell) keep the
// sequential adds.  Columns up to dim_l, rows of W with that pitch; memory
// bound (8 bytes written per cell).
constexpr int kSumCols = 128;
constexpr int kSumStage = kSumCols + kW;  // 192: windows of 65 around 128 columns

__global__ void __launch_bounds__(kWarps * 32)
    k_lradon_sums(DevGeometry g, Batch b, int slot0, const float* __restrict__ SI, int64_t stride,
                  double* __restrict__ W, int64_t wstride, int col_blocks) {
    __shared__ float cells[kWarps][kSumStage];
    __shared__ long long prefix[kWarps][kSumStage + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = slot0 + blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    const int unit = blockIdx.x * kWarps + warp;
    const int r = unit / col_blocks, j0 = (unit % col_blocks) * kSumCols;
    if (r >= d.H || j0 >= d.diml) return;  // warp-uniform
    const int f = g.first[d.row_off + r], l = g.last[d.row_off + r];
    double* out = W + blockIdx.y * wstride + (int64_t)r * d.diml;
    if (l <= f || j0 + kSumCols + kHalf <= f || j0 - kHalf >= l) {  // no valid cell in any window
        for (int j = j0 + lane; j < min(j0 + kSumCols, d.diml); j += 32) out[j] = 0.0;
        return;
    }
    const float* row = SI + slot * stride + (int64_t)r * d.dim_i;
    float* s = cells[warp];
#pragma unroll
    for (int t = 0; t < kSumStage / 32; t++) {
        const int c = j0 - kHalf + lane + 32 * t;
        s[lane + 32 * t] = c >= f && c < l ? row[c] : 0.0f;
    }
    __syncwarp();
    constexpr int kPer = kSumStage / 32;  // 6 consecutive cells per lane
    unsigned u[kPer], m[kPer];
    int ee[kPer], emin = INT_MAX, emax = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        u[k] = __float_as_uint(s[kPer * lane + k]);
        const int e8 = (int)((u[k] >> 23) & 0xffu);
        m[k] = (u[k] & 0x7fffffu) | (e8 ? 0x800000u : 0u);
        ee[k] = m[k] ? max(e8, 1) : INT_MAX;
        emin = min(emin, ee[k]);
        emax = max(emax, e8);
    }
    emin = __reduce_min_sync(0xffffffffu, emin);
    emax = __reduce_max_sync(0xffffffffu, emax);
    bool exact = emax != 0xff && (emin == INT_MAX || emax - emin <= 28);
    long long incl = 0;
    if (exact && emin != INT_MAX) {
        long long v[kPer], excl = 0;
        unsigned long long mag = 0;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const long long x = m[k] ? (long long)m[k] << (ee[k] - emin) : 0;  // < 2^52
            v[k] = (u[k] >> 31) ? -x : x;
            mag += (unsigned long long)x;
            incl += v[k];
        }
        excl = incl;
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        excl = incl - excl;
        for (int o = 16; o > 0; o >>= 1) mag += __shfl_xor_sync(0xffffffffu, mag, o);
        exact = mag < (1ull << 53);
        if (exact) {
            long long* pre = prefix[warp];
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                pre[kPer * lane + k] = excl;
                excl += v[k];
            }
            if (lane == 31) pre[kSumStage] = excl;
            __syncwarp();
            const double scale = __longlong_as_double((long long)(emin - 150 + 1023) << 52);
            for (int t = lane; t < kSumCols && j0 + t < d.diml; t += 32)
                out[j0 + t] = __dmul_rn(__ll2double_rn(pre[t + kW + 1] - pre[t]), scale);
        }
    } else if (exact) {  // all cells zero
        for (int t = lane; t < kSumCols && j0 + t < d.diml; t += 32) out[j0 + t] = 0.0;
    }
    if (!exact) {
        for (int t = lane; t < kSumCols && j0 + t < d.diml; t += 32) {
            double acc = 0.0;
            for (int k = 0; k <= kW; k++) acc = __dadd_rn(acc, (double)s[t + k]);
            out[j0 + t] = acc;
        }
    }
}

// ---- composed filters --------------------------------------------------------
// F_m[q] = gauss[32-q] K_m[q] for m = kM0 .. 31, with
// K_m[q] = 1/64 sum over k < 26 of (-1)^k taper[k] cos(2 pi k q / 64)
// e^(-2 pi i k m / 64) from the host (lradon_init_tables).
constexpr int kM0 = 4;
constexpr int kMn = kHalf - kM0;  // 28
constexpr int kQn = kHalf + 1;    // 33
constexpr int kQp = kQn + 1;      // row pitch of the float table (16-byte rows)

struct LrTable {
    int4 fix[kQn][kMn];    // {re, im} in 2^-33 units, {re, im} as float bits
    float2 rest[kQn][kMn];  // what the integers leave of re and im
    float2 one[kMn][kQp];  // {re, im}, rows for the float search
    float sf[kMn], sw[kMn];  // SF_m and SW_m, rounded up
    float sg;                // sum of the 64 weights, rounded up
    float unused[7];
};

__device__ double2 g_lr_kernel[kQn * kMn];  // K_m[q] at [q][m]

__global__ void __launch_bounds__(256)
    k_lradon_tables(Batch b, int slot0, const double* __restrict__ gauss_all, LrTable* __restrict__ tab) {
    const int slot = slot0 + blockIdx.x;
    const double* gauss = gauss_all + (int64_t)b.angle[slot] * kW;
    LrTable& t = tab[blockIdx.x];
    for (int k = threadIdx.x; k < kQn * kMn; k += blockDim.x) {
        const int q = k / kMn, m = k % kMn;
        const double2 K = g_lr_kernel[k];
        const double re = K.x * gauss[kHalf - q], im = K.y * gauss[kHalf - q];
        const int ri = __double2int_rn(re * 8589934592.0), ii = __double2int_rn(im * 8589934592.0);
        t.fix[q][m] = make_int4(ri, ii, __float_as_int((float)re), __float_as_int((float)im));
        t.rest[q][m] = make_float2((float)(re - ri * 1.1641532182693481e-10), (float)(im - ii * 1.1641532182693481e-10));
        t.one[m][q] = make_float2((float)re, (float)im);
        if (q == 0) t.one[m][kQn] = make_float2(0.0f, 0.0f);
    }
    if (threadIdx.x < kMn) {
        double s = 0.0, w = 0.0;
        for (int q = 0; q < kQn; q++) {
            const double2 K = g_lr_kernel[q * kMn + threadIdx.x];
            const double v = (q == 0 || q == kHalf ? 1.0 : 2.0) * gauss[kHalf - q] * sqrt(K.x * K.x + K.y * K.y);
            s += v;
            w += v * (q / 2 + 5);
        }
        t.sf[threadIdx.x] = (float)(s * 1.001);
        t.sw[threadIdx.x] = (float)(w * 1.001);
    }
    if (threadIdx.x == kMn) {
        double s = 0.0;
        for (int m = 0; m < kW; m++) s += gauss[m];
        t.sg = (float)(s * 1.001);
    }
}

// ---- cells ---------------------------------------------------------------------
constexpr int kTI = 128;              // cell rows per tile: 191 rows of W and one copy of the filters serve them (64
                                      // rows: 2.68 ms against 2.42 at 512 x 512)
constexpr int kTJ = 32;               // cell columns per tile (one lane each)
constexpr int kRows = kTI + kW - 1;   // rows of W a tile needs
constexpr int kPerWarp = (kRows + kWarps - 1) / kWarps;
constexpr float kUndecided = -1.0f;   // left in SO for k_lradon_exact (no output is negative)

struct CellSmem {
    int2 w[kRows][kTJ];      // W = hi + lo in units of the column's g: {hi, lo as float bits}
    float hif[kRows][kTJ];   // hi as float
    int top[kWarps][kTJ];    // largest exponent field of the column, per warp's rows
    int2 range[kTI];         // {first, last} of the tile's cell rows ({0, 0} past the last)
    LrTable tab;
};

// Binary64 w in units of 2^(emax - 1023 - 26), emax at least w's exponent field:
// hi the nearest integer, lo the rest to 2^-25 (bit operations: conversions run
// on the FP64 pipe).  A w below 2^-26 units counts as one of them, so that only zeros
// have neither (a texture beside 1e17 lies below).
__device__ __forceinline__ void split(double w, int emax, int* hi, float* lo) {
    const long long bits = __double_as_longlong(w);
    const int e = (int)((bits >> 52) & 0x7ff);
    const long long s = (bits & 0xfffffffffffffll) | (e ? 1ll << 52 : 0);
    const int t = min(26 + emax - e, 78);  // w = s 2^-t units
    long long h = 0, rem = s;
    if (t <= 60) {
        h = (s + (1ll << (t - 1))) >> t;
        rem = s - (h << t);
    }
    const float l = __fmul_rn(__int2float_rn((int)(rem >> (t - 26))), 1.4901161193847656e-8f);  // 2^-26
    *hi = bits < 0 ? -(int)h : (int)h;
    *lo = bits < 0 ? -l : l;
}

__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// acc 2^-33 + c as a normalised float pair (|acc 2^-33| < 2^30, |c| small).
__device__ __forceinline__ void to_pair(long long acc, float c, float& h, float& l) {
    const int ah = (int)(acc >> 33);
    const float fh = __int2float_rn(ah);
    const float rest = __int2float_rn(ah - __float2int_rn(fh));
    const float low = __fmaf_rn(__int2float_rn((int)((acc >> 3) & 0x3fffffff)), 9.3132257461547852e-10f, rest);
    two_sum(fh, __fadd_rn(low, c), h, l);
}

__global__ void __launch_bounds__(kWarps * 32, 2)
    k_lradon_cells(DevGeometry g, Batch b, int slot0, const double* __restrict__ W, int64_t wstride,
                   const LrTable* __restrict__ tabs, float* __restrict__ SO, int64_t stride, int tiles_j) {
    extern __shared__ __align__(16) unsigned char smem_lr[];
    CellSmem& sm = *reinterpret_cast<CellSmem*>(smem_lr);
    const int slot = slot0 + blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    const int i0 = (blockIdx.x / tiles_j) * kTI, j0 = (blockIdx.x % tiles_j) * kTJ;
    if (i0 >= d.H || j0 >= d.diml) return;
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    int any = 0;
    for (int r = threadIdx.x; r < kTI; r += blockDim.x) {
        const int i = i0 + r;
        const int2 fl = i < d.H ? make_int2(first[i], last[i]) : make_int2(0, 0);
        sm.range[r] = fl;
        if (fl.x < j0 + kTJ && fl.y > j0 && fl.x < fl.y) any = 1;
    }
    if (!__syncthreads_or(any)) return;
    // The sector's filters, while the window sums are fetched and split.
    for (int k = threadIdx.x; k < (int)(sizeof(LrTable) / 16); k += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (unsigned)__cvta_generic_to_shared(reinterpret_cast<int4*>(&sm.tab) + k)),
                     "l"(reinterpret_cast<const int4*>(tabs + blockIdx.y) + k));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = j0 + lane;
    int emax = 0;  // largest exponent field of the column's W
    {
        const double* wcol = W + blockIdx.y * wstride + j;
        double w[kPerWarp];
#pragma unroll
        for (int t = 0; t < kPerWarp; t++) {
            const int r = warp + t * kWarps, k = i0 - kHalf + r;
            w[t] = r < kRows && k >= 0 && k < d.H && j < d.diml ? wcol[(int64_t)k * d.diml] : 0.0;
            emax = max(emax, (int)((__double_as_longlong(w[t]) >> 52) & 0x7ff));
        }
        sm.top[warp][lane] = emax;
        __syncthreads();
        for (int t = 0; t < kWarps; t++) emax = max(emax, sm.top[t][lane]);
#pragma unroll
        for (int t = 0; t < kPerWarp; t++) {
            const int r = warp + t * kWarps;
            if (r >= kRows) continue;
            int h;
            float l;
            split(w[t], emax, &h, &l);
            sm.w[r][lane] = make_int2(h, __float_as_int(l));
            sm.hif[r][lane] = __int2float_rn(h);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    constexpr float u = 5.9604644775390625e-8f;  // 2^-24
    const float sg = sm.tab.sg;
    // g as a float; columns with a non-finite W or one outside the range where g
    // and the squares stay normal floats are left undecided.
    const bool col_ok = emax == 0 || (emax > 1023 - 30 && emax < 1023 + 80);
    const float unit = __uint_as_float((unsigned)min(max(emax - 1023 - 26 + 127, 1), 254) << 23);
    float* out = SO + slot * stride;
    for (int ca = 2 * warp; ca < kTI; ca += 2 * kWarps) {
        // Cells (i, j) and (i + 1, j), i = i0 + ca; cell i is staged row ca + 32.
        bool valid[2];
        int64_t p[2];
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int i = i0 + ca + c;
            valid[c] = j >= sm.range[ca + c].x && j < sm.range[ca + c].y;
            p[c] = (int64_t)i * d.dim_i + j;
            if (valid[c] && j >= d.dim_i && owner_row(d, first, last, p[c]) != i) valid[c] = false;
        }
        if (!__any_sync(0xffffffffu, valid[0] || valid[1])) continue;
        // V_q of both cells.
        const int c0 = ca + kHalf;
        float V[2][kQn], mw[2];
        {
            float up = sm.hif[c0 + 1][lane], dn = sm.hif[c0][lane];
            V[0][0] = dn;
            V[1][0] = up;
            mw[0] = fabsf(dn);
            mw[1] = fabsf(up);
            // Row c0 - q + 1 is cell i+1's lower row and cell i's previous one.
#pragma unroll
            for (int q = 1; q < kHalf; q++) {
                const float a0 = sm.hif[c0 - q][lane], b1 = sm.hif[c0 + 1 + q][lane];
                V[0][q] = __fadd_rn(a0, up);
                V[1][q] = __fadd_rn(dn, b1);
                mw[0] = fmaxf(fmaxf(mw[0], fabsf(a0)), fabsf(up));
                mw[1] = fmaxf(fmaxf(mw[1], fabsf(dn)), fabsf(b1));
                up = b1;
                dn = a0;
            }
            V[0][kHalf] = sm.hif[c0 - kHalf][lane];
            V[1][kHalf] = dn;
            mw[0] = fmaxf(mw[0], fabsf(V[0][kHalf]));
            mw[1] = fmaxf(mw[1], fabsf(dn));
        }
        // First ascent in float.  state: 0 searching, 1 found (at[c] = m - 1), 2
        // undecided, 3 too close between at[c] = m - 1 and m.
        float prev[2] = {0.0f, 0.0f}, ptol[2] = {0.0f, 0.0f};
        int state[2], at[2] = {kM0, kM0};
#pragma unroll
        for (int c = 0; c < 2; c++) state[c] = valid[c] && col_ok && mw[c] != 0.0f ? 0 : 2;
        for (int m = kM0; m < kHalf; m++) {
            if (!__any_sync(0xffffffffu, state[0] == 0 || state[1] == 0)) break;
            const float4* t4 = reinterpret_cast<const float4*>(sm.tab.one[m - kM0]);
            float zr[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}}, zi[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
            for (int q = kHalf; q >= 0; q -= 2) {
                const float4 t = t4[q / 2];
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    zr[c][0] = __fmaf_rn(V[c][q], t.x, zr[c][0]);
                    zi[c][0] = __fmaf_rn(V[c][q], t.y, zi[c][0]);
                    if (q + 1 < kQn) {
                        zr[c][1] = __fmaf_rn(V[c][q + 1], t.z, zr[c][1]);
                        zi[c][1] = __fmaf_rn(V[c][q + 1], t.w, zi[c][1]);
                    }
                }
            }
            const float sf = 0.51f * sm.tab.sf[m - kM0], sw = u * sm.tab.sw[m - kM0];
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const float re = __fadd_rn(zr[c][0], zr[c][1]), im = __fadd_rn(zi[c][0], zi[c][1]);
                const float nm = __fmaf_rn(re, re, __fmul_rn(im, im));
                // |Z|^2 is off by at most 2 |Z| e + e^2 and its own rounding.
                const float e = __fmaf_rn(sw, mw[c] + 1.0f, sf);
                const float tol = __fmaf_rn(e, __fmaf_rn(2.01f, sqrt_approx(nm), e), 4.0f * u * nm);
                const float diff = __fsub_rn(nm, prev[c]);
                if (m > kM0 && state[c] == 0) {
                    const bool sure = fabsf(diff) > 1.01f * (tol + ptol[c]);
                    if (!sure || diff > 0.0f) {
                        state[c] = sure ? 1 : 3;
                        at[c] = m - 1;
                    }
                }
                prev[c] = nm;
                ptol[c] = tol;
            }
        }
        // The one |Z_m|^2 the output is in integers, rounded where its whole error
        // interval rounds to the same float.  Cells float left too close go on
        // from there, one m at a time.
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int cc = c0 + c;
            float res = kUndecided;
            if (state[c] == 0) res = 0.0f;  // no ascent up to m = 31
            if (mw[c] == 0.0f && col_ok) {
                // Every hi is zero: where every W is (no lo either), there is no ascent.
                float l = 0.0f;
                for (int k = -kHalf; k < kHalf; k++) l = fmaxf(l, fabsf(__int_as_float(sm.w[cc + k][lane].y)));
                if (l == 0.0f) res = 0.0f;
            }
            float pa = 0.0f, pr = 0.0f, pd = 0.0f;  // |Z|^2 of the last m: pa + pr, off by at most pd
            int mi = at[c] - kM0;
            for (int step = 0; __any_sync(0xffffffffu, step == 0 ? (state[c] & 1) : state[c] == 3); step++) {
                long long ar = 0, ai = 0;
                float lr = 0.0f, li = 0.0f, fr = 0.0f, fi = 0.0f;
                auto tap = [&](int q, int vi, float vl) {
                    const float vf = __int2float_rn(vi);
                    const int4 F = sm.tab.fix[q][mi];
                    const float2 R = sm.tab.rest[q][mi];
                    ar += (long long)vi * F.x;
                    ai += (long long)vi * F.y;
                    lr = __fmaf_rn(vl, __int_as_float(F.z), lr);
                    li = __fmaf_rn(vl, __int_as_float(F.w), li);
                    fr = __fmaf_rn(vf, R.x, fr);
                    fi = __fmaf_rn(vf, R.y, fi);
                };
                const int2 wc = sm.w[cc][lane], we = sm.w[cc - kHalf][lane];
                tap(0, wc.x, __int_as_float(wc.y));
                tap(kHalf, we.x, __int_as_float(we.y));
#pragma unroll
                for (int q = 1; q < kHalf; q++) {
                    const int2 wa = sm.w[cc - q][lane], wb = sm.w[cc + q][lane];
                    tap(q, wa.x + wb.x, __fadd_rn(__int_as_float(wa.y), __int_as_float(wb.y)));
                }
                float zr, zrl, zi, zil;
                to_pair(ar, __fadd_rn(lr, fr), zr, zrl);
                to_pair(ai, __fadd_rn(li, fi), zi, zil);
                // |Z|^2 = a + r, a the larger part.
                const float p0 = __fmul_rn(zr, zr), p1 = __fmul_rn(zi, zi);
                float r0 = __fmaf_rn(zr, zr, -p0), r1 = __fmaf_rn(zi, zi, -p1);
                r0 = __fmaf_rn(2.0f * zr, zrl, r0);
                r1 = __fmaf_rn(2.0f * zi, zil, r1);
                float a, r;
                two_sum(p0, p1, a, r);
                r = __fadd_rn(r, __fadd_rn(r0, r1));
                // 2^-46 of F, 5e-15 sum gauss of the reference; 2^-42 a of the squares.
                const float e = __fmaf_rn(mw[c] + 1.0f, 1.4210854715202004e-14f + 5.05e-15f * sg, 5e-6f);
                const float del = __fmaf_rn(e, __fmaf_rn(2.01f, sqrt_approx(a), e), 2.2737367544323206e-13f * a);
                bool next = true;  // this m becomes the last one
                if (step > 0) {
                    const float diff = __fadd_rn(__fsub_rn(a, pa), __fsub_rn(r, pr));
                    const bool sure = fabsf(diff) > 1.01f * (del + pd) + 2.0f * u * fabsf(diff);
                    next = state[c] == 3 && sure && diff < 0.0f;
                    if (state[c] == 3 && !next) state[c] = sure ? 1 : 2;
                }
                if (next) pa = a, pr = r, pd = del;
                if (state[c] == 3 && ++mi == kMn) {
                    state[c] = 2;
                    res = 0.0f;  // no ascent up to m = 31
                }
            }
            const float lo = __fadd_rn(pa, __fsub_rd(pr, pd)), hi = __fadd_rn(pa, __fadd_ru(pr, pd));
            // In the input's units, where that loses nothing.
            const float v = __fmul_rn(__fmul_rn(lo, unit), unit);
            if (state[c] == 1 && lo == hi && v > 1e-35f && v < 1e38f) res = v;
            if (valid[c]) out[p[c]] = res;
        }
    }
}

// ---- undecided cells -------------------------------------------------------------
// The reference's operations: one warp per cell, both 64-point transforms with
// one butterfly per lane per stage (warp_fft: the reference's DIF order and
// twiddle sequence, binary64, no fused operations).  The 1/sqrt(64) scaling is
// the reference's complex multiplication by (0.125, 0).  Cells whose W are all
// finite use warp_fft_real and real scalings: the same values up to the sign of
// zeros, so the squared magnitudes are bit-identical.  The cells are
// those that hold the mark k_lradon_cells left (MarkScan).  98 binary64 operations a
// cell hold this kernel at that pipe's rate (81%), so its time is the number of
// cells: 98.8 thousand of a 512 x 512 texture's 47 million and 0.64 ms with F in
// 2^-30 units and wider bounds, 0.35 ms as it is.
//
// kDirect: every cell, each window sum formed here from the skewed input; what runs
// where the memory for W is not to be had (a 256 x 256 image at 180 angles: 252 ms, 2.5
// with it).
template <bool kDirect>
__global__ void __launch_bounds__(kWarps * 32)
    k_lradon_exact(DevGeometry g, Batch b, int slot0, const float* __restrict__ SI, const double* __restrict__ W,
                   int64_t wstride, float* __restrict__ SO, int64_t stride, int64_t len, MarkShape shape,
                   const double* __restrict__ gauss_all, const double* __restrict__ taper_all,
                   const double* __restrict__ tw64) {
    __shared__ cd xs[kWarps][kW];
    __shared__ double tw[2 * (kW - 1)], gauss[kW], taper[kLocalRadonKeep];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = slot0 + blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    for (int t = threadIdx.x; t < 2 * (kW - 1); t += blockDim.x) tw[t] = tw64[t];
    for (int t = threadIdx.x; t < kW; t += blockDim.x) gauss[t] = gauss_all[(int64_t)b.angle[slot] * kW + t];
    for (int t = threadIdx.x; t < kLocalRadonKeep; t += blockDim.x) taper[t] = taper_all[t];
    __syncthreads();
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    const double* w = W + blockIdx.y * wstride;
    const float* in = SI + slot * stride;
    float* out = SO + slot * stride;
    cd* x = xs[warp];
    const cd scale{0.125, 0.0};  // 1/sqrt(64) (helper.h:102-104)
    const int64_t end = min((int64_t)len, (int64_t)(d.H - 1) * d.dim_i + d.diml);
    const int step = kDirect ? 1 : shape.step, groups = kDirect ? 1 : shape.groups;
    const int64_t far = (int64_t)gridDim.x * kWarps * step;
    for (int64_t q0 = ((int64_t)blockIdx.x * kWarps + warp) * step; q0 < end; q0 += far * groups) {
        MarkScan marks;
        if (!kDirect) marks.read(out, q0, far, end, shape, kUndecided, lane);
        int64_t p = q0;
        for (bool some = kDirect ? true : marks.next(q0, far, p); some; some = !kDirect && marks.next(q0, far, p)) {
            const int i = owner_row(d, first, last, p);  // warp-uniform; only valid cells are marked
            if (kDirect && i < 0) continue;
            const int j = (int)(p - (int64_t)i * d.dim_i);
            bool fin = true;
            for (int m = lane; m < kW; m += 32) {
                const int k = i - kHalf + m;
                double v = 0.0;
                if (kDirect && k >= 0 && k < d.H) {
                    const int f = first[k], l = last[k];
                    for (int c = j - kHalf; c <= j + kHalf; c++)
                        v = __dadd_rn(v, c >= f && c < l ? (double)in[(int64_t)k * d.dim_i + c] : 0.0);
                }
                if (!kDirect && k >= 0 && k < d.H) v = w[(int64_t)k * d.diml + j];
                fin = fin && isfinite(v);
                x[m] = cd{__dmul_rn(v, gauss[m]), 0.0};
            }
            const bool finite = __all_sync(0xffffffffu, fin);
            __syncwarp();
            // Only Re X_k for k < 26 is read: the pruned FFT forms Re X_k, k < 32.
            if (finite) warp_fft_real<kKeepLowRe>(x, kW, tw, lane);
            else warp_fft(x, kW, tw, lane);
            for (int m = lane; m < kW; m += 32) {
                double y = 0.0;
                if (m < kLocalRadonKeep) {
                    // Finite: x * (0.125, 0) is (re/8, im/8) up to the sign of zeros.
                    const double re = finite ? __dmul_rn(x[m].re, 0.125) : cmul(x[m], scale).re;
                    y = __dmul_rn(taper[m], re);
                }
                x[m] = cd{y, 0.0};
            }
            __syncwarp();
            // Y is zero from bin 26 on; only Z_m for m < 32 is read.
            if (finite) warp_fft_real<kKeepLow, true>(x, kW, tw, lane);
            else warp_fft(x, kW, tw, lane);
            x[lane] = finite ? cd{__dmul_rn(x[lane].re, 0.125), __dmul_rn(x[lane].im, 0.125)} : cmul(x[lane], scale);
            __syncwarp();
            // getParameter: from m = 5 the first |Z_m|^2 > |Z_{m-1}|^2 gives
            // |Z_{m-1}|^2 (none: 0).  Lane m forms |Z_m|^2 (the reference's
            // products and sum); a ballot finds the first ascent.
            const double nm = __dadd_rn(__dmul_rn(x[lane].re, x[lane].re), __dmul_rn(x[lane].im, x[lane].im));
            const double prev = __shfl_up_sync(0xffffffffu, nm, 1);
            const unsigned asc = __ballot_sync(0xffffffffu, lane >= 5 && lane < kHalf && nm > prev);
            const int ia = asc ? __ffs(asc) - 1 : 1;
            const double v = __shfl_sync(0xffffffffu, nm, ia - 1);
            if (lane == 0) out[p] = __double2float_rn(asc ? v : 0.0);
            __syncwarp();
        }
    }
}

}  // namespace

cudaError_t lradon_init_tables() {
    static double2 K[kQn * kMn];
    for (int q = 0; q < kQn; q++)
        for (int m = 0; m < kMn; m++) {
            double re = 0.0, im = 0.0;
            for (int k = 1; k < kLocalRadonKeep; k++) {
                const double taper = std::sin((k / (0.4 * kW - 1)) * M_PI_2);  // kernelRADN.h:157-161
                const double c = std::cos(2.0 * M_PI * ((k * q) % kW) / kW) * taper * (k & 1 ? -1.0 : 1.0);
                const double a = 2.0 * M_PI * ((k * (m + kM0)) % kW) / kW;
                re += c * std::cos(a);
                im -= c * std::sin(a);
            }
            K[q * kMn + m] = make_double2(re / kW, im / kW);
        }
    return cudaMemcpyToSymbol(g_lr_kernel, K, sizeof(K));
}

size_t lradon_scratch_bytes(int64_t max_rows, int diml, int slots) {
    const size_t w = ((size_t)max_rows * diml * sizeof(double) + 255) / 256 * 256;
    return (w + sizeof(LrTable)) * (size_t)slots;
}

cudaError_t launch_local_radon(const DevGeometry& g, const Batch& b, int slot0, int count, const float* SI, float* SO,
                               int64_t stride, int64_t len, int max_H, int max_cols, const double* gauss,
                               const double* taper, const double* tw64, void* scratch, cudaStream_t st) {
    if (count <= 0) return cudaSuccess;
    const int64_t wstride = (int64_t)(((size_t)max_H * max_cols * sizeof(double) + 255) / 256 * 256 / sizeof(double));
    double* W = static_cast<double*>(scratch);
    LrTable* tabs = reinterpret_cast<LrTable*>(W + wstride * count);
    k_lradon_tables<<<count, 256, 0, st>>>(b, slot0, gauss, tabs);
    const int col_blocks = (max_cols + kSumCols - 1) / kSumCols;
    const int64_t units = (int64_t)max_H * col_blocks;
    k_lradon_sums<<<dim3((unsigned)((units + kWarps - 1) / kWarps), count), kWarps * 32, 0, st>>>(
        g, b, slot0, SI, stride, W, wstride, col_blocks);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(CellSmem);
    e = cudaFuncSetAttribute(k_lradon_cells, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int tiles_i = (max_H + kTI - 1) / kTI, tiles_j = (max_cols + kTJ - 1) / kTJ;
    k_lradon_cells<<<dim3((unsigned)(tiles_i * tiles_j), count), kWarps * 32, smem, st>>>(g, b, slot0, W, wstride, tabs,
                                                                                        SO, stride, tiles_j);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const MarkShape shape = mark_shape(len, kWarps, count);
    k_lradon_exact<false><<<dim3(shape.blocks, count), kWarps * 32, 0, st>>>(g, b, slot0, SI, W, wstride, SO, stride, len,
                                                                            shape, gauss, taper, tw64);
    return cudaGetLastError();
}

cudaError_t launch_local_radon_direct(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                                      int64_t len, const double* gauss, const double* taper, const double* tw64,
                                      cudaStream_t st) {
    if (b.count == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)std::min<int64_t>((len + kWarps - 1) / kWarps, 8192);
    k_lradon_exact<true><<<dim3(blocks, b.count), kWarps * 32, 0, st>>>(g, b, 0, SI, nullptr, 0, SO, stride, len,
                                                                       MarkShape(), gauss, taper, tw64);
    return cudaGetLastError();
}

}  // namespace ske
