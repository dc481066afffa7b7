// Radon ray sums + ramp-filtered back-projection (kernelRADN global mode,
// src/kernelRADN.h:221-258).
//
// Per sector: p_r = sum of the valid cells of skewed row r (double, in column
// order), P = FFT(p) over H2 = 2^ceil(log2 H) points, P_i *= i/H for i <= H/2
// and 0 above, q = IFFT(P), and every valid cell of row r gets (float)Re q_r.
// The FFT is the reference's radix-2 decimation-in-frequency transform
// (helper.h:59-106) with its exact twiddle sequence, computed in binary64 with
// no fused operations, so the result is bit-identical to the reference.
//
// Three launches per batch: row sums (k_radon_sums, one warp per row), transform (a
// cluster of four CTAs per sector, or one CTA), back-projection (one thread per
// cell).  Where no row is longer than
// twice its width (every grid up to 2:1) the engine skips the back-projection
// (its deskew reads the filtered row values) and the skew (k_radon_rows, a lane
// per row, gathers the skewed cells from the oriented input itself).  Selectable for sectors
// whose rows stay within their width: sums and transform as one fused sector
// kernel (k_radon_sector, a thread-block cluster per sector).
#include <climits>

#include <cooperative_groups.h>

#include "f32x2.cuh"
#include "kernels.h"

namespace ske {

namespace {

__device__ __forceinline__ int pow2_at_least(int h) {
    int p = 1;
    while (p < h) p <<= 1;
    return p;
}

// Row sums p[r] = the reference's left-to-right binary64 sum of row r's valid
// cells (kernelRADN.h:223-229); p[r] = 0 for H <= r < H2.  One warp per row.
// Every float is m * 2^e with an integer m of at most 24 bits; in units of the
// row's smallest 2^e the values are integers, and when the sum of their
// magnitudes stays below 2^53 every partial sum of the reference is exactly
// representable, i.e. its result is the exact sum, which does not depend on the
// order of additions.  The warp then forms that sum with coalesced loads and
// 64-bit integer partial sums (exponent spread <= 28, rows <= 2048 cells: no
// overflow) and returns sum * 2^emin.  Rows with a non-finite value or failing
// these conditions are added in binary64, left to right, by one lane.
//
constexpr int kSumWarps = 8;
constexpr int kMaxSpread = 28;
constexpr int kMaxExactRow = 2048;

// x << n for 0 <= n; n >= 64 gives 0 (PTX clamps the shift amount).
__device__ __forceinline__ unsigned long long shl64(unsigned long long x, int n) {
    unsigned long long y;
    asm("shl.b64 %0, %1, %2;" : "=l"(y) : "l"(x), "r"(n));
    return y;
}

// Per-lane part of an exact row sum.  A float with biased exponent field e8
// and significand m (hidden bit included) is m * 2^(max(e8, 1) - 150).  The
// lane keeps the sums of its positive and of its negative values as integers
// in units of 2^(emin - 150), emin its smallest exponent of a nonzero value so
// far (they are shifted left when emin drops); emax is its largest exponent
// field (255 for an infinity or NaN).  Values far apart in exponent may wrap
// the integers: the spread test at the end rejects those rows.
struct ExactPart {
    unsigned long long pos = 0, neg = 0;
    int emin = INT_MAX, emax = 0;
    __device__ __forceinline__ void add(float v) {
        const unsigned u = __float_as_uint(v);
        const int e8 = (int)((u >> 23) & 0xffu);
        const unsigned m = (u & 0x7fffffu) | (e8 ? 0x800000u : 0u);
        const int ee = m ? max(e8, 1) : INT_MAX;  // zeros leave emin alone
        if (ee < emin) {
            const int sh = emin == INT_MAX ? 0 : emin - ee;
            pos = shl64(pos, sh);
            neg = shl64(neg, sh);
            emin = ee;
        }
        emax = max(emax, e8);
        const unsigned long long x = shl64(m, ee - emin);  // m = 0: shift clamps, x = 0
        const unsigned long long xn = (u >> 31) ? x : 0ull;
        neg += xn;
        pos += x - xn;
    }
    // Not an exact candidate: a non-finite value or a spread above kMaxSpread.
    __device__ __forceinline__ bool bad() const {
        return emax == 0xff || (emin != INT_MAX && emax - emin > kMaxSpread);
    }
};

__global__ void __launch_bounds__(kSumWarps * 32)
    k_radon_sums(DevGeometry g, Batch b, const float* __restrict__ SI, int64_t stride, cd* __restrict__ P,
                 int64_t pstride) {
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.y;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int H2 = pow2_at_least(d.H);
    const float* in = SI + slot * stride;
    cd* p = P + slot * pstride;
    const int nwarps = gridDim.x * kSumWarps;
    for (int r = blockIdx.x * kSumWarps + (threadIdx.x >> 5); r < H2; r += nwarps) {
        if (r >= d.H) {
            if (lane == 0) p[r] = {0.0, 0.0};
            continue;
        }
        const int f = g.first[d.row_off + r], l = g.last[d.row_off + r];
        const float* row = in + (int64_t)r * d.dim_i;
        ExactPart a;
#pragma unroll 2
        for (int j = f + lane; j < l; j += 32) a.add(row[j]);
        const bool lane_bad = a.bad();
        int gmin = a.emin, gmax = a.emax;
        for (int o = 16; o > 0; o >>= 1) {
            gmin = min(gmin, __shfl_xor_sync(0xffffffffu, gmin, o));
            gmax = max(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
        }
        bool bad = __any_sync(0xffffffffu, lane_bad) || l - f > kMaxExactRow ||
                   (gmin != INT_MAX && gmax - gmin > kMaxSpread);  // gmax: largest field, >= any nonzero's

        double s = 0.0;
        if (!bad && gmin != INT_MAX) {
            // Units of 2^(gmin - 150): every value < 2^52, at most 2048 of them.
            const int sh = a.emin == INT_MAX ? 0 : a.emin - gmin;
            unsigned long long pos = shl64(a.pos, sh), neg = shl64(a.neg, sh);
            for (int o = 16; o > 0; o >>= 1) {
                pos += __shfl_xor_sync(0xffffffffu, pos, o);
                neg += __shfl_xor_sync(0xffffffffu, neg, o);
            }
            if (pos + neg < (1ull << 53)) {  // every partial sum exact: the exact sum
                const double scale = __longlong_as_double((long long)(gmin - 150 + 1023) << 52);
                s = __dmul_rn(__ll2double_rn((long long)(pos - neg)), scale);
            } else {
                bad = true;
            }
        }
        if (bad && lane == 0)
            for (int j = f; j < l; j++) s = __dadd_rn(s, (double)row[j]);
        if (lane == 0) p[r] = {s, 0.0};
    }
}

// Row sums formed from the oriented input, without a skewed grid (every sector
// with dim_l <= 2 dim_i).  A lane owns a row: 32 rows per CTA, each of its four
// warps a quarter of their columns.  All lanes are at the same column, so its
// shift, weight and address are one broadcast, and its 32 (or 33) source cells
// are consecutive: read from the transposed orientation (plain and mirrored
// sectors from orientation 2, transposed ones from the plain grid), where a
// column of the sector's own orientation is a row.  A warp per row, lanes along
// its columns, touched up to 32 lines a load at 45 degrees, took 15 integer
// operations a cell to add it up exactly and reduced every row over the lanes:
// 137 us per 512 x 512 image at 180 angles, this form 62 us in binary64's stead
// (13 instructions a cell are the cuts) and 48 us in float at 383 x 509.
// Where all 32 rows hold a batch of 32 columns with both their sources, which is
// most of a sector, a cell is two loads at one address, two products and a sum,
// 16 columns in flight; elsewhere each source is tested, about 70 us for all of
// them (both shapes).  The next batch's shifts and weights are on their way meanwhile.
// A cell is the skew's, w x[r-t-1] + (1-w) x[r-t], up to the sign of a zero.
//
// Exact sums in float.  With |cell| <= 2^E (E from the grid's largest finite
// magnitude) a cell is cut into multiples of q1 = 2^(E+1-B), q2 = q1 2^-B and
// q3, B = 24 - ceil(log2 n) for n columns: each part is added without rounding,
// its sum staying below 2^24 of its units.  q3 is at least 2^(E-53) n, so where
// nothing is left below it every partial sum of the reference's left-to-right
// binary64 loop is exact too: its result is the parts' sum.  Rows with a rest
// (exponents too far apart, a non-finite cell) are summed in 64-bit integers
// (RowPart), and where those do not fit either, left to right in binary64.
//
// kOver: rows may overrun their width into the next row's cells (and past the
// last row into zeros).  kF32: float sums, of kRowStep columns by pairs, those in
// turn with their roundings carried along: plainly added the output's error was 2 to 8%
// larger than by a warp's lanes, so it is 3 to 9% smaller (383 x 509: 45.5 -> 47.6 us).
//
// kFlight * kRowStep columns are in flight.  With fewer CTAs than the SMs hold (one to
// a dozen sectors) the float32 sums wait for their loads, and twice as many at a time
// take less (a whole run of 2000 x 2000, one sector: 235 -> 220 us; 15 sectors, 1920
// CTAs: 292 both; 45: 409 both; all 180: 944 and 947).  The binary64 cuts have no registers
// for more than 16 (one sector 260 -> 276).  The same sums.
constexpr int kRowWarps = 4;
constexpr int kRowStep = 8;  // columns of one addition
constexpr int64_t kRowFewCtas = 12 * 152;

// Exact integer sum of one row's cells in units of 2^(emin - 150).
struct RowPart {
    long long sum = 0;
    unsigned long long mag = 0;  // of the magnitudes
    int emin = INT_MAX, emax = 0;
    __device__ __forceinline__ void add(float v) {
        const unsigned u = __float_as_uint(v);
        const int e8 = (int)((u >> 23) & 0xffu);
        const unsigned m = (u & 0x7fffffu) | (e8 ? 0x800000u : 0u);
        const int ee = max(e8, 1);
        if (m && ee < emin) {
            const int sh = emin == INT_MAX ? 0 : emin - ee;
            sum = (long long)shl64((unsigned long long)sum, sh);
            mag = shl64(mag, sh);
            emin = ee;
        }
        emax = max(emax, e8);
        const unsigned long long x = shl64(m, ee - emin);  // m = 0: x = 0 whatever the shift
        mag += x;
        sum += (u >> 31) ? -(long long)x : (long long)x;
    }
    // Joins another part of the row.
    __device__ __forceinline__ void join(const RowPart& o) {
        const int e = min(emin, o.emin);
        const int sa = emin == INT_MAX ? 0 : emin - e, sb = o.emin == INT_MAX ? 0 : o.emin - e;
        sum = (long long)(shl64((unsigned long long)sum, sa) + shl64((unsigned long long)o.sum, sb));
        mag = shl64(mag, sa) + shl64(o.mag, sb);
        emin = e;
        emax = max(emax, o.emax);
    }
};

template <bool kF32, bool kOver, int kFlight>
__global__ void __launch_bounds__(kRowWarps * 32)
    k_radon_rows(DevGeometry g, Batch b, const float* __restrict__ orient, int64_t n_cells, int dimx, int dimy,
                 const unsigned* __restrict__ xmax, cd* __restrict__ P, int64_t pstride) {
    struct Column {
        float w;
        int t;
        int64_t off;  // of the w term's source cell from the lane's row
        // Columns taken by `inside`: w and t's bits are the weights of the lower
        // and the upper address.
    };
    __shared__ Column meta[kRowWarps][32];
    __shared__ RowPart parts[kF32 ? 1 : kRowWarps][32];
    __shared__ float sums[3][kRowWarps][32];
    __shared__ int marks[kRowWarps][32];  // the warp's part of the row has a rest
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.y;
    const SectorDesc& d = g.desc[b.angle[slot]];
    const int H = d.H, H2 = pow2_at_least(H), dim_i = d.dim_i, dim_o = d.dim_o;
    const int r = blockIdx.x * 32 + lane;
    if (blockIdx.x * 32 >= H2) return;
    cd* p = P + slot * pstride;
    const int f = r < H ? g.first[d.row_off + r] : 0, l = r < H ? g.last[d.row_off + r] : 0;
    const int lo = __reduce_min_sync(0xffffffffu, f < l ? f : INT_MAX), hi = __reduce_max_sync(0xffffffffu, f < l ? l : 0);
    if (hi == 0) {  // no valid cell in these rows
        if (warp == 0 && r < H2) p[r] = {0.0, 0.0};
        return;
    }
    // Cell (i, c) of the sector's orientation is base[c * cs + i * is].
    const bool tr = d.type == 1 || d.type == 2;
    const float* base = orient + (tr ? 0 : 2 * n_cells);
    int64_t cs = tr ? -dimx : dimy;
    int is = -1;
    if (d.type == 0) base += dimy - 1;
    if (d.type == 3) base += n_cells - 1, cs = -dimy;
    if (d.type == 1) base += n_cells - 1;
    if (d.type == 2) base += n_cells - dimx, is = 1;
    const float* mine = base + (int64_t)r * is;
    const float* low = mine + min(is, 0);
    const unsigned width = (unsigned)max(l - f, 0);
    auto column = [&](int j) {
        const int over = kOver && j >= dim_i ? 1 : 0, c = j - (over ? dim_i : 0);
        Column m;
        const bool in = c < dim_i;
        m.w = in ? g.weight[d.col_off + c] : 0.0f;
        m.t = (in ? g.target[d.col_off + c] : 0) - over;
        m.off = c * cs - (int64_t)(m.t + 1) * is;
        return m;
    };
    // Cell j of the lane's row (0 outside its valid range).
    auto cell = [&](int j, const Column& m) {
        bool ok = (unsigned)(j - f) < width;
        if (kOver) ok = ok && (j < dim_i || r + 1 < H);
        const unsigned i0 = (unsigned)(r - m.t - 1);
        const float* q = mine + m.off;
        const float a = ok && i0 < (unsigned)dim_o ? q[0] : 0.0f;
        const float e = ok && i0 + 1u < (unsigned)dim_o ? q[is] : 0.0f;
        return __fadd_rn(__fmul_rn(m.w, a), __fmul_rn(__fsub_rn(1.0f, m.w), e));
    };
    const int each = ((hi - lo + kRowWarps - 1) / kRowWarps + kRowStep - 1) / kRowStep * kRowStep;
    const int j0 = lo + warp * each, j1 = min(j0 + each, hi);
    // add(v): kRowStep cells of consecutive columns.
    auto walk = [&](auto add) {
        Column next = column(j0 + lane);  // a batch ahead
        for (int jb = j0; jb < j1; jb += 32) {
            Column m = next;
            next = column(jb + 32 + lane);
            const int n = min(32, j1 - jb), n8 = (n + kRowStep - 1) / kRowStep * kRowStep;
            const int ta = __reduce_min_sync(0xffffffffu, lane < n8 ? m.t : INT_MAX);
            const int tb = __reduce_max_sync(0xffffffffu, lane < n8 ? m.t : INT_MIN);
            // Every cell of the 32 rows valid and with both its sources.
            const bool inside = __all_sync(0xffffffffu, f <= jb && l >= jb + n8 && r > tb && r - ta < dim_o) &&
                                (!kOver || jb + n8 <= dim_i);
            if (inside) {
                const float w1 = __fsub_rn(1.0f, m.w);
                m.t = __float_as_int(is > 0 ? w1 : m.w);
                m.w = is > 0 ? m.w : w1;
            }
            __syncwarp();
            meta[warp][lane] = m;
            __syncwarp();
            int k = 0;
            for (; inside && k + kFlight * kRowStep <= n8; k += kFlight * kRowStep) {
                float v[kFlight * kRowStep];
#pragma unroll
                for (int q = 0; q < kFlight * kRowStep; q++) {
                    const Column c = meta[warp][k + q];
                    const float* x = low + c.off;
                    v[q] = __fadd_rn(__fmul_rn(c.w, x[0]), __fmul_rn(__int_as_float(c.t), x[1]));
                }
#pragma unroll
                for (int q = 0; q < kFlight; q++) add(v + q * kRowStep);
            }
            for (; k < n; k += kRowStep) {
                float v[kRowStep];
                if (inside) {
#pragma unroll
                    for (int q = 0; q < kRowStep; q++) {
                        const Column c = meta[warp][k + q];
                        const float* x = low + c.off;
                        v[q] = __fadd_rn(__fmul_rn(c.w, x[0]), __fmul_rn(__int_as_float(c.t), x[1]));
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < kRowStep; q++) v[q] = cell(jb + k + q, meta[warp][k + q]);
                }
                add(v);
            }
        }
    };
    if (kF32) {
        CarriedSum acc;
        walk([&](const float* v) { acc.add(((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]))); });
        sums[0][warp][lane] = acc.sum;
        sums[1][warp][lane] = acc.rest;
        __syncthreads();
        if (warp != 0 || r >= H2) return;
        CarriedSum s;
        for (int k = 0; k < kRowWarps; k++) s.add(make_float2(sums[0][k][lane], sums[1][k][lane]));
        p[r] = {(double)s.value(), 0.0};
        return;
    }
    // Exponents of the cuts; 1.5 * 2^23 units of q added and taken away leave the
    // nearest multiple of q.
    const int ln = 32 - __clz(hi - lo - 1);  // n <= 2^ln
    const int E = (int)(xmax[0] >> 23) - 127 + 1, B = 24 - ln;
    const int e1 = E + 1 - B, e2 = E + 1 - 2 * B, e3 = max(E + 1 - 3 * B, E - 53 + ln);
    bool rest = hi - lo > kMaxExactRow || E < -70 || E > 100;
    if (!rest) {
        const float c1 = __uint_as_float((unsigned)(e1 + 23 + 127) << 23 | 0x400000u);
        const float c2 = __uint_as_float((unsigned)(e2 + 23 + 127) << 23 | 0x400000u);
        const float c3 = __uint_as_float((unsigned)(e3 + 23 + 127) << 23 | 0x400000u);
        const f2 C1 = pk(c1, c1), C2 = pk(c2, c2), C3 = pk(c3, c3);
        f2 s1 = 0, s2 = 0, s3 = 0;
        float left[2] = {0.0f, 0.0f};
        walk([&](const float* v) {
#pragma unroll
            for (int q = 0; q < kRowStep; q += 2) {
                const f2 x = pk(v[q], v[q + 1]);
                const f2 h1 = sub2(add2(x, C1), C1), x1 = sub2(x, h1);
                const f2 h2 = sub2(add2(x1, C2), C2), x2 = sub2(x1, h2);
                const f2 h3 = sub2(add2(x2, C3), C3), x3 = sub2(x2, h3);
                s1 = add2(s1, h1);
                s2 = add2(s2, h2);
                s3 = add2(s3, h3);
                float r0, r1;
                upk(x3, r0, r1);
                left[0] += fabsf(r0);  // not zero, or NaN: something is left
                left[1] += fabsf(r1);
            }
        });
        rest = !(left[0] + left[1] == 0.0f);
        const f2 cut[3] = {s1, s2, s3};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float a, c;
            upk(cut[k], a, c);
            sums[k][warp][lane] = a + c;
        }
    }
    marks[warp][lane] = rest;
    const bool again = __syncthreads_or(rest);
    double s = 0.0;
    if (warp == 0 && !(marks[0][lane] | marks[1][lane] | marks[2][lane] | marks[3][lane])) {
        float t[3];
#pragma unroll
        for (int k = 0; k < 3; k++) t[k] = (sums[k][0][lane] + sums[k][1][lane]) + (sums[k][2][lane] + sums[k][3][lane]);
        s = __dadd_rn(__dadd_rn((double)t[0], (double)t[1]), (double)t[2]);
    }
    if (again) {
        // All rows of the CTA are summed again, the marked ones take the result.
        RowPart part;
        walk([&](const float* v) {
#pragma unroll
            for (int q = 0; q < kRowStep; q++) part.add(v[q]);
        });
        parts[warp][lane] = part;
        __syncthreads();
        if (warp == 0 && (marks[0][lane] | marks[1][lane] | marks[2][lane] | marks[3][lane])) {
#pragma unroll
            for (int k = 1; k < kRowWarps; k++) part.join(parts[k][lane]);
            const bool bad = l - f > kMaxExactRow || part.emax == 0xff ||
                             (part.emin != INT_MAX && (part.emax - part.emin > kMaxSpread || part.mag >= (1ull << 53)));
            s = 0.0;
            if (!bad && part.emin != INT_MAX)
                s = __dmul_rn(__ll2double_rn(part.sum), __longlong_as_double((long long)(part.emin - 150 + 1023) << 52));
            if (bad)
                for (int j = f; j < l; j++) s = __dadd_rn(s, (double)cell(j, column(j)));
        }
    }
    if (warp == 0 && r < H2) p[r] = {s, 0.0};
}

// In-place reference DIF FFT of x[0..n) by one CTA, then bit reversal.
// kFinite (every input finite): butterflies with the twiddle (1, 0) skip the
// multiplication, the others use cmul_finite, and with kRealIn (all imaginary
// parts zero) the first stage multiplies the real difference only.  The values
// are the reference's up to the sign of zero results (finite float-derived
// sums cannot overflow, so no infinity or NaN arises).
template <bool kFinite, bool kRealIn>
__device__ void cta_fft(cd* x, int n, const double* __restrict__ tw) {
    for (int h = n >> 1; h >= 1; h >>= 1) {
        const double* t = tw + 2 * (size_t)(n - 2 * h);
        const bool real_stage = kRealIn && h == (n >> 1);
        for (int k = threadIdx.x; k < (n >> 1); k += blockDim.x) {
            const int l = k & (h - 1);
            const int a = ((k - l) << 1) + l;
            const int bb = a + h;
            const cd xa = x[a], xb = x[bb];
            if (!kFinite) {
                x[a] = cadd(xa, xb);
                x[bb] = cmul(csub(xa, xb), cd{t[2 * l], t[2 * l + 1]});
            } else if (real_stage) {
                const double dr = __dsub_rn(xa.re, xb.re);
                x[a] = cd{__dadd_rn(xa.re, xb.re), 0.0};
                x[bb] = cd{__dmul_rn(dr, t[2 * l]), __dmul_rn(dr, t[2 * l + 1])};
            } else {
                x[a] = cadd(xa, xb);
                x[bb] = l == 0 ? csub(xa, xb) : cmul_finite(csub(xa, xb), cd{t[2 * l], t[2 * l + 1]});
            }
        }
        __syncthreads();
    }
    const unsigned bits = 31 - __clz(n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int j = (int)bitrev((unsigned)i, bits);
        if (j > i) {
            const cd tmp = x[i];
            x[i] = x[j];
            x[j] = tmp;
        }
    }
    __syncthreads();
}

// Ramp filter: i > H/2 -> 0, else (i/H) * P_i (real scalar times complex),
// then the conjugation that starts the inverse transform (helper.h:110).
__device__ void ramp_filter(cd* x, int H, int H2) {
    for (int i = threadIdx.x; i < H2; i += blockDim.x) {
        cd v = x[i];
        if (i > H / 2) {
            v = {0.0, 0.0};
        } else {
            const double s = __ddiv_rn((double)i, (double)H);
            v = {__dmul_rn(v.re, s), __dmul_rn(v.im, s)};
        }
        x[i] = {v.re, -v.im};
    }
    __syncthreads();
}

// Filtered row value i of a sector, as the deskew reads it.
__device__ __forceinline__ void store_row(cd* p, int i, double q) {
    reinterpret_cast<RowValue*>(p)[i] = RowValue{q, __double2float_rn(__dadd_rn(0.0, q))};
}

// One CTA per sector.  Sectors with H2 <= kSmemH2 transform a copy of their
// row sums in shared memory (smem > 0), larger ones work in place in P.  The
// final division by H2 (kernelRADN.h:255) is a multiplication by the exact
// power of two 1/H2: the same correctly rounded quotient.
constexpr int kTransformThreads = 256;
constexpr int kSmemH2 = 8192;

__global__ void __launch_bounds__(kTransformThreads)
    k_radon_transform(DevGeometry g, Batch b, cd* __restrict__ P, int64_t pstride,
                      const double* __restrict__ twiddles, const int64_t* __restrict__ tw_off, int smem) {
    extern __shared__ cd xs[];
    const int slot = blockIdx.x;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int H = d.H;
    const int H2 = pow2_at_least(H);
    cd* p = P + slot * pstride;
    cd* x = smem ? xs : p;
    const double* tw = twiddles + tw_off[31 - __clz(H2)];
    int bad = 0;
    for (int i = threadIdx.x; i < H2; i += blockDim.x) {
        const cd v = p[i];
        if (smem) x[i] = v;
        bad |= !isfinite(v.re);
    }
    if (!__syncthreads_or(bad)) {
        cta_fft<true, true>(x, H2, tw);
        ramp_filter(x, H, H2);
        cta_fft<true, false>(x, H2, tw);
    } else {
        cta_fft<false, false>(x, H2, tw);
        ramp_filter(x, H, H2);
        cta_fft<false, false>(x, H2, tw);
    }
    // conj, then divide by H2: only the real part is used (kernelRADN.h:255).
    const double inv = 1.0 / (double)H2;
    for (int i = threadIdx.x; i < H; i += blockDim.x) store_row(p, i, __dmul_rn(x[i].re, inv));
}

// The same transform by a cluster of four CTAs per sector.  After its first two
// stages a decimation-in-frequency transform is four independent ones of a
// quarter of the size, so each CTA forms its quarter's input from the row sums
// (which all four read) and transforms it: CTA c holds the spectrum's lines i =
// rev2(c) mod 4 (rev2 swaps the two bits).  The ramp filter and the first two
// stages of the inverse stay within a residue mod 4 too; their results go to the
// CTAs of the four quarters through distributed shared memory, and each ends
// with the rows of its residue.  Every value is formed by the operations of
// k_radon_transform (up to the sign of zeros where all inputs are finite).
// One CTA per sector left 28 of 180 sectors to a second round of the 152 SMs and
// its barriers to a lone CTA: 75 us per 512 x 512 image, so 52 us; the
// binary64 operations take 27 us at the pipe's rate.
constexpr int kQuad = 4;
constexpr int kQuadThreads = 128;
constexpr int kQuadMinH2 = 64;

// One DIF butterfly (a, b) with twiddle t (one: it is (1, 0)).
template <bool kFinite>
__device__ __forceinline__ void dif(cd& a, cd& b, const double* __restrict__ t, bool one) {
    const cd d = csub(a, b);
    a = cadd(a, b);
    if (kFinite) b = one ? d : cmul_finite(d, cd{t[0], t[1]});
    else b = cmul(d, cd{t[0], t[1]});
}

template <bool kFinite>
__device__ void quad_transform(cd* x, cd* y, const double* sums, int H, int n, const double* __restrict__ tw,
                               unsigned rank, RowValue* out, cooperative_groups::cluster_group& cluster) {
    const int n4 = n >> 2, n8 = n >> 3, n16 = n >> 4;
    const double* t1 = tw;                  // half-span n / 2
    const double* t2 = tw + 2 * (n - n / 2);  // half-span n / 4
    const double* tq = tw + 2 * (n - n4);   // the quarters' transforms
    const int res = ((rank & 1) << 1) | (rank >> 1);
    // This quarter's input, from the real row sums.
    for (int k = threadIdx.x; k < n4; k += kQuadThreads) {
        cd v[2];  // the half's entries k and k + n/4
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int l = k + u * n4;
            const double a = sums[l], b = sums[l + 2 * n4];
            if (!(rank & 2)) v[u] = cd{__dadd_rn(a, b), 0.0};
            else if (kFinite) v[u] = cd{__dmul_rn(__dsub_rn(a, b), t1[2 * l]), __dmul_rn(__dsub_rn(a, b), t1[2 * l + 1])};
            else v[u] = cmul(csub(cd{a, 0.0}, cd{b, 0.0}), cd{t1[2 * l], t1[2 * l + 1]});
            if (!kFinite && !(rank & 2)) v[u] = cadd(cd{a, 0.0}, cd{b, 0.0});
        }
        dif<kFinite>(v[0], v[1], t2 + 2 * k, k == 0);
        x[k] = v[rank & 1];
    }
    __syncthreads();
    cta_fft<kFinite, false>(x, n4, tq);
    // Ramp filter and conjugation: line i = 4 q + res, 0 past H / 2.
    for (int q = threadIdx.x; q < n4; q += kQuadThreads) {
        const int i = 4 * q + res;
        cd v = x[q];
        if (i > H / 2) {
            v = {0.0, 0.0};
        } else {
            const double s = __ddiv_rn((double)i, (double)H);
            v = {__dmul_rn(v.re, s), __dmul_rn(v.im, s)};
        }
        x[q] = {v.re, -v.im};
    }
    cluster.sync();  // every CTA runs, and this one's lines are filtered
    // First two stages of the inverse for k = 4 q + res < n/4, to the quarters.
    for (int q = threadIdx.x; q < n16; q += kQuadThreads) {
        const int k = 4 * q + res;
        cd x0 = x[q], x1 = x[q + n16], x2 = x[q + n8], x3 = x[q + n8 + n16];
        dif<kFinite>(x0, x2, t1 + 2 * k, k == 0);
        dif<kFinite>(x1, x3, t1 + 2 * (k + n4), false);
        dif<kFinite>(x0, x1, t2 + 2 * k, k == 0);
        dif<kFinite>(x2, x3, t2 + 2 * k, k == 0);
        cluster.map_shared_rank(y, 0)[k] = x0;
        cluster.map_shared_rank(y, 1)[k] = x1;
        cluster.map_shared_rank(y, 2)[k] = x2;
        cluster.map_shared_rank(y, 3)[k] = x3;
    }
    cluster.sync();  // every quarter is complete; no CTA reaches into another after this
    cta_fft<kFinite, false>(y, n4, tq);
    const double inv = 1.0 / (double)n;
    for (int q = threadIdx.x; q < n4; q += kQuadThreads)
        if (4 * q + res < H) store_row(reinterpret_cast<cd*>(out), 4 * q + res, __dmul_rn(y[q].re, inv));
}

__global__ void __cluster_dims__(kQuad, 1, 1) __launch_bounds__(kQuadThreads)
    k_radon_transform_quad(DevGeometry g, Batch b, cd* __restrict__ P, int64_t pstride,
                           const double* __restrict__ twiddles, const int64_t* __restrict__ tw_off) {
    extern __shared__ cd xq[];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int slot = blockIdx.x / kQuad;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int H = d.H, H2 = pow2_at_least(H);
    cd* p = P + slot * pstride;
    cd* x = xq;
    cd* y = xq + (H2 >> 2);
    double* sums = reinterpret_cast<double*>(y + (H2 >> 2));
    int bad = 0;
    for (int i = threadIdx.x; i < H2; i += kQuadThreads) {
        const double v = p[i].re;
        sums[i] = v;
        bad |= !isfinite(v);
    }
    bad = __syncthreads_or(bad);
    const double* tw = twiddles + tw_off[31 - __clz(H2)];
    RowValue* out = reinterpret_cast<RowValue*>(p);
    if (!bad) quad_transform<true>(x, y, sums, H, H2, tw, rank, out, cluster);
    else quad_transform<false>(x, y, sums, H, H2, tw, rank, out, cluster);
}

// The whole Radon operator of a sector whose rows stay within its width, in
// one launch: a cluster of kClusterCtas CTAs per sector.  Every CTA of the
// cluster forms exact row sums (as k_radon_sums, gathering the skewed cells
// from the oriented input) for its share of the rows and stores them straight
// into the leader CTA's shared memory (distributed shared memory); after the
// cluster barrier the leader applies the transform, ramp filter and inverse
// transform in place (as k_radon_transform) and writes the filtered row values
// q to P, which the deskew reads.  The other CTAs exit at the barrier, so
// their SM slots take other sectors' sums while the leaders run the binary64
// transforms.  Bit-identical to the three-launch path.
constexpr int kClusterCtas = 8;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kTransformThreads, 6)
    k_radon_sector(DevGeometry g, Batch b, const float* __restrict__ orient, int64_t n_cells, cd* __restrict__ P,
                   int64_t pstride, const double* __restrict__ twiddles, const int64_t* __restrict__ tw_off) {
    namespace cg = cooperative_groups;
    extern __shared__ cd xs[];
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.y;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int H = d.H;
    const int H2 = pow2_at_least(H);
    const float* src = orient + (int64_t)d.type * n_cells;
    const int32_t* tgt = g.target + d.col_off;
    const float* wgt = g.weight + d.col_off;
    cd* x0 = cluster.map_shared_rank(xs, 0);  // the leader's buffer
    constexpr int kWarps = kTransformThreads / 32;
    for (int r = rank * kWarps + (threadIdx.x >> 5); r < H2; r += kClusterCtas * kWarps) {
        if (r >= H) {
            if (lane == 0) x0[r] = {0.0, 0.0};
            continue;
        }
        const int f = g.first[d.row_off + r], l = g.last[d.row_off + r];
        ExactPart a;
#pragma unroll 2
        for (int j = f + lane; j < l; j += 32) a.add(skew_gather(d, tgt, wgt, src, r, j));
        const bool lane_bad = a.bad();
        int gmin = a.emin, gmax = a.emax;
        for (int o = 16; o > 0; o >>= 1) {
            gmin = min(gmin, __shfl_xor_sync(0xffffffffu, gmin, o));
            gmax = max(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
        }
        bool bad = __any_sync(0xffffffffu, lane_bad) || l - f > kMaxExactRow ||
                   (gmin != INT_MAX && gmax - gmin > kMaxSpread);
        double s = 0.0;
        if (!bad && gmin != INT_MAX) {
            const int sh = a.emin == INT_MAX ? 0 : a.emin - gmin;
            unsigned long long pos = shl64(a.pos, sh), neg = shl64(a.neg, sh);
            for (int o = 16; o > 0; o >>= 1) {
                pos += __shfl_xor_sync(0xffffffffu, pos, o);
                neg += __shfl_xor_sync(0xffffffffu, neg, o);
            }
            if (pos + neg < (1ull << 53)) {
                const double scale = __longlong_as_double((long long)(gmin - 150 + 1023) << 52);
                s = __dmul_rn(__ll2double_rn((long long)(pos - neg)), scale);
            } else {
                bad = true;
            }
        }
        if (bad && lane == 0)
            for (int j = f; j < l; j++) s = __dadd_rn(s, (double)skew_gather(d, tgt, wgt, src, r, j));
        if (lane == 0) x0[r] = {s, 0.0};
    }
    cluster.sync();  // every row sum is in the leader's shared memory
    if (rank != 0) return;
    const double* tw = twiddles + tw_off[31 - __clz(H2)];
    int bad = 0;
    for (int i = threadIdx.x; i < H2; i += blockDim.x) bad |= !isfinite(xs[i].re);
    if (!__syncthreads_or(bad)) {
        cta_fft<true, true>(xs, H2, tw);
        ramp_filter(xs, H, H2);
        cta_fft<true, false>(xs, H2, tw);
    } else {
        cta_fft<false, false>(xs, H2, tw);
        ramp_filter(xs, H, H2);
        cta_fft<false, false>(xs, H2, tw);
    }
    cd* p = P + slot * pstride;
    const double inv = 1.0 / (double)H2;
    for (int i = threadIdx.x; i < H; i += blockDim.x) store_row(p, i, __dmul_rn(xs[i].re, inv));
}

// ---- float32 mode (SKE_FLAG_RADON_F32) -------------------------------------
// The same operator on the FP32 pipes: row sums in float (a warp per row,
// lanes over columns, a shuffle tree), the radix-2 DIF transform, ramp filter
// and inverse transform in float in shared memory (twiddles rounded from the
// binary64 table), the filtered row values written to P as doubles for the
// deskew or back-projection.  Values differ from the reference's binary64 in
// their low bits (the sums' order and float rounding); the relative error of
// the output is measured and stated (tests/test_gpu_parity.py).
__global__ void __launch_bounds__(kSumWarps * 32)
    k_radon_sums_f32(DevGeometry g, Batch b, const float* __restrict__ SI, int64_t stride, cd* __restrict__ P,
                     int64_t pstride) {
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.y;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int H2 = pow2_at_least(d.H);
    const float* in = SI + slot * stride;
    cd* p = P + slot * pstride;
    const int nwarps = gridDim.x * kSumWarps;
    for (int r = blockIdx.x * kSumWarps + (threadIdx.x >> 5); r < H2; r += nwarps) {
        if (r >= d.H) {
            if (lane == 0) p[r] = {0.0, 0.0};
            continue;
        }
        const int f = g.first[d.row_off + r], l = g.last[d.row_off + r];
        const float* row = in + (int64_t)r * d.dim_i;
        float acc = 0.0f;
        for (int j = f + lane; j < l; j += 32) acc += row[j];
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) p[r] = {(double)acc, 0.0};
    }
}

__device__ void cta_fft_f32(float2* x, int n, const double* __restrict__ tw) {
    for (int h = n >> 1; h >= 1; h >>= 1) {
        const double* t = tw + 2 * (size_t)(n - 2 * h);
        for (int k = threadIdx.x; k < (n >> 1); k += blockDim.x) {
            const int l = k & (h - 1);
            const int a = ((k - l) << 1) + l;
            const int bb = a + h;
            const float2 xa = x[a], xb = x[bb];
            const float dr = xa.x - xb.x, di = xa.y - xb.y;
            const float c = (float)t[2 * l], sn = (float)t[2 * l + 1];
            x[a] = make_float2(xa.x + xb.x, xa.y + xb.y);
            x[bb] = make_float2(dr * c - di * sn, dr * sn + di * c);
        }
        __syncthreads();
    }
    const unsigned bits = 31 - __clz(n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int j = (int)bitrev((unsigned)i, bits);
        if (j > i) {
            const float2 tmp = x[i];
            x[i] = x[j];
            x[j] = tmp;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kTransformThreads)
    k_radon_transform_f32(DevGeometry g, Batch b, cd* __restrict__ P, int64_t pstride,
                          const double* __restrict__ twiddles, const int64_t* __restrict__ tw_off) {
    extern __shared__ float2 xf[];
    const int slot = blockIdx.x;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int H = d.H;
    const int H2 = pow2_at_least(H);
    cd* p = P + slot * pstride;
    const double* tw = twiddles + tw_off[31 - __clz(H2)];
    for (int i = threadIdx.x; i < H2; i += blockDim.x) xf[i] = make_float2((float)p[i].re, 0.0f);
    __syncthreads();
    cta_fft_f32(xf, H2, tw);
    for (int i = threadIdx.x; i < H2; i += blockDim.x) {  // ramp filter, then the conjugation
        float2 v = xf[i];
        if (i > H / 2) {
            v = make_float2(0.0f, 0.0f);
        } else {
            const float sc = __fdiv_rn((float)i, (float)H);
            v = make_float2(v.x * sc, v.y * sc);
        }
        xf[i] = make_float2(v.x, -v.y);
    }
    __syncthreads();
    cta_fft_f32(xf, H2, tw);
    const float inv = 1.0f / (float)H2;
    for (int i = threadIdx.x; i < H; i += blockDim.x) store_row(p, i, (double)(xf[i].x * inv));
}

__global__ void k_radon_backproject(DevGeometry g, Batch b, const cd* __restrict__ P, int64_t pstride,
                                    float* __restrict__ SO, int64_t stride, int64_t len) {
    const int slot = blockIdx.y;
    const SectorDesc d = g.desc[b.angle[slot]];
    const int32_t* first = g.first + d.row_off;
    const int32_t* last = g.last + d.row_off;
    const cd* q = P + slot * pstride;
    float* out = SO + slot * stride;
    for (int64_t p = gtid(); p < len; p += gstride()) {
        // Rows that can cover p, in increasing order (`+=` in row order).
        int rhi = (int)(p / d.dim_i);
        if (rhi > d.H - 1) rhi = d.H - 1;
        int64_t lo_row = (p - d.diml) / d.dim_i;
        int rlo = lo_row < 0 ? 0 : (int)lo_row;
        float v = 0.0f;
        for (int r = rlo; r <= rhi; r++) {
            const int64_t base = (int64_t)r * d.dim_i;
            if (p >= base + first[r] && p < base + last[r]) v = (float)__dadd_rn((double)v, q[r].re);
        }
        out[p] = v;
    }
}

}  // namespace

// 0: the fused sector kernel where it applies; 1 (default): row sums and
// transform as two launches, measured faster (radon_select).
int g_radon_path = 1;

int radon_launches(bool rows_only, int max_H2, bool f32, bool in_width) {
    if (f32 && max_H2 <= kSmemH2) return rows_only ? 2 : 3;
    return rows_only ? (in_width && max_H2 <= kSmemH2 && g_radon_path == 0 ? 1 : 2) : 3;
}

int radon_select(int path) {
    if (path != 0 && path != 1) return -1;
    g_radon_path = path;
    return 0;
}

cudaError_t launch_radon(const DevGeometry& g, const Batch& b, const float* SI, float* SO, int64_t stride,
                         int64_t len, double* P, int64_t pstride, const double* twiddles, const int64_t* tw_off,
                         int max_H2, cudaStream_t st, bool backproject, const float* orient, int64_t n_cells,
                         int dimx, int dimy, const unsigned* xmax, bool f32, bool in_width) {
    if (orient && backproject) return cudaErrorInvalidValue;  // the gathered cells are not kept for SO
    cd* Pc = reinterpret_cast<cd*>(P);
    if (f32 && max_H2 <= kSmemH2) {
        dim3 g1((max_H2 + kSumWarps - 1) / kSumWarps, b.count), gr((max_H2 + 31) / 32, b.count);
        if (orient) {
            const bool few = (int64_t)gr.x * gr.y <= kRowFewCtas;
            auto kern = in_width ? (few ? k_radon_rows<true, false, 4> : k_radon_rows<true, false, 2>)
                                 : (few ? k_radon_rows<true, true, 4> : k_radon_rows<true, true, 2>);
            kern<<<gr, kRowWarps * 32, 0, st>>>(g, b, orient, n_cells, dimx, dimy, xmax, Pc, pstride);
        } else {
            k_radon_sums_f32<<<g1, kSumWarps * 32, 0, st>>>(g, b, SI, stride, Pc, pstride);
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        const int smem = max_H2 * (int)sizeof(float2);
        if (smem > 48 * 1024) {
            e = allow_smem(k_radon_transform_f32, smem);
            if (e != cudaSuccess) return e;
        }
        k_radon_transform_f32<<<b.count, kTransformThreads, smem, st>>>(g, b, Pc, pstride, twiddles, tw_off);
        e = cudaGetLastError();
        if (e != cudaSuccess || !backproject) return e;
        int64_t blocks = (len + 255) / 256;
        if (blocks > 4096) blocks = 4096;
        k_radon_backproject<<<dim3((unsigned)blocks, b.count), 256, 0, st>>>(g, b, Pc, pstride, SO, stride, len);
        return cudaGetLastError();
    }
    if (orient && in_width && max_H2 <= kSmemH2 && g_radon_path == 0) {  // one fused launch: a cluster per sector
        const int smem = max_H2 * (int)sizeof(cd);
        cudaError_t e = cudaSuccess;
        if (smem > 48 * 1024) e = allow_smem(k_radon_sector, smem);
        if (e != cudaSuccess) return e;
        k_radon_sector<<<dim3(kClusterCtas, b.count), kTransformThreads, smem, st>>>(g, b, orient, n_cells, Pc, pstride,
                                                                                   twiddles, tw_off);
        return cudaGetLastError();
    }
    dim3 g1((max_H2 + kSumWarps - 1) / kSumWarps, b.count), gr((max_H2 + 31) / 32, b.count);
    if (orient && in_width)
        k_radon_rows<false, false, 2><<<gr, kRowWarps * 32, 0, st>>>(g, b, orient, n_cells, dimx, dimy, xmax, Pc, pstride);
    else if (orient)
        k_radon_rows<false, true, 2><<<gr, kRowWarps * 32, 0, st>>>(g, b, orient, n_cells, dimx, dimy, xmax, Pc, pstride);
    else
        k_radon_sums<<<g1, kSumWarps * 32, 0, st>>>(g, b, SI, stride, Pc, pstride);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // H >= dim_o: every sector's transform is at least this long.
    int min_H2 = 1;
    while (min_H2 < dimx && min_H2 < dimy) min_H2 <<= 1;
    if (max_H2 <= kSmemH2 && min_H2 >= kQuadMinH2) {  // H2 / 4 entries twice, and H2 row sums
        const int smem = max_H2 * (int)(sizeof(cd) / 2 + sizeof(double));
        if (smem > 48 * 1024) {
            e = allow_smem(k_radon_transform_quad, smem);
            if (e != cudaSuccess) return e;
        }
        k_radon_transform_quad<<<kQuad * b.count, kQuadThreads, smem, st>>>(g, b, Pc, pstride, twiddles, tw_off);
        e = cudaGetLastError();
        if (e != cudaSuccess || !backproject) return e;
        int64_t blocks = (len + 255) / 256;
        if (blocks > 4096) blocks = 4096;
        k_radon_backproject<<<dim3((unsigned)blocks, b.count), 256, 0, st>>>(g, b, Pc, pstride, SO, stride, len);
        return cudaGetLastError();
    }
    const int smem = max_H2 <= kSmemH2 ? max_H2 * (int)sizeof(cd) : 0;
    if (smem > 48 * 1024) {
        e = allow_smem(k_radon_transform, smem);
        if (e != cudaSuccess) return e;
    }
    k_radon_transform<<<b.count, kTransformThreads, smem, st>>>(g, b, Pc, pstride, twiddles, tw_off, smem);
    e = cudaGetLastError();
    if (e != cudaSuccess || !backproject) return e;
    int64_t blocks = (len + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    k_radon_backproject<<<dim3((unsigned)blocks, b.count), 256, 0, st>>>(g, b, Pc, pstride, SO, stride, len);
    return cudaGetLastError();
}

}  // namespace ske
