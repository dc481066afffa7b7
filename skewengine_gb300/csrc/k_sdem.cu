// Total-viewshed line-of-sight sweep (kernelSDEM, src/kernelSDEM.h:168-222).
//
// For every valid cell j of a skewed row (the observer) the reference scans the
// row forward (k = j+1 ..) and backward (k = j-1 ..), tracking the horizon slope
// max((S[k] - h)/d) with h = S[j] + POVh; each step is visible when its slope
// beats the horizon, and every visible run that closes before the row end adds
// d_close^2 - d_open^2 to cv.  The output is cv * (float)scale^2.
//
// This is the chunked sweep, whose only scratch is its work list: it serves the
// allocation-free entry point.  The engine's runs take the compacting sweep
// (k_sweep.cu), whose survivor lists grow with the grid.
//  * Persistent kernel; a warp takes one work item = (sector slot, skewed row,
//    chunk of 128 consecutive observers) from a global queue ordered longest row
//    first.  Every lane owns 4 consecutive observers.
//  * The row is staged in shared memory once per item; lanes read it through a
//    register sliding window refilled by one aligned 16-byte load per 4 steps,
//    so shared-memory traffic is 1 byte per observer-step.
//  * The step distance d is warp-uniform, so -d, RN(1/d) and 2d+1 come from a
//    constant-memory table.  The slopes of two observers at a time use packed
//    f32x2 instructions (div2, sdem_math.cuh).
//  * Accumulation: a closed visible run [o, c) contributes c^2 - o^2 to the
//    reference's cv, which is the sum of the ring areas 2d+1 over its steps
//    d = o .. c-1.  So each visible step adds 2d+1 to a running sum acc, and
//    every invisible step (the one that closes a run, or any later one) copies
//    acc into cl, the sum over closed runs.  The initial run starts at distance
//    0 (ring 1 not swept), hence cl starts at -1 and cv = 1 + cl; a run still
//    open at the row end never reaches cl, exactly as the reference does not
//    count it.  All values are integers below 2^24 for rows up to 4096 cells,
//    so the float result is exact and equal to the reference's.  Longer rows
//    use the reference-order path.
//  * Horizon pruning (exact): after step d the remaining targets (distances
//    d+1 .. n) are all invisible when the bound b = fl(a/(d+1)), a >= 0, is at
//    most the horizon, with a = fl(Smax - h) and Smax an upper bound of the
//    remaining heights from per-8-cell suffix (forward) and prefix (backward)
//    maxima.  Rounding is monotonic, so every remaining slope fl(fl(S[k]-h)/d')
//    is at most fl(a/d'), and a/d' is largest at d' = d+1.  An observer that
//    passes is finished: every later step would be invisible, so cv = 1 + sum
//    (its last run closes at the next step).  Tested every kCheck steps; a warp
//    stops when all its observers are finished.
#include <algorithm>
#include <vector>

#include "sdem_math.cuh"

namespace ske {

namespace {

constexpr int kChunk = 128;        // observers per work item (4 per lane)
constexpr int kWarps = 8;          // warps per CTA
constexpr int kPadFront = 136;     // zero cells before the row (backward window overrun)
constexpr int kPadBack = 144;      // zero cells after the row (forward window overrun)
constexpr int kBlk = 8;            // cells per block of the pruning maxima
constexpr int kCheck = 32;         // steps between pruning tests (multiple of 4)

// {-d, RN(1/d), 2d+1, d+1} for d = 0..4095 (entry 0 unused).
__constant__ float4 c_step[kFastMaxRow];

__host__ __device__ inline int row_pad(int max_row) { return kPadFront + ((max_row + 3) & ~3) + kPadBack; }
__host__ __device__ inline int blocks_pad(int max_row) { return ((max_row + kBlk - 1) / kBlk + 3) & ~3; }
// Shared floats per warp: the padded row plus suffix and prefix block maxima.
__host__ __device__ inline int warp_floats(int max_row) { return row_pad(max_row) + 2 * blocks_pad(max_row); }

// State of the 4 observers of a lane in one scan direction.  acc is the ring
// sum of all visible steps; cl is acc at the last invisible step, i.e. the ring
// sum of the closed runs (-1 before any: the initial run starts at distance 0).
struct Scan4 {
    float h[4], mx[4], acc[4], cl[4];
    int n[4];        // steps of each observer (-1: observer outside the row)
    bool done[4];    // finished by pruning
};

// One block of 4 steps d = d0 .. d0+3.  The window holds the 8 row values the
// block needs: forward w = A[x0+d0 .. x0+d0+7], step e of observer q reads
// w[e+q]; backward w = A[x0-d0-4 .. x0-d0+3], step e reads w[q-e+4].  Slopes of
// observer pairs (0,1) and (2,3) use packed f32x2 operations; the horizon test,
// the horizon update and the two sums are per observer.
template <bool kFwd, bool kTail>
__device__ __forceinline__ void block4(Scan4& s, const float w[8], int d0) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int d = d0 + e;
        if (d == 0) continue;  // only in the first block
        const float4 st = c_step[d];
        const f2 nd2 = pk(st.x, st.x), y2 = pk(st.y, st.y);
        const float ring = st.z;
        float qv[4];
#define SKE_W(q) (kFwd ? w[e + (q)] : w[(q)-e + 4])
        upk(div2(sub2(pk(SKE_W(0), SKE_W(1)), pk(s.h[0], s.h[1])), nd2, y2), qv[0], qv[1]);
        upk(div2(sub2(pk(SKE_W(2), SKE_W(3)), pk(s.h[2], s.h[3])), nd2, y2), qv[2], qv[3]);
#undef SKE_W
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (kTail && d > s.n[q]) continue;
            const bool above = qv[q] > s.mx[q];
            s.mx[q] = above ? qv[q] : s.mx[q];
            s.cl[q] = above ? s.cl[q] : s.acc[q];
            s.acc[q] = above ? __fadd_rn(s.acc[q], ring) : s.acc[q];
        }
    }
}

// Pruning test after step dc for the 4 observers: smax is an upper bound of
// every remaining target height of all four.
__device__ __forceinline__ void prune4(Scan4& s, float smax, int dc) {
    const float4 st = c_step[dc + 1];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float a = __fsub_rn(smax, s.h[q]);
        const float b = div_fast(a, st.x, st.y);
        s.done[q] = s.done[q] || (dc < s.n[q] && a >= 0.0f && b <= s.mx[q]);
    }
}

// Scan of the lane's observers x0..x0+3 in one direction (fast path).
// A: the row (16-byte aligned, zero padded), bmax: suffix (forward) or prefix
// (backward) maxima of kBlk-cell blocks.
template <bool kFwd>
__device__ __forceinline__ void scan_fast(const float* __restrict__ A, const float* __restrict__ bmax, int x0, int L,
                                          float povh, float cv[4]) {
    Scan4 s;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int x = x0 + q;
        s.n[q] = x < L ? (kFwd ? L - 1 - x : x) : -1;
        s.h[q] = __fadd_rn(A[x], povh);
        s.mx[q] = -2000.0f;
        s.acc[q] = 0.0f;
        s.cl[q] = -1.0f;
        s.done[q] = false;
    }
    // Steps every observer of the warp takes (no bounds test) and the most any takes.
    const int lane_min = kFwd ? s.n[3] : s.n[0];
    const int lane_max = max(max(s.n[0], s.n[1]), max(max(s.n[2], s.n[3]), 0));
    const int dmain = __reduce_min_sync(0xffffffffu, lane_min < 0 ? 0 : lane_min);
    const int dall = __reduce_max_sync(0xffffffffu, lane_max);
    const float4* A4 = reinterpret_cast<const float4*>(A) + (x0 >> 2);
    float4 cur = A4[0];
    for (int m = 0; 4 * m <= dall; m++) {
        const float4 nx = kFwd ? A4[m + 1] : A4[-m - 1];
        const float4 lo = kFwd ? cur : nx, hi = kFwd ? nx : cur;
        const float w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        if (4 * m + 3 <= dmain) block4<kFwd, false>(s, w, 4 * m);
        else block4<kFwd, true>(s, w, 4 * m);
        cur = nx;
        const int dc = 4 * m + 3;
        if ((dc + 1) % kCheck == 0 && dc < dall) {
            // Remaining targets: forward x+dc+1 .., backward .. x-dc-1 (all four
            // observers' targets lie on the same side of the bound's block).
            // Backward: the lane's largest in-row observer bounds its targets.
            const int k = kFwd ? x0 + dc + 1 : min(x0 + 3, L - 1) - dc - 1;
            if (kFwd ? k < L : k >= 0) prune4(s, bmax[k / kBlk], dc);
            bool fin = true;
#pragma unroll
            for (int q = 0; q < 4; q++) fin = fin && (s.done[q] || dc >= s.n[q]);
            if (__all_sync(0xffffffffu, fin)) break;
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (s.n[q] < 0) {
            cv[q] = 0.0f;
            continue;
        }
        // A pruned observer's open run closes at its next step: every run counts.
        cv[q] = __fadd_rn(1.0f, s.done[q] ? s.acc[q] : s.cl[q]);
    }
}

// Block maxima for pruning: suf[b] = max A[kBlk*b ..] (to the row end),
// pre[b] = max A[.. kBlk*b + kBlk-1] (from the row start).  Rows on the fast
// path are finite.
__device__ void block_maxima(const float* __restrict__ A, int L, float* suf, float* pre, int lane) {
    const float ninf = __int_as_float(0xff800000);
    const int nb = (L + kBlk - 1) / kBlk;
    const int per = (nb + 31) / 32;
    const int b0 = lane * per, b1 = min(b0 + per, nb);
    float run = ninf;
    for (int b = b0; b < b1; b++) {  // block maxima, then lane-local prefix
        float m = ninf;
        for (int c = b * kBlk; c < min(b * kBlk + kBlk, L); c++) m = fmaxf(m, A[c]);
        suf[b] = m;
        run = fmaxf(run, m);
        pre[b] = run;
    }
    // Inclusive prefix / suffix max of the lane totals (Hillis-Steele), then
    // shift by one lane for the exclusive values.
    float inc_p = run, inc_s = run;
    for (int off = 1; off < 32; off <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, inc_p, off);
        const float dn = __shfl_down_sync(0xffffffffu, inc_s, off);
        if (lane >= off) inc_p = fmaxf(inc_p, up);
        if (lane + off < 32) inc_s = fmaxf(inc_s, dn);
    }
    float before = __shfl_up_sync(0xffffffffu, inc_p, 1);
    float after = __shfl_down_sync(0xffffffffu, inc_s, 1);
    if (lane == 0) before = ninf;
    if (lane == 31) after = ninf;
    float r = after;
    for (int b = b1 - 1; b >= b0; b--) {
        r = fmaxf(r, suf[b]);
        suf[b] = r;
    }
    for (int b = b0; b < b1; b++) pre[b] = fmaxf(pre[b], before);
}

__global__ void __launch_bounds__(kWarps * 32) k_sdem_chunked(SdemLaunch a) {
    extern __shared__ float4 smem4[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wf = warp_floats(a.max_row);
    float* buf = reinterpret_cast<float*>(smem4) + (size_t)warp * wf;
    float* A = buf + kPadFront;
    float* suf = buf + row_pad(a.max_row);
    float* pre = suf + blocks_pad(a.max_row);
    for (;;) {
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(a.counter, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if ((int64_t)idx >= a.n_items) break;
        const Item it = decode(a.items[idx]);
        const SectorDesc& d = a.g.desc[a.b.angle[it.slot]];
        const int32_t* first = a.g.first + d.row_off;
        const int32_t* last = a.g.last + d.row_off;
        const int f = first[it.row];
        const int L = last[it.row] - f;
        if (L > a.max_row || L <= 0) {
            if (lane == 0) atomicExch(a.status, 1);
            continue;
        }
        const int64_t rowbase = (int64_t)it.row * d.dim_i + f;  // flat index of the row start
        const float* src = a.SI + it.slot * a.stride + rowbase;
        bool ok = true;
        for (int x = lane; x < L; x += 32) {
            const float v = src[x];
            A[x] = v;
            ok = ok && div_safe(v) && div_safe(__fadd_rn(v, a.povh));
        }
        for (int x = lane; x < kPadFront; x += 32) buf[x] = 0.0f;
        const int tail_end = ((L + 3) & ~3) + kPadBack;
        for (int x = L + lane; x < tail_end; x += 32) A[x] = 0.0f;
        const bool fast = __all_sync(0xffffffffu, ok) && L <= kFastMaxRow && div_safe(a.povh);
        __syncwarp();
        if (fast) {
            block_maxima(A, L, suf, pre, lane);
            __syncwarp();
        }

        const int x0 = it.chunk * kChunk + 4 * lane;
        float cv[4];
        if (fast) {
            float cb[4];
            scan_fast<true>(A, suf, x0, L, a.povh, cv);
            scan_fast<false>(A, pre, x0, L, a.povh, cb);
#pragma unroll
            for (int q = 0; q < 4; q++) cv[q] = __fadd_rn(cv[q], cb[q]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) cv[q] = (x0 + q < L) ? scan_reference(A, x0 + q, L, a.povh) : 0.0f;
        }
        float* out = a.SO + it.slot * a.stride;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int x = x0 + q;
            if (x >= L) continue;
            const int64_t p = rowbase + x;
            if (owner_row(d, first, last, p) != it.row) continue;
            out[p] = a.counts_only ? cv[q] : __fmul_rn(cv[q], d.r2);
        }
        __syncwarp();
    }
}

// Exhaustive check of div_fast against IEEE division: every float bit pattern a
// with div_safe-compatible magnitude (zero or |a| in [2^-103, 2^91], the range
// of S[k]-h when both operands pass div_safe) and every d in [1, dmax].
__global__ void k_div_check(int dmax, unsigned long long* checked, unsigned long long* bad,
                            unsigned* first_bad) {
    unsigned long long n_ok = 0, n_bad = 0;
    for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < (1ull << 32);
         u += (uint64_t)gridDim.x * blockDim.x) {
        const float a = __uint_as_float((unsigned)u);
        const float m = fabsf(a);
        // 0x0c000000 = 2^-103, 0x6d000000 = 2^91; NaN fails both comparisons.
        if (!(a == 0.0f || (m >= __uint_as_float(0x0c000000u) && m <= __uint_as_float(0x6d000000u)))) continue;
        for (int d = 1; d <= dmax; d++) {
            const float4 st = c_step[d];
            const float q = div_fast(a, st.x, st.y);
            const float ref = __fdiv_rn(a, -st.x);
            if (__float_as_uint(q) != __float_as_uint(ref) && !(q == 0.0f && ref == 0.0f)) {
                n_bad++;
                atomicCAS(first_bad, 0xffffffffu, (unsigned)u);
            }
            n_ok++;
        }
    }
    atomicAdd(checked, n_ok);
    if (n_bad) atomicAdd(bad, n_bad);
}

}  // namespace

cudaError_t sdem_division_selftest(int dmax, int num_sms, unsigned long long* h_checked,
                                   unsigned long long* h_bad, unsigned* h_first_bad) {
    if (dmax < 1 || dmax >= kFastMaxRow) return cudaErrorInvalidValue;
    unsigned long long* d_cnt = nullptr;
    unsigned* d_first = nullptr;
    cudaError_t e = cudaMalloc(&d_cnt, 2 * sizeof(unsigned long long));
    if (e != cudaSuccess) return e;
    e = cudaMalloc(&d_first, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(d_cnt, 0, 2 * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(d_first, 0xff, sizeof(unsigned));
    if (e == cudaSuccess) {
        k_div_check<<<num_sms * 8, 256>>>(dmax, d_cnt, d_cnt + 1, d_first);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    unsigned long long cnt[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpy(cnt, d_cnt, sizeof(cnt), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(h_first_bad, d_first, sizeof(unsigned), cudaMemcpyDeviceToHost);
    *h_checked = cnt[0];
    *h_bad = cnt[1];
    cudaFree(d_cnt);
    cudaFree(d_first);
    return e;
}

int sdem_chunk() { return kChunk; }

namespace {
struct StepTable {
    float4 v[kFastMaxRow];
    StepTable() {
        for (int d = 0; d < kFastMaxRow; d++) {
            const float df = (float)d;
            v[d] = make_float4(-df, d ? 1.0f / df : 0.0f, 2.0f * df + 1.0f, df + 1.0f);
        }
    }
};
}  // namespace

cudaError_t sdem_init_tables() {
    static const StepTable tab;  // built once, thread-safe, no heap
    cudaError_t e = cudaMemcpyToSymbol(c_step, tab.v, sizeof(tab.v));
    if (e == cudaSuccess) e = sweep_init_tables();
    return e;
}

void sdem_items(const Geometry& geo, const Batch& b, std::vector<uint64_t>& items, int* max_row) {
    // Counting sort of rows by valid length, longest first: a row's work grows
    // about as L^2, so long rows go first.
    int lmax = 0;
    for (int s = 0; s < b.count; s++) {
        const SectorDesc& d = geo.desc[b.angle[s]];
        for (int r = 0; r < d.H; r++) lmax = std::max(lmax, geo.last[d.row_off + r] - geo.first[d.row_off + r]);
    }
    std::vector<int64_t> start(lmax + 2, 0);
    for (int s = 0; s < b.count; s++) {
        const SectorDesc& d = geo.desc[b.angle[s]];
        for (int r = 0; r < d.H; r++) {
            const int L = geo.last[d.row_off + r] - geo.first[d.row_off + r];
            if (L > 0) start[L]++;
        }
    }
    int64_t total = 0;
    for (int L = lmax; L >= 1; L--) {
        const int64_t cnt = start[L];
        start[L] = total;
        total += cnt;
    }
    items.assign(total, 0);
    for (int s = 0; s < b.count; s++) {
        const SectorDesc& d = geo.desc[b.angle[s]];
        for (int r = 0; r < d.H; r++) {
            const int L = geo.last[d.row_off + r] - geo.first[d.row_off + r];
            if (L > 0) items[start[L]++] = ((uint64_t)s << 48) | ((uint64_t)(uint32_t)r << 16);
        }
    }
    *max_row = lmax;
}

cudaError_t launch_sdem_chunked(const SdemLaunch& a, int num_sms, cudaStream_t st) {
    if (a.n_items == 0) return cudaSuccess;
    const size_t smem = sizeof(float) * (size_t)warp_floats(a.max_row) * kWarps;
    cudaError_t e = allow_smem(k_sdem_chunked, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sdem_chunked, kWarps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    int64_t blocks = (int64_t)per_sm * num_sms;
    const int64_t need = (a.n_items + kWarps - 1) / kWarps;
    if (blocks > need) blocks = need;
    e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    k_sdem_chunked<<<(int)blocks, kWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace ske

