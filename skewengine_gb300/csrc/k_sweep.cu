// Total-viewshed line-of-sight sweep of the engine (kernelSDEM,
// src/kernelSDEM.h:168-222).
//
// For every valid cell j of a skewed row (the observer) the reference scans the
// row forward (k = j+1 ..) and backward (k = j-1 ..), tracking the horizon slope
// max((S[k] - h)/d) with h = S[j] + POVh; each step is visible when its slope
// beats the horizon, and every visible run that closes before the row end adds
// d_close^2 - d_open^2 to cv.  The output is cv * (float)scale^2.
//
//  * Persistent kernel; a warp takes one skewed row from a global queue ordered
//    longest row first, stages it in shared memory and scans it in both
//    directions.
//  * Work proceeds in levels of up to 64 steps.  Level 0 takes every observer of
//    the row; after each level an exact horizon test (retire) drops the
//    observers that can see nothing further, and the survivors are appended to
//    a per-warp list (one per direction) in global scratch.  The next level
//    processes only those lists, 32 observers (one per lane) at a time.  An
//    observer's work therefore ends within a level of the test that retires it,
//    instead of with the slowest of a fixed group: on 2000x2000 fractal terrain
//    this runs about a fifth of the line-of-sight steps.
//  * All observers of a batch are at the same step distance d, so -d and
//    RN(1/d) come from the constant table, packed for two steps at a time: the
//    two quotients of a lane's observer take one packed f32x2 chain whose
//    constants are used as they are loaded.
//  * Two steps of an observer cost 14 instructions: two loads, the packed
//    subtraction, the three packed operations of the division, two horizon
//    differences and two maxima, two funnel shifts that collect the sign of
//    (horizon - slope), the visible flag, into a mask of 32 steps, and two
//    loads of constants.  The ring sums follow from the mask once per 32 steps
//    (close_run).  With a comparison and three selections per step in place of
//    the mask it was 11 instructions a step.  The sweep is bound by issue (88%
//    of the slots, FMA and ALU pipes about half busy): on 1000x1000 terrain all
//    angles took 13.6 ms in that form and take 13.0 now in levels of 64, 12.1
//    with a first level of 32.
//  * Lists of more than 128 observers go two to a lane, which halves the
//    constant loads, their moves and the loop's own instructions (1000x1000:
//    12.4 ms with one, 12.1 with two); the remainder and shorter lists go one
//    to a lane, where a half empty second place would cost more (rows of 64:
//    39 us against 43).  The two-observer body is unrolled by 8 steps, the
//    other by 16: with 16 in both the four bodies crowd the instruction cache
//    (500x500: 2.93 ms against 2.77).
//  * Division: the quotient (S[k]-h)/d must be the correctly rounded one, since
//    visibility compares it strictly against the running maximum (div2,
//    sdem_math.cuh; rows whose values leave its range take scan_reference).
//  * Accumulation: a closed visible run [o, c) contributes c^2 - o^2, the sum of
//    the ring areas 2d+1 over its steps.  acc is the ring sum of all visible
//    steps, cl the part of it in runs that have closed: -1 before any (the
//    initial run starts at distance 0, ring 1 not swept), acc less the visible
//    steps since the last invisible one afterwards.  An observer that reaches
//    its row end has cv = 1 + cl (a run still open there is not counted, as in
//    the reference), a retired one 1 + acc (its run closes at the next step).
//    All are integers below 2^24, so the float result is the reference's.
#include <algorithm>

#include "sdem_math.cuh"

namespace ske {

namespace {

constexpr int kLevel = 64;   // line-of-sight steps of a level past the first two
constexpr int kSeg = 32;     // steps of a visibility mask
constexpr int kUnroll = 16;  // steps of a mask's blocks; levels are multiples of it
constexpr int kPairList = 128;  // lists longer than this go two observers to a lane
constexpr int kLWarps = 4;   // warps per CTA
// Per-warp scratch, in units of max_row int4 entries: four survivor lists and
// the two directions' counts (2*max_row floats, within one more unit).
constexpr int kListsPerWarp = 5;
constexpr int kLPad = 64;    // NaN cells on both sides of the row (>= kLevel - 1)
// Longest row on the fast path: every step distance a level touches (at most
// the last survivor's n + kLevel) stays inside the constant table.
constexpr int kLFastMaxRow = kFastMaxRow - kLevel;

// Steps 2i+1 and 2i+2: {-(2i+1), -(2i+2), RN(1/(2i+1)), RN(1/(2i+2))}.
__constant__ ulonglong2 c_pair[kFastMaxRow / 2];

// Retirement bound terms: kT blocks of kB1 cells, then kT blocks of kB2 cells,
// then the suffix (prefix) maximum of everything beyond.
constexpr int kB1 = 16, kB1Log = 4;
constexpr int kB2 = 128, kB2Log = 7;
constexpr int kT = 4;
constexpr int kMPad = 8;  // -inf entries on both sides of the kB1 and kB2 maxima
// 1 - 2^-20: the factor that keeps fl(fl(mx * kShrink) * ds) below mx * ds.
constexpr float kShrink = 0.99999904632568359375f;
// 1 + 2^-20: keeps fl(fl(mx * kGrow) * n) below mx * n for mx < 0.
constexpr float kGrow = 1.00000095367431640625f;

__host__ __device__ inline int lrow_pad(int max_row) { return kLPad + ((max_row + 3) & ~3) + kLPad; }
__host__ __device__ inline int nblk(int max_row, int size) { return (max_row + size - 1) / size; }

// Per-warp shared memory of the compacting sweep, in floats from the warp's base:
// the padded row; suffix maxima of kB2-cell blocks (one -inf entry after);
// prefix maxima of kB2-cell blocks (one -inf entry before); kB1-cell and
// kB2-cell block maxima (kMPad -inf entries on both sides).  About 1.17 floats
// per cell of the longest row: 2335 per warp at 2000 cells, so six 4-warp CTAs
// share an SM's 228 KB.
struct LLayout {
    int s128, p128, b16, b128, total;
    __host__ __device__ explicit LLayout(int max_row) {
        const int n16 = nblk(max_row, kB1), n128 = nblk(max_row, kB2);
        s128 = lrow_pad(max_row);
        p128 = s128 + n128 + 2;
        b16 = p128 + n128 + kMPad;
        b128 = b16 + n16 + 2 * kMPad;
        total = b128 + n128 + kMPad;
    }
};

// The block maxima of the row being swept.
struct RowMax {
    const float *s128, *p128, *b16, *b128;
    int n128;
};

// One lane's observer of a batch.
struct Observer {
    int x;         // position in the row
    int n;         // steps in the batch's direction
    float h, mx;   // observer height, horizon slope
    int acc, cl;   // ring sums: visible steps, closed runs
};

// Steps ds .. ds + kUnroll*blocks - 1 (ds odd, at most kSeg steps) of the lane's
// kObs observers: the masks of the visible ones, the first step in the highest of
// the kUnroll*blocks bits.  A step past an observer's last target reads the row's
// NaN padding: its slope is NaN, the horizon keeps its value and the bit is
// dropped by close_run.
template <bool kF, int kObs>
__device__ __forceinline__ void scan_segment(const float* const (&p0)[kObs], int ds, int blocks, const float (&h)[kObs],
                                             float (&mx)[kObs], unsigned (&seen)[kObs]) {
    f2 hh[kObs];
    const float* p[kObs];
#pragma unroll
    for (int o = 0; o < kObs; o++) {
        hh[o] = pk(h[o], h[o]);
        seen[o] = 0;
        p[o] = p0[o];
    }
    int i = ds >> 1;
    constexpr int kBody = kObs == 2 ? 8 : kUnroll;
#pragma unroll 1
    for (int b = blocks * (kUnroll / kBody); b > 0; b--) {
#pragma unroll
        for (int e = 0; e < kBody; e += 2) {
            const ulonglong2 st = c_pair[i + e / 2];
#pragma unroll
            for (int o = 0; o < kObs; o++) {
                const float z0 = kF ? p[o][e] : p[o][-e];
                const float z1 = kF ? p[o][e + 1] : p[o][-e - 1];
                float q0, q1;
                upk(div2(sub2(pk(z0, z1), hh[o]), st.x, st.y), q0, q1);
                // Negative differences: the slope beats the horizon.
                const float t0 = __fsub_rn(mx[o], q0), m1 = fmaxf(mx[o], q0);
                const float t1 = __fsub_rn(m1, q1);
                mx[o] = fmaxf(m1, q1);
                seen[o] = __funnelshift_l(__float_as_uint(t0), seen[o], 1);
                seen[o] = __funnelshift_l(__float_as_uint(t1), seen[o], 1);
            }
        }
#pragma unroll
        for (int o = 0; o < kObs; o++) p[o] += kF ? kBody : -kBody;
        i += kBody / 2;
    }
}

// Adds the visible steps of a segment of `steps` steps from ds to the sums.
__device__ __forceinline__ void close_run(Observer& s, unsigned seen, int ds, int steps) {
    const int v = min(s.n - ds + 1, steps);  // steps the observer has in the segment
    unsigned m;                              // its own steps, the last in bit 0 (v <= 0: none)
    asm("shr.b32 %0, %1, %2;" : "=r"(m) : "r"(seen), "r"(steps - v));
    const int end = ds + v;  // distance after its last step; bit k is distance end - 1 - k
    // Sum of 2d + 1 over the set bits: the bits' count and positions.
    const int cnt = __popc(m);
    const int pos = __popc(m & 0xaaaaaaaau) + 2 * __popc(m & 0xccccccccu) + 4 * __popc(m & 0xf0f0f0f0u) +
                    8 * __popc(m & 0xff00ff00u) + 16 * __popc(m & 0xffff0000u);
    s.acc += cnt * (2 * end - 1) - 2 * pos;
    // Visible steps since the last invisible one; none invisible: the run goes on.
    const int open = __popc(m & ~(m + 1u));
    if (open < v) s.cl = s.acc - open * (2 * end - open);
}

// Where a row's results go.
struct RowOut {
    float* out;           // the sector's output grid
    int64_t rowbase;      // flat index of the row's first valid cell
    int first;            // its column
    int row;
    const SectorDesc* sd;
    const int32_t* rfirst;
    const int32_t* rlast;
    int counts_only;
    bool compact;         // batched run: the row's cells are its own compact row
};

// Cells that lie in the row's own span of the flat grid (column < dim_i) are
// always the row's; cells past it may belong to a later row (owner_row).  A
// compact row (batched runs) owns all its cells.
__device__ __forceinline__ bool owns(const RowOut& o, int x) {
    return o.compact || o.first + x < o.sd->dim_i || owner_row(*o.sd, o.rfirst, o.rlast, o.rowbase + x) == o.row;
}

// The maxima arrays of a fast-path row (finite, at most 32 * kB2 cells, so one
// kB2 block per lane): kB1- and kB2-cell block maxima with their -inf padding,
// s128[b] = max A[kB2*b ..] to the row end (s128[n128] = -inf) and
// p128[b] = max A[.. kB2*b + kB2-1] from the row start (p128[-1] = -inf).
__device__ void row_maxima(const float* __restrict__ A, int L, float* s128, float* p128, float* b16, float* b128,
                           int lane) {
    const float ninf = __int_as_float(0xff800000);
    const int n16 = nblk(L, kB1), n128 = nblk(L, kB2);
    // kB1 = 16 cells: half a warp per block, a row segment of 32 cells per pass.
    for (int c0 = 0; c0 < n16 * kB1; c0 += 32) {
        float m = c0 + lane < L ? A[c0 + lane] : ninf;
#pragma unroll
        for (int off = kB1 / 2; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
        const int b = (c0 + lane) >> kB1Log;
        if ((lane & (kB1 - 1)) == 0 && b < n16) b16[b] = m;
    }
    if (lane < kMPad) {
        b16[-1 - lane] = ninf;
        b16[n16 + lane] = ninf;
        b128[-1 - lane] = ninf;
        b128[n128 + lane] = ninf;
    }
    __syncwarp();
    constexpr int kPer = kB2 / kB1;
    float m = ninf;  // this lane's kB2 block
    if (lane < n128) {
        for (int c = lane * kPer; c < min(lane * kPer + kPer, n16); c++) m = fmaxf(m, b16[c]);
        b128[lane] = m;
    }
    // Inclusive prefix and suffix maxima over the lanes (Hillis-Steele).
    float inc_p = m, inc_s = m;
    for (int off = 1; off < 32; off <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, inc_p, off);
        const float dn = __shfl_down_sync(0xffffffffu, inc_s, off);
        if (lane >= off) inc_p = fmaxf(inc_p, up);
        if (lane + off < 32) inc_s = fmaxf(inc_s, dn);
    }
    if (lane < n128) {
        s128[lane] = inc_s;
        p128[lane] = inc_p;
    }
    if (lane == 0) {
        s128[n128] = ninf;
        p128[-1] = ninf;
    }
}

// Retirement test after step dc: true when no target beyond distance dc can be
// visible from observer x (n steps in this direction, height h, horizon mx).
// The remaining targets are covered by kT blocks of kB1 cells from the one
// holding the nearest target, kT blocks of kB2 cells from the next uncovered
// cell, and the suffix (prefix) maximum beyond; blocks past the row end read
// -inf.  The first block may also hold up to kB1-1 passed targets, which only
// raises the bound.
//  * mx >= 0: a block of remaining targets with maximum M and nearest
//    remaining distance ds holds no visible target when
//    M - h <= fl(fl(mx * kShrink) * ds): that product is below mx * ds, so
//    every target u = fl(z - h) <= M - h at distance d' >= ds has
//    u / d' <= mx (u >= 0) or u / d' < 0 <= mx (u < 0), and fl(u / d') <= mx.
//  * mx < 0: the same with the farthest distance n and the factor kGrow: M - h <=
//    fl(fl(mx * kGrow) * n) < mx * n < 0, so u / d' <= u / n < mx.
template <bool kFwd>
__device__ __forceinline__ bool retire(const RowMax& rm, int x, int n, int dc, float h, float mx) {
    const int k = kFwd ? x + dc + 1 : x - dc - 1;  // nearest remaining target
    const int b = k >> kB1Log;
    float m1[kT], m2[kT];
#pragma unroll
    for (int j = 0; j < kT; j++) m1[j] = rm.b16[kFwd ? b + j : b - j];
    const int c = kFwd ? (b + kT) * kB1 : (b - kT + 1) * kB1 - 1;  // first uncovered cell
    const int b2 = c >> kB2Log;                                     // arithmetic shift: floor
#pragma unroll
    for (int j = 0; j < kT; j++) m2[j] = rm.b128[kFwd ? b2 + j : b2 - j];
    const float tail = kFwd ? rm.s128[min(b2 + kT, rm.n128)] : rm.p128[max(b2 - kT, -1)];
    // Distances ds of the blocks: n for all of them where mx < 0.
    const bool neg = mx < 0.0f;
    const float nf = __int2float_rn(n), mxc = __fmul_rn(mx, neg ? kGrow : kShrink);
    const float in1 = neg ? 0.0f : (float)kB1, in2 = neg ? 0.0f : (float)kB2;
    bool ok = __fsub_rn(m1[0], h) <= __fmul_rn(mxc, neg ? nf : __int2float_rn(dc + 1));
    float ds = neg ? nf : __int2float_rn(kFwd ? (b + 1) * kB1 - x : x - (b * kB1 - 1));
#pragma unroll
    for (int j = 1; j < kT; j++) {
        ok &= __fsub_rn(m1[j], h) <= __fmul_rn(mxc, ds);
        ds = __fadd_rn(ds, in1);
    }
    ok &= __fsub_rn(m2[0], h) <= __fmul_rn(mxc, ds);  // the next uncovered cell follows the kB1 blocks
    ds = neg ? nf : __int2float_rn(kFwd ? (b2 + 1) * kB2 - x : x - (b2 * kB2 - 1));
#pragma unroll
    for (int j = 1; j < kT; j++) {
        ok &= __fsub_rn(m2[j], h) <= __fmul_rn(mxc, ds);
        ds = __fadd_rn(ds, in2);
    }
    ok &= __fsub_rn(tail, h) <= __fmul_rn(mxc, ds);
    return ok;
}

// The survivor lists and results of one row's sweep (per-warp global scratch).
struct RowLists {
    const int4* in[2];  // this level's survivors, forward / backward (null: level 0)
    int4* out[2];       // the next level's, forward / backward
    int n[2];           // entries of in[]
    int made[2];        // entries appended to out[]
    float* cv[2];       // finished observers' counts by position, forward / backward
};

// One batch of a level: kObs * 32 entries from i0, kObs to a lane.
template <bool kF, int kObs>
__device__ __forceinline__ void sweep_batch(const float* __restrict__ A, const RowMax& rm, int L, float povh,
                                            RowLists& rl, int d0, int len, int lane, const int4* in, int n_in, int i0,
                                            int& made) {
    constexpr int dir = kF ? 0 : 1;
    const unsigned below = (1u << lane) - 1u;
    Observer s[kObs];
    bool valid[kObs];
    int own = 0;
#pragma unroll
    for (int o = 0; o < kObs; o++) {
        const int idx = i0 + 32 * o + lane;
        valid[o] = idx < n_in;
        if (valid[o]) {
            if (in) {
                const int4 e = in[idx];
                s[o].x = e.x;
                s[o].mx = __int_as_float(e.y);
                s[o].acc = e.z;
                s[o].cl = e.w;
            } else {
                s[o].x = idx;
                s[o].mx = -2000.0f;
                s[o].acc = 0;
                s[o].cl = -1;
            }
            s[o].n = kF ? L - 1 - s[o].x : s[o].x;
            s[o].h = __fadd_rn(A[s[o].x], povh);
        } else {
            // Empty: its reads stay in A[-(kLevel-1) .. kLevel-1].
            s[o].x = kF ? -d0 : d0;
            s[o].n = 0;
            s[o].h = s[o].mx = 0.0f;
            s[o].acc = s[o].cl = 0;
        }
        own = max(own, s[o].n);
    }
    const int most = __reduce_max_sync(0xffffffffu, own);
    const int steps = min(len, (most - d0 + kUnroll) & ~(kUnroll - 1));
    const float* p[kObs];
    float h[kObs], mx[kObs];
#pragma unroll
    for (int o = 0; o < kObs; o++) {
        p[o] = A + (kF ? s[o].x + d0 : s[o].x - d0);
        h[o] = s[o].h;
        mx[o] = s[o].mx;
    }
    int ds = d0;
    for (int left = steps; left > 0; left -= kSeg) {
        const int seg = min(left, kSeg);
        unsigned seen[kObs];
        scan_segment<kF, kObs>(p, ds, seg / kUnroll, h, mx, seen);
#pragma unroll
        for (int o = 0; o < kObs; o++) {
            close_run(s[o], seen[o], ds, seg);
            p[o] += kF ? kSeg : -kSeg;
        }
        ds += kSeg;
    }
    // Retire finished observers, keep the others for the next level.
    const int dc = d0 + steps - 1;  // last step taken
#pragma unroll
    for (int o = 0; o < kObs; o++) {
        bool keep = false;
        if (valid[o]) {
            bool done = false;
            if (s[o].n > dc) {
                done = retire<kF>(rm, s[o].x, s[o].n, dc, h[o], mx[o]);
                keep = !done;
            }
            if (!keep) rl.cv[dir][s[o].x] = __int2float_rn(1 + (done ? s[o].acc : s[o].cl));
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep)
            rl.out[dir][made + __popc(m & below)] = make_int4(s[o].x, __float_as_int(mx[o]), s[o].acc, s[o].cl);
        made += __popc(m);
    }
}

// One level of one direction: the list's observers, len steps from d0 (fewer
// where no observer of a batch has as many left).
template <bool kF>
__device__ __forceinline__ void sweep_level(const float* __restrict__ A, const RowMax& rm, int L, float povh,
                                            RowLists& rl, int d0, int len, int lane) {
    constexpr int dir = kF ? 0 : 1;
    const int4* in = rl.in[dir];
    const int n_in = rl.n[dir];
    int made = 0, i0 = 0;
    if (n_in > kPairList) {
        for (; n_in - i0 > 32; i0 += 64)
            sweep_batch<kF, 2>(A, rm, L, povh, rl, d0, len, lane, in, n_in, i0, made);
    }
    for (; n_in > i0; i0 += 32) sweep_batch<kF, 1>(A, rm, L, povh, rl, d0, len, lane, in, n_in, i0, made);
    rl.made[dir] = made;
}

// Both scan directions of the row, level by level: lvl0 steps, then lvl1 (when
// non-zero), then kLevel each.
// lists: four lists of L_max entries (forward in/out, backward in/out);
// cvf, cvb: the two directions' counts, added and scaled at the end.
__device__ __forceinline__ void sweep_row(const float* __restrict__ A, const RowMax& rm, int L, float povh,
                                          int4* lists, int max_row, float* cvf, float* cvb, const RowOut& o, int lane,
                                          int lvl0, int lvl1) {
    RowLists rl;
    rl.in[0] = rl.in[1] = nullptr;
    rl.out[0] = lists;
    rl.out[1] = lists + 2 * (int64_t)max_row;
    rl.n[0] = rl.n[1] = L;
    rl.cv[0] = cvf;
    rl.cv[1] = cvb;
    int len = lvl0, next = lvl1 > 0 ? lvl1 : kLevel;
    for (int d0 = 1; rl.n[0] > 0 || rl.n[1] > 0;) {
        sweep_level<true>(A, rm, L, povh, rl, d0, len, lane);
        sweep_level<false>(A, rm, L, povh, rl, d0, len, lane);
        __syncwarp();  // this level's lists and counts are visible to every lane
#pragma unroll
        for (int dir = 0; dir < 2; dir++) {
            int4* base = lists + 2 * (int64_t)max_row * dir;
            rl.in[dir] = rl.out[dir];
            rl.out[dir] = rl.out[dir] == base ? base + max_row : base;
            rl.n[dir] = rl.made[dir];
        }
        d0 += len;
        len = next;
        next = kLevel;
    }
    for (int x = lane; x < L; x += 32) {
        if (!owns(o, x)) continue;
        const float t = __fadd_rn(cvf[x], cvb[x]);  // forward count, then backward
        o.out[o.rowbase + x] = o.counts_only ? t : __fmul_rn(t, o.sd->r2);
    }
}

// kBatch: the items are batch_item()s of a batched run over several grids,
// whose rows are compact rows of the pools SI/SO (kernels.h, BatchGrid).
template <bool kBatch>
__global__ void __launch_bounds__(kLWarps * 32) k_sweep(SdemLaunch a) {
    extern __shared__ float4 smem4[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const LLayout lay(a.max_row);
    float* buf = reinterpret_cast<float*>(smem4) + (size_t)warp * lay.total;
    float* A = buf + kLPad;
    float* s128 = buf + lay.s128;
    float* p128 = buf + lay.p128;
    float* b16 = buf + lay.b16;
    float* b128 = buf + lay.b128;
    const int64_t gwarp = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    int4* lists = a.lists + gwarp * kListsPerWarp * (int64_t)a.max_row;
    float* cvf = reinterpret_cast<float*>(lists + 4 * (int64_t)a.max_row);
    float* cvb = cvf + a.max_row;
    for (;;) {
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(a.counter, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if ((int64_t)idx >= a.n_items) break;
        const SectorDesc* dp;
        const int32_t *first = nullptr, *last = nullptr;
        int row, f, L;
        int64_t slot_off = 0;  // the sector's slot in SI/SO (per-engine runs)
        RowOut o;
        if (kBatch) {
            const uint64_t raw = a.items[idx];
            const BatchSector bs = a.bt.sectors[(int)(raw >> 32)];
            const BatchGrid& G = a.bt.grids[bs.grid];
            row = (int)(raw & 0xffffffffu);
            dp = &G.desc[bs.angle];
            const int4 m = G.rowtab[dp->row_off + row];  // {first, last, rowoff}
            f = m.x;
            L = m.y - m.x;
            o.out = a.SO;
            o.rowbase = bs.cells + m.z;
        } else {
            const Item it = decode(a.items[idx]);
            row = it.row;
            dp = &a.g.desc[a.b.angle[it.slot]];
            first = a.g.first + dp->row_off;
            last = a.g.last + dp->row_off;
            f = first[row];
            L = last[row] - f;
            slot_off = it.slot * a.stride;
            o.out = a.SO + slot_off;
            o.rowbase = (int64_t)row * dp->dim_i + f;
        }
        const SectorDesc& d = *dp;
        if (L > a.max_row || L <= 0) {
            if (lane == 0) atomicExch(a.status, 1);
            continue;
        }
        o.first = f;
        o.row = row;
        o.sd = &d;
        o.rfirst = first;
        o.rlast = last;
        o.counts_only = a.counts_only;
        o.compact = kBatch;
        const float* src = a.SI + slot_off + o.rowbase;
        bool ok = true;
        for (int x = lane; x < L; x += 32) {
            const float v = src[x];
            A[x] = v;
            ok = ok && div_safe(v) && div_safe(__fadd_rn(v, a.povh));
        }
        const float pad = __int_as_float(0x7fc00000);  // NaN (see scan_segment)
        for (int x = lane; x < kLPad; x += 32) buf[x] = pad;
        const int tail_end = ((L + 3) & ~3) + kLPad;
        for (int x = L + lane; x < tail_end; x += 32) A[x] = pad;
        const bool fast = __all_sync(0xffffffffu, ok) && L <= kLFastMaxRow && div_safe(a.povh);
        __syncwarp();
        if (fast) {
            row_maxima(A, L, s128, p128, b16, b128, lane);
            __syncwarp();
            const RowMax rm{s128, p128, b16, b128, nblk(L, kB2)};
            sweep_row(A, rm, L, a.povh, lists, a.max_row, cvf, cvb, o, lane, a.lvl0, a.lvl1);
        } else {
            for (int x = lane; x < L; x += 32) {
                if (!owns(o, x)) continue;
                const float cv = scan_reference(A, x, L, a.povh);
                o.out[o.rowbase + x] = a.counts_only ? cv : __fmul_rn(cv, d.r2);
            }
        }
        __syncwarp();
    }
}

}  // namespace

cudaError_t sweep_init_tables() {
    static float4 pair[kFastMaxRow / 2];
    for (int i = 0; i < kFastMaxRow / 2; i++) {
        const float a = (float)(2 * i + 1), b = (float)(2 * i + 2);
        pair[i] = make_float4(-a, -b, 1.0f / a, 1.0f / b);
    }
    return cudaMemcpyToSymbol(c_pair, pair, sizeof(pair));
}

size_t sdem_list_bytes(int max_row, int num_sms) {
    // kListsPerWarp units of max_row entries per warp, for as many warps as an SM holds.
    int dev = 0, threads = 2048;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&threads, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
    return (size_t)num_sms * (size_t)(threads / 32) * kListsPerWarp * (size_t)std::max(max_row, 1) * sizeof(int4);
}

int sdem_max_ctas_per_sm(const SdemLaunch& a) {
    const size_t smem = sizeof(float) * (size_t)LLayout(std::max(a.max_row, 1)).total * kLWarps;
    auto kern = a.batched ? k_sweep<true> : k_sweep<false>;
    if (allow_smem(kern, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kLWarps * 32, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return per_sm;
}

cudaError_t launch_sdem(const SdemLaunch& a, int num_sms, cudaStream_t st) {
    if (a.n_items == 0) return cudaSuccess;
    auto level_ok = [](int v) { return v == 16 || v == 32 || v == 48 || v == 64; };
    if (!level_ok(a.lvl0) || (a.lvl1 != 0 && !level_ok(a.lvl1)) || a.ctas_per_sm < 0) return cudaErrorInvalidValue;
    const size_t smem = sizeof(float) * (size_t)LLayout(a.max_row).total * kLWarps;
    auto kern = a.batched ? k_sweep<true> : k_sweep<false>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kLWarps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    if (a.ctas_per_sm > 0 && per_sm > a.ctas_per_sm) per_sm = a.ctas_per_sm;
    int64_t blocks = (int64_t)per_sm * num_sms;
    const int64_t need = (a.n_items + kLWarps - 1) / kLWarps;
    if (blocks > need) blocks = need;
    // Every warp owns kListsPerWarp units of max_row entries in the scratch.
    const size_t list_per_block = (size_t)kLWarps * kListsPerWarp * (size_t)a.max_row * sizeof(int4);
    const int64_t fit = a.lists ? (int64_t)(a.list_bytes / list_per_block) : 0;
    if (fit < 1) return cudaErrorInvalidValue;
    if (blocks > fit) blocks = fit;
    e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    kern<<<(int)blocks, kLWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace ske
