// Cepstrum blur estimation in float32, fused over the whole sector loop
// (kernelBLUR, src/kernelBLUR.h:267-302 -> lineCepstrum :153-228, with the
// max+angle deskew of skewEngine.cuh:774-785), for batches of square images.
//
// The reference computes each skewed cell's cepstrum in binary64; the engine's
// exact operator (k_cepstrum.cu) does the same and is FP64-pipe bound.  This
// mode computes the same quantities in float32 on the FP32 pipes:
//   X = FFT64(window)/8          64-sample real window as a 32-point complex
//                                FFT in registers (even/odd packing) and the
//                                real-input split;
//   l_k = log(|X_k|^2), k < 32   (CUDA's logf);
//   c_k = sum_n l_n cos(2 pi k n / 32) / sqrt(32), k < 16, folded (l_n and
//                                l_{32-n} share a cosine);
//   s_k = -min(0, c_k), the reference's peak search, output 10000 * peak.
// Rounding differs from the reference's, so an output can land in another
// 1000-wide bin where a value sits at a bin edge: the bin-mismatch rate against
// the exact operator is measured and stated, and the exact operator stays the
// parity mode.
//
// Most cells never run it: only the 1000-wide bin of a value is deskewed, and
// cepstrum_bin (cepstrum_bin.cuh) arrives at it with half the operations wherever
// its bound and this evaluation's leave no doubt; the cells they leave open (a few
// in a hundred) are listed and take this one, a thread each; windows of one value
// (empty borders and backgrounds) are left open by the bound and answered without it
// (an empty 512 x 512 image: 7.3 -> 3.7 ms, a phantom 7.0 -> 5.2).  The same bits:
// 90.1 ms for 16 images of 512 x 512 with every cell here, 46.5 so, 40.3 with
// 256-row tiles (1.13 cepstra per skewed cell, 128-row tiles form 1.27), 34.7
// with two cells to a thread (16 warps of 128 registers; 12 of 168 take 35.9, 8
// of 188 41.7).
//
// Fusion: a CTA owns a 256 x 32 tile of one orientation's accumulator of one
// image and walks that orientation's sectors in angle order.  Per sector it
// gathers the skewed rows the tile needs (the reference's skew, gathered from
// the orientation: skew_gather) as 96-cell row segments into shared memory,
// computes the cepstrum of every band cell (a thread per two rows' cells, the
// 64-cell windows read from the staged segments), and max-deskews into the tile's
// accumulator in shared memory.  The skewed input and output never reach HBM; the orientations
// (4 x N floats per image) stay L2-resident.
#include <algorithm>
#include <atomic>

#include <cooperative_groups.h>

#include "cepstrum_bin.cuh"

namespace ske {

namespace {

constexpr int kCTall = 256, kCLow = 64;  // accumulator tile rows, by launch_cepstrum_f32
constexpr int kCSeg = 96;              // staged cells per band row: columns j0-32 .. j0+63
constexpr int kCThreads = 512;
constexpr int kCWarps = kCThreads / 32;

// W64^k = exp(-2 pi i k / 64) as float (cos, -sin), filled on the host.
__constant__ float2 c_w64[64];

__device__ __forceinline__ void cmulf(float ar, float ai, float br, float bi, float& r, float& i) {
    r = __fsub_rn(__fmul_rn(ar, br), __fmul_rn(ai, bi));
    i = __fadd_rn(__fmul_rn(ar, bi), __fmul_rn(ai, br));
}

// 32-point complex FFT in registers, radix-2 decimation in time: input in
// bit-reversed order, output in natural order.
__device__ __forceinline__ void fft32(float (&re)[32], float (&im)[32]) {
#pragma unroll
    for (int span = 1; span < 32; span <<= 1) {
#pragma unroll
        for (int start = 0; start < 32; start += 2 * span) {
#pragma unroll
            for (int k = 0; k < span; k++) {
                const int a = start + k, b = a + span;
                const float2 w = c_w64[k * (32 / span)];  // W_{2 span}^k = W64^(k * 64 / (2 span))
                float tr, ti;
                if (k == 0) {
                    tr = re[b];
                    ti = im[b];
                } else {
                    cmulf(re[b], im[b], w.x, w.y, tr, ti);
                }
                re[b] = __fsub_rn(re[a], tr);
                im[b] = __fsub_rn(im[a], ti);
                re[a] = __fadd_rn(re[a], tr);
                im[a] = __fadd_rn(im[a], ti);
            }
        }
    }
}

// Cepstrum peak of the 64-sample window w[0..63] (zeros outside the row), as
// lineCepstrum computes it, in float32.  w: its samples, two floats apart.
__device__ __forceinline__ float cepstrum_f32(const float* __restrict__ w) {
    float re[32], im[32];
#pragma unroll
    for (int n = 0; n < 32; n++) {  // z_n = w[2n] + i w[2n+1], stored bit-reversed
        re[brev5(n)] = w[4 * n];
        im[brev5(n)] = w[4 * n + 2];
    }
    fft32(re, im);
    // X_k = E_k + W64^k O_k, E = (Z_k + conj Z_{32-k}) / 2, O = -i (Z_k - conj Z_{32-k}) / 2;
    // l_k = log(|X_k / 8|^2).
    float l[32];
#pragma unroll
    for (int k = 0; k < 32; k++) {
        const int m = (32 - k) & 31;
        const float er = __fmul_rn(0.5f, __fadd_rn(re[k], re[m]));
        const float ei = __fmul_rn(0.5f, __fsub_rn(im[k], im[m]));
        const float orr = __fmul_rn(0.5f, __fadd_rn(im[k], im[m]));
        const float oi = __fmul_rn(-0.5f, __fsub_rn(re[k], re[m]));
        float xr, xi;
        if (k == 0) {
            xr = __fadd_rn(er, orr);
            xi = __fadd_rn(ei, oi);
        } else {
            const float2 t = c_w64[k];
            float pr, pi;
            cmulf(orr, oi, t.x, t.y, pr, pi);
            xr = __fadd_rn(er, pr);
            xi = __fadd_rn(ei, pi);
        }
        xr = __fmul_rn(xr, 0.125f);
        xi = __fmul_rn(xi, 0.125f);
        l[k] = logf(__fadd_rn(__fmul_rn(xr, xr), __fmul_rn(xi, xi)));
    }
    // c_k = (l_0 + (-1)^k l_16 + sum_{n=1}^{15} (l_n + l_{32-n}) cos(2 pi k n / 32)) / sqrt(32)
    float e[16];
#pragma unroll
    for (int n = 1; n < 16; n++) e[n] = __fadd_rn(l[n], l[32 - n]);
    const float inv = 0.17677669529663687f;  // 1 / sqrt(32)
    float s[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
        float acc = (k & 1) ? __fsub_rn(l[0], l[16]) : __fadd_rn(l[0], l[16]);
#pragma unroll
        for (int n = 1; n < 16; n++) acc = __fmaf_rn(e[n], c_w64[(2 * k * n) & 63].x, acc);
        const float c = __fmul_rn(acc, inv);
        s[k] = c < 0.0f ? -c : -0.0f;  // -std::min(0, c)
    }
    // getBlurParameter2 (kernelBLUR.h:88-110): from index 5 skip the
    // non-ascending head; the peak is the sample before the first ascent or any
    // larger sample after the ascending one.
    float best = 0.0f;
    int asc = 16;
#pragma unroll
    for (int i = 15; i >= 5; i--)
        if (s[i] > s[i - 1]) asc = i;
    if (asc < 16) {
#pragma unroll
        for (int i = 4; i < 16; i++) {
            if (i == asc - 1) best = s[i];
        }
#pragma unroll
        for (int i = 6; i < 16; i++)
            if (i > asc && s[i] > best) best = s[i];
    }
    return __fmul_rn(best, 10000.0f);
}

// Whether all 64 samples of the window are one moderate value (as cepstrum_f32's
// w).  Every X_k but X_0 is then exactly zero, its logarithm -inf, every c_k past
// the first a sum of both infinities, and no sample ascends: the value is 0.
__device__ __forceinline__ bool constant_window(const float* __restrict__ w) {
    const float a = w[0];
    if (a != w[64] || a != w[126] || !(fabsf(a) < 1e15f)) return false;
    bool same = true;
#pragma unroll
    for (int n = 1; n < 63; n++) same = same && w[2 * n] == a;
    return same;
}

template <int kCRows>
struct CSmem {
    static constexpr int kCBand = kCRows + 34;  // skewed rows of a tile per sector (drift <= 32 over 32 columns)
    f2 seg[kCBand / 2][kCSeg];  // two band rows in the halves
    int val[kCBand][32];   // bins
    int acc[kCRows][32];   // the tile's accumulator: see k_cepstrum_fused
    unsigned short open_cells[kCBand * 32];  // band cells cepstrum_bin left open
    int n_open;
    int n_formed;  // of those, formed by cepstrum_f32
    int direct, wait;  // sectors to go without cepstrum_bin; how many the next time
};

// A tile three quarters of whose cells cepstrum_bin left for cepstrum_f32 (a flat
// image's, one far from 1) goes without it for a sector, then for two, four and up
// to kMostDirect, until it decides again: a flat 512 x 512 image 7.09 -> 5.85 ms (6.64
// with every cell in cepstrum_f32), one of 1e-30 7.23 -> 5.50 (5.25), a flat 2048 x 2048
// one 99.0 -> 82.9 (79.3).  Waits that grow by four (80.3) cost a 512 x 512 ramp, flat
// along some angles only, 3.97 ms for 3.19.
constexpr int kFirstDirect = 1, kMostDirect = 16;

// The reference's max+angle update o = angle + 1000*(int)(max(o, m)/1000) keeps
// the last sector's angle and the largest bin (int)(m/1000), except that the bin
// of an infinite m saturates and 1000 times it wraps to -1000: the cell becomes
// angle - 1000, as if its largest bin were -1, whatever came before.  So a cell's
// state over any run of sectors is that bin (-1: none, or just emptied) and
// whether it was emptied, and runs of consecutive sectors can be formed apart.
constexpr int kEmptied = 1 << 30;  // in CSmem::acc, beside the largest bin + 1

// One launch: blockIdx.y = image; blockIdx.x = (type, tile row, tile column);
// blockIdx.z, the rank in the cluster: which of the type's runs of sectors.  The
// CTAs of a cluster join their runs through distributed shared memory.
template <int kCRows>
__global__ void __launch_bounds__(kCThreads, 1)
    k_cepstrum_fused(BatchTables T, DevGeometry g, TypeLists tl, int dim, int tiles_x, int tiles_y) {
    extern __shared__ __align__(16) unsigned char smem_c[];
    typedef CSmem<kCRows> Smem;
    Smem& sm = *reinterpret_cast<Smem*>(smem_c);
    f2(*seg)[kCSeg] = sm.seg;
    int(*val)[32] = sm.val;
    const int per_type = tiles_x * tiles_y;
    const int t = blockIdx.x / per_type;
    const int tile = blockIdx.x - t * per_type;
    const int cnt = tl.count[t];
    if (cnt == 0) return;
    const BatchGrid& G = T.grids[blockIdx.y];
    const int64_t n = G.n;
    const int j0 = (tile % tiles_x) * 32, i0 = (tile / tiles_x) * kCRows;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int j = j0 + tx;
    const bool col_ok = j < dim;
    const int jlast = min(j0 + 32, dim) - 1;
    const int i_end = min(i0 + kCRows, dim);
    const int ni = i_end - i0;
    float* A = G.acc + t * n;
    const float* src = G.orient + t * n;
    if (threadIdx.x == 0) {  // (the first sector's staging ends in a barrier)
        sm.n_open = sm.n_formed = sm.direct = 0;
        sm.wait = kFirstDirect;
    }
    // The accumulators are zero before the first sector: bin 0.
    for (int i = ty; i < ni; i += kCWarps) sm.acc[i][tx] = blockIdx.z == 0 ? 1 : 0;
    const int q0 = cnt * (int)blockIdx.z / (int)gridDim.z, q1 = cnt * ((int)blockIdx.z + 1) / (int)gridDim.z;
    for (int q = q0; q < q1; q++) {
        const SectorDesc d = g.desc[tl.angle[t][q]];
        const int32_t* tg = g.target + d.col_off;
        const float* wg = g.weight + d.col_off;
        const int32_t* rfirst = g.first + d.row_off;
        const int32_t* rlast = g.last + d.row_off;
        const int tmin = tg[j0], tmax = tg[jlast];
        const int r0 = i0 + tmin;
        const int nrows = ni + 1 + (tmax - tmin);  // <= Smem::kCBand for square grids
        // Stage the band's row segments (skewed cells gathered from the orientation).
        // A warp per row, three columns per lane whose shifts and weights stay in
        // registers.
        int tc[kCSeg / 32];
        float wc[kCSeg / 32];
#pragma unroll
        for (int k = 0; k < kCSeg / 32; k++) {
            const int x = j0 - 32 + tx + 32 * k, xc = min(max(x, 0), dim - 1);
            tc[k] = tg[xc];
            wc[k] = wg[xc];
        }
#pragma unroll 2
        for (int p = ty; 2 * p < nrows; p += kCWarps) {
            float cell[2][kCSeg / 32];
#pragma unroll
            for (int y = 0; y < 2; y++) {
                const int r = r0 + 2 * p + y;
                const int f = r < d.H ? rfirst[r] : 0, l = r < d.H ? rlast[r] : 0;
#pragma unroll
                for (int k = 0; k < kCSeg / 32; k++) {
                    const int x = j0 - 32 + tx + 32 * k, i = r - tc[k] - 1;
                    const bool in = x >= f && x < l;
                    const bool v0 = in && (unsigned)i < (unsigned)d.dim_o;
                    const bool v1 = in && (unsigned)(i + 1) < (unsigned)d.dim_o;
                    const float* p0 = src + ((int64_t)i * d.dim_i + x);
                    const float a = v0 ? p0[0] : 0.0f, e = v1 ? p0[d.dim_i] : 0.0f;
                    float acc = 0.0f;  // as skew_gather
                    acc = v0 ? __fadd_rn(acc, __fmul_rn(wc[k], a)) : acc;
                    acc = v1 ? __fadd_rn(acc, __fmul_rn(__fsub_rn(1.0f, wc[k]), e)) : acc;
                    cell[y][k] = acc;
                }
            }
#pragma unroll
            for (int k = 0; k < kCSeg / 32; k++) seg[p][tx + 32 * k] = pk(cell[0][k], cell[1][k]);
        }
        __syncthreads();
        // Bin of every valid band cell: warp = two band rows, lane = column.
        const bool direct = sm.direct > 0;
        for (int p = ty; 2 * p < nrows; p += kCWarps) {
            const int r = r0 + 2 * p;
            bool valid[2], full[2];
#pragma unroll
            for (int y = 0; y < 2; y++) {
                const int f = r + y < d.H ? rfirst[r + y] : 0, l = r + y < d.H ? rlast[r + y] : 0;
                valid[y] = 2 * p + y < nrows && j >= f && j < l;
                full[y] = j - 32 >= f && j + 32 <= l;
            }
            float2 bin = make_float2(-1.0f, -1.0f);
            if ((valid[0] || valid[1]) && !direct) {
                float m0, m1;
                upk(seg[p][tx + 32], m0, m1);
                bin = cepstrum_bin<true>(&seg[p][tx], pk(full[0] ? m0 : 0.0f, full[1] ? m1 : 0.0f));
            }
#pragma unroll
            for (int y = 0; y < 2; y++) {
                const float v = y ? bin.y : bin.x;
                const bool open = valid[y] && v < 0.0f;
                val[2 * p + y][tx] = valid[y] ? __float2int_rz(v) : 0;
                const unsigned m = __ballot_sync(0xffffffffu, open);
                if (m) {
                    int at = 0;
                    if (tx == 0) at = atomicAdd(&sm.n_open, __popc(m));
                    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << tx) - 1u));
                    if (open) sm.open_cells[at] = (unsigned short)((2 * p + y) * 32 + tx);
                }
            }
        }
        __syncthreads();
        // The open cells, a thread each: the value itself.
        int formed = 0;
        for (int k = threadIdx.x; k < sm.n_open; k += kCThreads) {
            const int rr = sm.open_cells[k] >> 5, x = sm.open_cells[k] & 31;
            const float* w = reinterpret_cast<const float*>(&seg[rr >> 1][x]) + (rr & 1);
            const bool constant = constant_window(w);
            formed += !constant;
            val[rr][x] = constant ? 0 : __float2int_rz(__fdiv_rn(cepstrum_f32(w), 1000.0f));
        }
        formed = __reduce_add_sync(0xffffffffu, formed);
        if (tx == 0 && formed) atomicAdd(&sm.n_formed, formed);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (direct) {
                sm.direct--;
            } else if (sm.n_formed > nrows * 24) {  // of 32 columns
                sm.direct = sm.wait;
                sm.wait = min(2 * sm.wait, kMostDirect);
            } else {
                sm.wait = kFirstDirect;
            }
            sm.n_open = sm.n_formed = 0;  // counted again after the barrier below
        }
        if (col_ok) {
            const int off = tg[j] - tmin;
#pragma unroll 4
            for (int i = ty; i < ni; i += kCWarps) {
                const int m = max(val[i + off][tx], val[i + 1 + off][tx]);
                const int o = sm.acc[i][tx];
                sm.acc[i][tx] = m == 0x7fffffff ? kEmptied : max(o & (kEmptied - 1), m + 1) | (o & kEmptied);
            }
        }
        __syncthreads();  // seg and val are rewritten for the next sector
    }
    // The runs in order, a share of the tile's rows to each CTA.
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    const int last_angle = tl.angle[t][cnt - 1];
    for (int i = ty + kCWarps * (int)blockIdx.z; i < ni; i += kCWarps * (int)gridDim.z) {
        int o = 0;
        for (unsigned z = 0; z < gridDim.z; z++) {
            const int v = *cluster.map_shared_rank(&sm.acc[i][tx], z);
            o = v & kEmptied ? v & (kEmptied - 1) : max(o, v);
        }
        if (col_ok) A[(int64_t)(i0 + i) * dim + j] = __int2float_rn(last_angle + 1000 * (o - 1));
    }
    cluster.sync();  // no CTA leaves while another reads its rows
}

}  // namespace

cudaError_t cepstrum_f32_init_tables() {
    float2 w[64];
    for (int k = 0; k < 64; k++) {
        const double a = 2.0 * 3.14159265358979323846 * k / 64.0;
        w[k] = make_float2((float)cos(a), (float)-sin(a));
    }
    return cudaMemcpyToSymbol(c_w64, w, sizeof(w));
}

// Resident clusters of `size` CTAs of the kernel with kCRows-row tiles (0: that size
// does not run), asked once per device.
template <int kCRows>
static int resident_clusters(int size, cudaLaunchConfig_t cfg) {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices][4];  // + 1
    int dev = 0, resident = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::atomic<int>* slot = dev < kDevices ? &known[dev][size < 2 ? 0 : size < 4 ? 1 : size < 8 ? 2 : 3] : nullptr;
    if (slot && slot->load(std::memory_order_relaxed) > 0) return slot->load(std::memory_order_relaxed) - 1;
    if (cudaOccupancyMaxActiveClusters(&resident, k_cepstrum_fused<kCRows>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        resident = 0;
    }
    if (slot) slot->store(resident + 1, std::memory_order_relaxed);
    return resident;
}

namespace {
struct FusedLaunch {
    int rows = 0, runs = 1;
    double time = 0.0;  // of the slowest SM, in rows of a band
};
}  // namespace

// kCRows-row tiles: notes in best which numbers of runs take less than what it holds,
// or (null) launches with `runs`.
template <int kCRows>
static cudaError_t fused(const BatchTables& t, int images, const DevGeometry& g, const TypeLists& tl, int dim,
                         cudaStream_t st, FusedLaunch* best, int runs) {
    const int tiles_x = (dim + 31) / 32, tiles_y = (dim + kCRows - 1) / kCRows;
    const int64_t blocks = (int64_t)4 * tiles_x * tiles_y;
    if (blocks > 0x7fffffff || images > 65535) return cudaErrorInvalidValue;
    const int smem = (int)sizeof(CSmem<kCRows>);
    cudaError_t e =
        cudaFuncSetAttribute(k_cepstrum_fused<kCRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kCThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (!best) {
        attr.val.clusterDim = {1, 1, (unsigned)runs};
        cfg.gridDim = dim3((unsigned)blocks, (unsigned)images, (unsigned)runs);
        return cudaLaunchKernelEx(&cfg, k_cepstrum_fused<kCRows>, t, g, tl, dim, tiles_x, tiles_y);
    }
    int types = 0, most = 0;
    for (int k = 0; k < 4; k++) {
        types += tl.count[k] > 0;
        most = std::max(most, tl.count[k]);
    }
    const int64_t clusters = (int64_t)types * tiles_x * tiles_y * images;
    const int band = std::min(kCRows, dim) + 34 + 24;  // and what a sector costs besides its rows
    for (int s = 1; s <= 8; s *= 2) {
        attr.val.clusterDim = {1, 1, (unsigned)s};
        cfg.gridDim = dim3((unsigned)blocks, (unsigned)images, (unsigned)s);
        const int resident = resident_clusters<kCRows>(s, cfg);
        if (resident < 1) continue;
        const int64_t waves = (clusters + resident - 1) / resident;
        const double length = waves > 1 ? std::max(1.0, (double)most / s) : (double)((most + s - 1) / s);
        const double time = (double)waves * length * band;
        if (best->rows == 0 || time < 0.98 * best->time) *best = FusedLaunch{kCRows, s, time};
    }
    return cudaSuccess;
}

// Tall tiles, 256 rows, form 1.13 cepstra per skewed cell, low ones, 64, 1.5.  The rows
// and the runs of sectors per tile: of the choices whose waves of clusters, each as
// long as a run, come within 2% of the least the first, tall tiles and few runs
// before low and many.  Two images of 64x64 have 16 tiles, and walking their 45
// sectors in turn left the other SMs idle: 1009 us with one run, 342 with eight (one
// image of 256x256: 2568 and 733).  16 images of 512x512 (2048 tiles, 13.5 waves of
// 152): 34.7 ms in one run, 34.0 in two.  One sector of 512x512, 32 tall tiles or 128
// low ones: 113 and 71 us, flat 207 and 107; eight of one type, one run or four: 498
// and 169.
cudaError_t launch_cepstrum_f32(const BatchTables& t, int images, const DevGeometry& g, const TypeLists& tl, int dim,
                                cudaStream_t st) {
    if (images <= 0) return cudaSuccess;
    FusedLaunch best;
    cudaError_t e = fused<kCTall>(t, images, g, tl, dim, st, &best, 0);
    if (e == cudaSuccess && dim > kCLow) e = fused<kCLow>(t, images, g, tl, dim, st, &best, 0);
    if (e != cudaSuccess) return e;
    return best.rows == kCLow ? fused<kCLow>(t, images, g, tl, dim, st, nullptr, best.runs)
                              : fused<kCTall>(t, images, g, tl, dim, st, nullptr, best.runs);
}

}  // namespace ske
