// The steps on either side of the pursuit, on the GPU (sm_100a): clip
// gathers, robust templates and the clip noise covariance that prepare the
// pursuit's inputs (spikesorting_fullpursuit/full_binary_pursuit.py:299-322),
// duplicate removal after it (analyze_spike_timing.py), the template-sum
// search (c_cython/sort_cython.pyx:333-458), and the Wiener-filter and ZCA
// passes over the voltage (wiener_filter.py, preprocessing.py:104-169).
//
// All of it is memory-bound or latency-bound integer and float work: the
// kernels stream rows once and coalesce along the contiguous axis; the few
// sequential recurrences of the reference (duplicate scans, running sums)
// run one thread per unit or row, many units at once.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "../../include/fbp_b200.h"
#include "../../include/fbp_prepost.h"
#include "fbp_common.cuh"

namespace fbp {
int set_last_error(int code, const char *msg);
}

namespace {

using fbp::ceil_div;

int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    return fbp::set_last_error(code, buf);
}

#define PP_LAUNCH_CHECK()                                                                  \
    do {                                                                                   \
        cudaError_t e_ = cudaGetLastError();                                               \
        if (e_ != cudaSuccess)                                                             \
            return fail(FBP_ERR_CUDA, "kernel launch failed at %s:%d: %s", __FILE__,       \
                        __LINE__, cudaGetErrorString(e_));                                 \
    } while (0)
#define PP_CUDA(call)                                                                      \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess)                                                             \
            return fail(FBP_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));     \
    } while (0)

int grid_of(u64 items, int threads, int cap = 148 * 16) {
    u64 b = (items + threads - 1) / threads;
    if (b > (u64)cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

// ------------------------------------------------------------------ clips

// 2^lg lanes per (clip, channel), as many as its samples up to a warp, along the
// samples, four loads in flight: an element at a time spent its time on two
// 64-bit divisions.  Clips of 16 channels x 101 samples for 64 units: 0.27 ms in
// one launch, 0.71 ms in 64 of the kernel before.  100,000 clips of 4 channels x
// 8 samples: 14 us, 43 with a warp each, 15 an element at a time.
// kWarp: lg is 5 (100 samples took 8 % longer with a stride that varies).
template <typename T, bool kWarp>
__global__ void k_gather_clips(const T *__restrict__ v, u64 n, const long long *__restrict__ chans, u32 nch,
                               const long long *__restrict__ ev, u32 first, u32 count, int w0, u32 W, u32 lg,
                               T *__restrict__ out) {
    if (kWarp) lg = 5;
    const u32 lanes = 1u << lg, lane = threadIdx.x & (lanes - 1);
    const u64 total = (u64)count * nch, step = (u64)gridDim.x * (blockDim.x >> lg);
    for (u64 q = (u64)blockIdx.x * (blockDim.x >> lg) + (threadIdx.x >> lg); q < total; q += step) {
        const u64 e = q / nch;
        const T *src = v + (u64)chans[q - e * nch] * n + (u64)(ev[first + e] + w0);
        T *dst = out + q * W;
#pragma unroll 4
        for (u32 i = lane; i < W; i += lanes) dst[i] = src[i];
    }
}

// ------------------------------------------------------------------ robust templates

// Float order as unsigned keys (negative values reversed); +-0 differ in key
// but compare equal as values.
__device__ __forceinline__ u32 fkey(float f) {
    const u32 b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float kfloat(u32 k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// The key of a stored value, from its bits as an integer: fkey() of a value that the
// compiler knows as a float may lose the sign of a NaN.
__device__ __forceinline__ u32 stored_key(const float *p) {
    const u32 b = *reinterpret_cast<const u32 *>(p);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ u32 stored_key(const short *p) { return fkey((float)*p); }
constexpr u32 kKeyLow = 0x007fffffu, kKeyHigh = 0xff800000u;     // of the infinities: NaN lies outside

// Products rounded on their own (no contraction into a following add), as
// numpy forms an array of squares before it sums them.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// The key of the k-th smallest (0-based) of m keys, radix select by one warp
// (8-bit digits, histogram `hist` of 256 words in shared memory).
template <class KeyOf>
__device__ u32 warp_select(u32 m, u32 k, KeyOf key_of, u32 *hist) {
    const u32 lane = threadIdx.x & 31;
    u32 prefix = 0, mask = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (u32 b = lane; b < 256; b += 32) hist[b] = 0;
        __syncwarp();
        for (u32 i = lane; i < m; i += 32) {
            const u32 key = key_of(i);
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
        }
        __syncwarp();
        u32 c[8], s = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            c[j] = hist[8 * lane + j];
            s += c[j];
        }
        const u32 incl = fbp::warp_incl_scan(s), excl = incl - s;
        const bool mine = k >= excl && k < incl;
        const u32 ball = __ballot_sync(0xffffffffu, mine);
        u32 digit = 0, before = 0;
        if (mine) {
            u32 acc = excl;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (k >= acc && k < acc + c[j]) { digit = 8 * lane + j; before = acc; }
                acc += c[j];
            }
        }
        const int src = __ffs(ball) - 1;
        digit = __shfl_sync(0xffffffffu, digit, src);
        before = __shfl_sync(0xffffffffu, before, src);
        k -= before;
        prefix |= digit << shift;
        mask |= 255u << shift;
        __syncwarp();
    }
    return prefix;
}

// A warp's histogram of m values in 256 equal bins of [lo, hi], kept in
// registers (lane l holds bins 8l .. 8l + 7).  A bin's index does not decrease
// with the value, so the bins bound ranks.
// Units of more spikes than this select by radix at once: a bin in the middle of
// 256 over a normal sample's range holds 1 %, which has to stay below kBinGather.
constexpr u32 kBinMax = 4096;
constexpr u32 kBinGather = 64;         // values of one rank's bins that a warp sorts out directly
struct WarpBins {
    float lo, scale;
    u32 c[8], sum, excl;
    bool ok, all;                      // all: few values, no bins needed
    __device__ u32 bin(float x) const { return min(255u, __float2uint_rz(__fmul_rn(__fsub_rn(x, lo), scale))); }
};

template <class ValOf>
__device__ void bins_build(WarpBins &b, u32 m, float lo, float hi, ValOf val, u32 *hist) {
    const u32 lane = threadIdx.x & 31;
    const float range = __fsub_rn(hi, lo);
    b.lo = lo;
    b.scale = __fdiv_rn(256.0f, range);
    b.all = m <= kBinGather;
    b.ok = b.all || (range > 0.0f && range < 3e38f && b.scale < 3e38f);   // no NaN, no infinity
    b.sum = b.excl = 0;
    if (b.all || !b.ok) return;
    for (u32 j = lane; j < 256; j += 32) hist[j] = 0;
    __syncwarp();
#pragma unroll 4
    for (u32 i = lane; i < m; i += 32) atomicAdd(&hist[b.bin(val(i))], 1u);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; j++) {
        b.c[j] = hist[8 * lane + j];
        b.sum += b.c[j];
    }
    b.excl = fbp::warp_incl_scan(b.sum) - b.sum;
    __syncwarp();
}

// The bin that holds rank k, the values below it and in it.
__device__ __forceinline__ void bins_find(const WarpBins &b, u32 k, u32 &bin, u32 &before, u32 &count) {
    const u32 lane = threadIdx.x & 31;
    const bool mine = k >= b.excl && k < b.excl + b.sum;
    u32 acc = b.excl;
    bin = before = count = 0;
    if (mine) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (k >= acc && k < acc + b.c[j]) { bin = 8 * lane + j; before = acc; count = b.c[j]; }
            acc += b.c[j];
        }
    }
    const int src = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
    bin = __shfl_sync(0xffffffffu, bin, src);
    before = __shfl_sync(0xffffffffu, before, src);
    count = __shfl_sync(0xffffffffu, count, src);
}

// The values of ranks k0 <= k1; false if their bins hold too many values.
template <class ValOf>
__device__ bool bins_pick(const WarpBins &b, u32 m, u32 k0, u32 k1, ValOf val, u32 *buf, float &v0, float &v1) {
    const u32 lane = threadIdx.x & 31;
    u32 b0 = 0, b1 = 255, before = 0, cnt = m;
    if (!b.all) {
        u32 c0, before1, c1;
        bins_find(b, k0, b0, before, c0);
        bins_find(b, k1, b1, before1, c1);
        cnt = before1 + c1 - before;
        if (cnt > kBinGather) return false;
    }
    u32 base = 0;
#pragma unroll 4
    for (u32 i0 = 0; i0 < m; i0 += 32) {
        const u32 i = i0 + lane;
        const float x = val(min(i, m - 1));
        const u32 j = b.all ? 0u : b.bin(x);
        const bool in = i < m && j >= b0 && j <= b1;
        const u32 ball = __ballot_sync(0xffffffffu, in);
        if (in) buf[base + __popc(ball & ((1u << lane) - 1u))] = fkey(x);
        base += __popc(ball);
    }
    __syncwarp();
    const bool ina = lane < cnt, inb = lane + 32 < cnt;
    const u32 ka = ina ? buf[lane] : 0u, kb = inb ? buf[lane + 32] : 0u;
    u32 ra = 0, rb = 0;                                  // ranks, equal keys in buffer order
    for (u32 j = 0; j < cnt; j++) {
        const u32 k = buf[j];
        ra += k < ka || (k == ka && j < lane);
        rb += k < kb || (k == kb && j < lane + 32);
    }
    auto key_at = [&](u32 r) {
        const u32 at = __ballot_sync(0xffffffffu, ina && ra == r), bt = __ballot_sync(0xffffffffu, inb && rb == r);
        const u32 x = __shfl_sync(0xffffffffu, ka, at ? __ffs(at) - 1 : 0);
        const u32 y = __shfl_sync(0xffffffffu, kb, bt ? __ffs(bt) - 1 : 0);
        return at ? x : y;
    };
    v0 = kfloat(key_at(k0 - before));
    v1 = kfloat(key_at(k1 - before));
    __syncwarp();
    return true;
}

template <typename T> struct RobustArith;
template <> struct RobustArith<float> {    // numpy float32 arithmetic
    typedef float A;
    static __device__ float half_sum(float a, float b) { return __fmul_rn(__fadd_rn(a, b), 0.5f); }
    static __device__ float mad_scale(float m) { return __fdiv_rn(m, 0.6745f); }
    static __device__ float store(float x) { return x; }
};
template <> struct RobustArith<short> {    // numpy: int16 medians in float64, stored truncated
    typedef double A;
    static __device__ double half_sum(double a, double b) { return (a + b) * 0.5; }
    static __device__ double mad_scale(double m) { return __ddiv_rn(m, 0.6745); }
    static __device__ short store(double x) { return (short)__double2int_rz(x); }
};

// Column values of a unit live contiguously in the transposed clips tr[dim][n_rows].
template <typename T>
__global__ void k_transpose(const T *__restrict__ in, u32 rows, u32 cols, T *__restrict__ out) {
    __shared__ T tile[32][33];
    const u32 tiles_c = ceil_div(cols, 32), tiles_r = ceil_div(rows, 32);
    for (u64 t = blockIdx.x; t < (u64)tiles_c * tiles_r; t += gridDim.x) {
        const u32 tr = (u32)(t / tiles_c), tc = (u32)(t % tiles_c);
        for (u32 y = threadIdx.y; y < 32; y += blockDim.y) {
            const u32 r = tr * 32 + y, c = tc * 32 + threadIdx.x;
            if (r < rows && c < cols) tile[y][threadIdx.x] = in[(u64)r * cols + c];
        }
        __syncthreads();
        for (u32 y = threadIdx.y; y < 32; y += blockDim.y) {
            const u32 c = tc * 32 + y, r = tr * 32 + threadIdx.x;
            if (r < rows && c < cols) out[(u64)c * rows + r] = tile[threadIdx.x][y];
        }
        __syncthreads();
    }
}

// calculate_robust_template (preprocessing.py:639-659), one warp per
// (unit, column): the median, the median absolute deviation, and the median of
// the values strictly within one MAD of the median, which are a contiguous
// range of ranks.  What bounds it are the passes over a column's values, each
// with its keys and shared atomics.  One histogram of 256 equal bins serves
// the medians of the values and one that of the deviations (2 passes with
// atomics, 7 in all, where four digits of a radix select for each rank took up
// to 25), and equal bins put few lanes on the same counter where the first
// digit, sign and exponent, put most.  64 units of 600 spikes, 1616 columns:
// 1.18 ms, radix selects 2.11 ms.
template <typename T>
__global__ void k_robust_template(const T *__restrict__ tr, u32 n_rows, u32 dim, const u32 *__restrict__ off,
                                  u32 n_units, T *__restrict__ out) {
    typedef RobustArith<T> R;
    typedef typename R::A A;
    __shared__ u32 hist_all[8][256];
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    u32 *hist = hist_all[warp];
    const u64 items = (u64)n_units * dim;
    for (u64 it = (u64)blockIdx.x * 8 + warp; it < items; it += (u64)gridDim.x * 8) {
        const u32 u = (u32)(it / dim), col = (u32)(it % dim);
        const u32 r0 = off[u], m = off[u + 1] - off[u];
        if (m == 0) continue;
        const T *x = tr + (u64)col * n_rows + r0;
        T *dst = out + (u64)u * dim + col;
        if (m == 1) {                                  // np.squeeze(clips): the clip itself
            if (lane == 0) *dst = x[0];
            continue;
        }
        auto xv = [&](u32 i) { return (float)x[i]; };
        auto med_of = [&](const WarpBins &b, u32 a, u32 cnt, auto val) -> A {   // median of ranks [a, a + cnt)
            const u32 k0 = a + (cnt - 1) / 2, k1 = a + cnt / 2;
            float v0, v1;
            if (!b.ok || !bins_pick(b, m, k0, k1, val, hist, v0, v1)) {
                auto key = [&](u32 i) { return fkey(val(i)); };
                v0 = kfloat(warp_select(m, k0, key, hist));
                v1 = k1 == k0 ? v0 : kfloat(warp_select(m, k1, key, hist));
            }
            return k1 == k0 ? (A)v0 : R::half_sum((A)v0, (A)v1);
        };
        WarpBins bx, bd;
        bx.ok = bd.ok = false;
        float vmin = 0.0f, vmax = 0.0f;
        if (m <= kBinMax) {
            u32 kmin = 0xffffffffu, kmax = 0;
#pragma unroll 4
            for (u32 i = lane; i < m; i += 32) {
                const u32 k = stored_key(x + i);
                kmin = min(kmin, k);
                kmax = max(kmax, k);
            }
            kmin = __reduce_min_sync(0xffffffffu, kmin);
            kmax = __reduce_max_sync(0xffffffffu, kmax);
            vmin = kfloat(kmin);
            vmax = kfloat(kmax);
            // a column with NaN, which lies in no bin and has no place among few
            // values either, is the radix selection's
            if (kmin >= kKeyLow && kmax <= kKeyHigh) bins_build(bx, m, vmin, vmax, xv, hist);
        }
        const A med = med_of(bx, 0, m, xv);
        auto dv = [&](A y) {
            const A d = y - med;
            return (float)(d < (A)0 ? -d : d);          // exact in float32 for both types
        };
        auto dvi = [&](u32 i) { return dv((A)x[i]); };
        // the largest deviation is that of the smallest or the largest value (NaN: the median is infinite)
        const float dmin = dv((A)vmin), dmax = dv((A)vmax);
        if (bx.ok && dmin == dmin && dmax == dmax) bins_build(bd, m, 0.0f, fmaxf(dmin, dmax), dvi, hist);
        const A mad = R::mad_scale(med_of(bd, 0, m, dvi));
        const A lo = med - mad, hi = med + mad;
        u32 nle = 0, nlt = 0;                           // #(x <= lo), #(x < hi)
        for (u32 i = lane; i < m; i += 32) {
            const A v = (A)x[i];
            nle += v <= lo;
            nlt += v < hi;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            nle += __shfl_xor_sync(0xffffffffu, nle, o);
            nlt += __shfl_xor_sync(0xffffffffu, nlt, o);
        }
        A res = med;
        if (nlt > nle) res = med_of(bx, nle, nlt - nle, xv);
        if (lane == 0) *dst = R::store(res);
    }
}

// ------------------------------------------------------------------ clip noise covariance

template <typename T>
__device__ __forceinline__ double resid_of(const T *clips, const T *tmpl, const u32 *row_unit, u64 row, u32 dim,
                                           u32 col) {
    const T a = clips[row * dim + col], b = tmpl[(u64)row_unit[row] * dim + col];
    return (double)(T)(a - b);                      // dtype arithmetic (int16 wraps), then float64
}

template <typename T>
__global__ void k_resid_mean(const T *__restrict__ clips, const T *__restrict__ tmpl, const u32 *__restrict__ row_unit,
                             const long long *__restrict__ rows, u32 n_sel, u32 dim, double *__restrict__ sums) {
    // block: 32 columns x 8 row lanes
    const u32 col = blockIdx.x * 32 + threadIdx.x;
    if (col >= dim) return;
    double s = 0.0;
    for (u32 r = blockIdx.y * blockDim.y + threadIdx.y; r < n_sel; r += gridDim.y * blockDim.y)
        s += resid_of(clips, tmpl, row_unit, (u64)rows[r], dim, col);
    atomicAdd(&sums[col], s);
}

constexpr u32 kCovMaxLL = 12288;         // L * L: L <= 110
constexpr u32 kCovT = 4, kCovRows = 32;  // outputs of a thread a side, rows staged at a time
inline u32 cov_tiles(u32 L) { const u32 t = ceil_div(L, kCovT); return t * (t + 1) / 2; }
// Groups of threads that share a block's rows: few tiles leave a block too small
// to stage its rows, so there are as many groups as 256 threads hold.
__host__ __device__ inline u32 cov_groups(u32 tiles) { return tiles >= 128 ? 1u : min(kCovRows, 256u / tiles); }
inline u32 cov_threads(u32 L) { return ceil_div(cov_tiles(L) * cov_groups(cov_tiles(L)), 32) * 32; }
inline size_t cov_smem_bytes(u32 L) {
    const size_t rows = (size_t)kCovRows * ceil_div(L, kCovT) * kCovT + L, g = cov_groups(cov_tiles(L));
    return std::max(rows, g > 1 ? g * cov_tiles(L) * kCovT * kCovT : (size_t)0) * sizeof(double);
}

// Per channel c, sum over the selected rows of (x_i - mean_i)(x_j - mean_j),
// i, j < L; blocks take row ranges and add their partial matrix atomically.
// FP64 work: a thread holds a 4 x 4 tile of outputs, four 16-byte shared reads
// for 16 products (an output at a time took two reads for each), and only the
// tiles on and above the diagonal, the others being the same sums.  16 channels
// of 101 samples: 0.48 ms, before 1.60 ms.  Short templates (up to 60 samples) have
// fewer than 128 tiles: cov_groups() groups of threads take the rows in turn and
// add up in shared memory (4 channels x 16 samples of 1,000 clips: 27 us in all, 71
// with one group, 34 an output at a time).  kGroups: more than one.
template <typename T, bool kGroups>
__global__ void __launch_bounds__(416)
k_resid_cov(const T *__restrict__ clips, const T *__restrict__ tmpl, const u32 *__restrict__ row_unit,
            const long long *__restrict__ rows, u32 n_sel, u32 C, u32 L, const double *__restrict__ sums,
            double *__restrict__ cov) {
    extern __shared__ __align__(16) double csm[];    // [32 rows][L up to a multiple of 4] centred values, [L] means
    const u32 c = blockIdx.x, dim = C * L, nt = ceil_div(L, kCovT), Lp = nt * kCovT;
    const u32 parts = gridDim.y, part = blockIdx.y;
    const u32 r_begin = (u32)((u64)n_sel * part / parts), r_end = (u32)((u64)n_sel * (part + 1) / parts);
    double *mean = csm + kCovRows * Lp;
    for (u32 i = threadIdx.x; i < L; i += blockDim.x) mean[i] = sums[c * L + i] / n_sel;
    // tile (threadIdx.x mod tiles) of the upper triangle, row by row
    const u32 tiles = nt * (nt + 1) / 2, groups = kGroups ? cov_groups(tiles) : 1u,
              grp = threadIdx.x / tiles;
    u32 ti = 0, tj = threadIdx.x - grp * tiles;
    while (tj >= nt - ti) { tj -= nt - ti; ti++; }
    const bool mine = grp < groups;
    tj += ti;
    double acc[kCovT][kCovT];
#pragma unroll
    for (u32 a = 0; a < kCovT; a++)
#pragma unroll
        for (u32 b = 0; b < kCovT; b++) acc[a][b] = 0.0;
    for (u32 r0 = r_begin; r0 < r_end; r0 += kCovRows) {
        const u32 nr = min(kCovRows, r_end - r0);
        __syncthreads();
        for (u32 e = threadIdx.x; e < nr * Lp; e += blockDim.x) {
            const u32 rr = e / Lp, i = e % Lp;
            csm[e] = i < L ? resid_of(clips, tmpl, row_unit, (u64)rows[r0 + rr], dim, c * L + i) - mean[i] : 0.0;
        }
        __syncthreads();
        if (mine) {
            const u32 r1 = kGroups ? grp : 0u, step = groups * (Lp / 2);
            const double2 *pa = reinterpret_cast<const double2 *>(csm + r1 * Lp + ti * kCovT);
            const double2 *pb = reinterpret_cast<const double2 *>(csm + r1 * Lp + tj * kCovT);
#pragma unroll 2
            for (u32 rr = r1; rr < nr; rr += groups, pa += step, pb += step) {
                const double2 a0 = pa[0], a1 = pa[1], b0 = pb[0], b1 = pb[1];
                const double av[kCovT] = {a0.x, a0.y, a1.x, a1.y}, bv[kCovT] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
                for (u32 a = 0; a < kCovT; a++)
#pragma unroll
                    for (u32 b = 0; b < kCovT; b++) acc[a][b] = fma(av[a], bv[b], acc[a][b]);
            }
        }
    }
    double *out = cov + (u64)c * L * L;
    if (kGroups) {
        __syncthreads();                             // the rows' readers are done
        if (mine)
#pragma unroll
            for (u32 a = 0; a < kCovT; a++)
#pragma unroll
                for (u32 b = 0; b < kCovT; b++) csm[(a * kCovT + b) * groups * tiles + threadIdx.x] = acc[a][b];
        __syncthreads();
        for (u32 e = threadIdx.x; e < tiles * kCovT * kCovT; e += blockDim.x) {
            const u32 k = e / tiles, t = e - k * tiles;
            double s = 0.0;
            for (u32 g = 0; g < groups; g++) s += csm[(k * groups + g) * tiles + t];
            u32 i0 = 0, j0 = t;
            while (j0 >= nt - i0) { j0 -= nt - i0; i0++; }
            j0 += i0;
            const u32 i = i0 * kCovT + k / kCovT, j = j0 * kCovT + k % kCovT;
            if (i >= L || j >= L) continue;
            atomicAdd(&out[i * L + j], s);
            if (i0 != j0) atomicAdd(&out[j * L + i], s);
        }
        return;
    }
    if (!mine) return;
#pragma unroll
    for (u32 a = 0; a < kCovT; a++)
#pragma unroll
        for (u32 b = 0; b < kCovT; b++) {
            const u32 i = ti * kCovT + a, j = tj * kCovT + b;
            if (i >= L || j >= L) continue;
            atomicAdd(&out[i * L + j], acc[a][b]);
            if (ti != tj) atomicAdd(&out[j * L + i], acc[a][b]);
        }
}

__global__ void k_scale(double *__restrict__ x, u64 n, double f) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) x[i] *= f;
}

// ------------------------------------------------------------------ numpy's pairwise sum

// np.add.reduce over a contiguous 1-D array (numpy's pairwise summation:
// below 8 elements a plain loop from 0; up to 128 eight accumulators, then
// ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) and the remainder in order; above,
// the halves split at a multiple of 8 below n/2).  f(i) gives element i.
template <typename A, class F>
__device__ A np_pairwise(u64 i0, u64 n, F f) {
    // explicit stack instead of recursion: leaves (<= 128 elements) are
    // summed in order of their position and combined as the recursion would
    struct Fr { u64 i0, n; int state; A left; };
    Fr st[40];
    int sp = 0;
    st[0] = {i0, n, 0, (A)0};
    A ret = (A)0;
    for (;;) {
        Fr &fr = st[sp];
        if (fr.n <= 128) {
            A res;
            if (fr.n < 8) {
                res = (A)0;
                for (u64 i = 0; i < fr.n; i++) res += f(fr.i0 + i);
            } else {
                A r[8];
#pragma unroll
                for (int j = 0; j < 8; j++) r[j] = f(fr.i0 + j);
                u64 i = 8;
                for (; i < fr.n - (fr.n % 8); i += 8) {
#pragma unroll
                    for (int j = 0; j < 8; j++) r[j] += f(fr.i0 + i + j);
                }
                res = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
                for (; i < fr.n; i++) res += f(fr.i0 + i);
            }
            // return res to the parent
            for (;;) {
                if (sp == 0) { ret = res; return ret; }
                sp--;
                Fr &p = st[sp];
                if (p.state == 1) {              // left half done: do the right half
                    p.left = res;
                    p.state = 2;
                    u64 n2 = p.n / 2;
                    n2 -= n2 % 8;
                    st[++sp] = {p.i0 + n2, p.n - n2, 0, (A)0};
                    break;
                }
                res = p.left + res;              // right half done
            }
        } else {
            u64 n2 = fr.n / 2;
            n2 -= n2 % 8;
            fr.state = 1;
            st[++sp] = {fr.i0, n2, 0, (A)0};
        }
    }
}

// ------------------------------------------------------------------ duplicates

// sum((clip - template)**2) of every event, np.sum's pairwise order; the
// event's unit found by binary search of the unit offsets.
template <typename TT, typename A>
__global__ void k_event_sse(const float *__restrict__ clips, const TT *__restrict__ tmpl, u32 dim,
                            const u32 *__restrict__ off, u32 n_units, u32 n_events, double *__restrict__ sse) {
    for (u32 e = blockIdx.x * blockDim.x + threadIdx.x; e < n_events; e += gridDim.x * blockDim.x) {
        u32 lo = 0, hi = n_units;                    // last u with off[u] <= e
        while (hi - lo > 1) {
            const u32 mid = (lo + hi) / 2;
            if (off[mid] <= e) lo = mid; else hi = mid;
        }
        const float *c = clips + (u64)e * dim;
        const TT *t = tmpl + (u64)lo * dim;
        auto f = [&](u64 i) -> A {
            const A d = (A)c[i] - (A)t[i];
            return mul_rn(d, d);
        };
        sse[e] = (double)np_pairwise<A>(0, dim, f);
    }
}

// The scans of analyze_spike_timing.py, one thread per unit (curr/next as
// the reference steps them).
__global__ void k_dup_scan(int mode, const long long *__restrict__ ev, const u8 *__restrict__ bp,
                           const double *__restrict__ sse, const u32 *__restrict__ off, u32 n_units, long long tol,
                           u8 *__restrict__ keep) {
    for (u32 u = blockIdx.x * blockDim.x + threadIdx.x; u < n_units; u += gridDim.x * blockDim.x) {
        const u32 a = off[u], n = off[u + 1] - a;
        for (u32 i = 0; i < n; i++) keep[a + i] = 1;
        u32 cur = 0, nxt = 1;
        while (nxt < n) {
            const u32 ci = a + cur, ni = a + nxt;
            if (ev[ni] - ev[ci] <= tol) {
                if (mode == 0) {                         // remove_binary_pursuit_duplicates :127-152
                    if (bp[ci] && bp[ni]) {
                        if (sse[ci] <= sse[ni]) { keep[ni] = 0; nxt++; }
                        else { keep[ci] = 0; cur = nxt; nxt++; }
                    } else if (bp[ci] && !bp[ni]) {
                        nxt++;
                    } else {
                        cur = nxt; nxt++;
                    }
                } else if (mode == 1) {                  // keep_binary_pursuit_duplicates :92-111
                    if (bp[ci] && !bp[ni]) { keep[ni] = 0; nxt++; }
                    else if (!bp[ci] && bp[ni]) { keep[ci] = 0; cur = nxt; nxt++; }
                    else { cur = nxt; nxt++; }
                } else {                                 // remove_spike_event_duplicates :166-182
                    if (sse[ci] <= sse[ni]) { keep[ni] = 0; nxt++; }
                    else { keep[ci] = 0; cur = nxt; nxt++; }
                }
            } else {
                cur = nxt; nxt++;
            }
        }
    }
}

// np.mean(clips, axis=0) for float32: rows added in order, then / count.
__global__ void k_unit_mean(const float *__restrict__ clips, u32 dim, const u32 *__restrict__ off, u32 n_units,
                            float *__restrict__ out) {
    const u64 items = (u64)n_units * dim;
    for (u64 q = (u64)blockIdx.x * blockDim.x + threadIdx.x; q < items; q += (u64)gridDim.x * blockDim.x) {
        const u32 u = (u32)(q / dim), col = (u32)(q % dim);
        const u32 a = off[u], m = off[u + 1] - a;
        float s = 0.0f;
        for (u32 r = 0; r < m; r++) s = __fadd_rn(s, clips[(u64)(a + r) * dim + col]);
        out[q] = m ? __fdiv_rn(s, (float)m) : __int_as_float(0x7fc00000);
    }
}

// ------------------------------------------------------------------ template-sum search

// One warp per (item, shift1): it scans shift2 in order over its lanes and
// keeps the first strictly smallest residual; the per-shift1 results are
// combined in shift order afterwards.  The residual follows the reference
// element by element: sum = float64(t1 shifted) + float64(t2 shifted);
// (test - sum)**2 summed with numpy's pairwise order.
__device__ __forceinline__ double shifted_tpl(const float *t, u32 L, u32 d, int s) {
    // get_shifted_template: within each channel, value at sample i is the
    // template's sample i - s (0 outside)
    const u32 ch = d / L, i = d - ch * L;
    const int j = (int)i - s;
    return (j >= 0 && j < (int)L) ? (double)t[ch * L + j] : 0.0;
}

__global__ void k_overlap_tpl(const float *__restrict__ T, u32 C, u32 L, int n_pre, int n_post,
                              const u32 *__restrict__ items, u32 n_items, double *__restrict__ part_ss,
                              int *__restrict__ part_s2) {
    const u32 S = (u32)(n_pre + n_post + 1), D = C * L;
    const u32 lane = threadIdx.x & 31;
    const u64 tasks = (u64)n_items * S;
    for (u64 task = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < tasks;
         task += ((u64)gridDim.x * blockDim.x) >> 5) {
        const u32 it = (u32)(task / S), s1i = (u32)(task % S);
        const float *x = T + (u64)items[3 * it] * D;
        const float *t1 = T + (u64)items[3 * it + 1] * D;
        const float *t2 = T + (u64)items[3 * it + 2] * D;
        const int s1 = (int)s1i - n_pre;
        double best = __longlong_as_double(0x7ff0000000000000ll);   // inf
        int bs2 = -1;
        for (u32 s2i = lane; s2i < S; s2i += 32) {
            const int s2 = (int)s2i - n_pre;
            auto f = [&](u64 d) -> double {
                const double sum = shifted_tpl(t1, L, (u32)d, s1) + shifted_tpl(t2, L, (u32)d, s2);
                const double r = (double)x[d] - sum;
                return mul_rn(r, r);
            };
            const double ss = np_pairwise<double>(0, D, f);
            if (ss < best) { best = ss; bs2 = (int)s2i; }
        }
        // first strictly smallest over the warp, in shift2 order
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int os = __shfl_xor_sync(0xffffffffu, bs2, o);
            if (os >= 0 && (bs2 < 0 || ob < best || (ob == best && os < bs2))) { best = ob; bs2 = os; }
        }
        if (lane == 0) {
            part_ss[task] = best;
            part_s2[task] = bs2;
        }
    }
}

__global__ void k_overlap_tpl_pick(const double *__restrict__ part_ss, const int *__restrict__ part_s2, u32 n_items,
                                   u32 S, int n_pre, double *__restrict__ best_ss, int *__restrict__ best_shift) {
    for (u32 it = blockIdx.x * blockDim.x + threadIdx.x; it < n_items; it += gridDim.x * blockDim.x) {
        double b = __longlong_as_double(0x7ff0000000000000ll);
        int s1b = -1, s2b = -1;
        for (u32 s1 = 0; s1 < S; s1++) {             // shift1 outer, strict <: the first minimum
            const double v = part_ss[(u64)it * S + s1];
            if (part_s2[(u64)it * S + s1] >= 0 && v < b) { b = v; s1b = (int)s1; s2b = part_s2[(u64)it * S + s1]; }
        }
        best_ss[it] = b;
        best_shift[2 * it] = s1b < 0 ? 0 : s1b - n_pre;
        best_shift[2 * it + 1] = s2b < 0 ? 0 : s2b - n_pre;
    }
}

// ------------------------------------------------------------------ Wiener filter

template <typename R>
__global__ void k_power(const R *__restrict__ spec, u64 n, R *__restrict__ p) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const R re = spec[2 * i], im = spec[2 * i + 1];
        p[i] = mul_rn(re, re) + mul_rn(im, im);          // abs2: x.real**2 + x.imag**2
    }
}

// The rolling box-car of wiener_filter.py:40-59, one thread per row, the
// reference's running sums in its order and precision (the spectra's: float32
// for float32 voltage, float64 otherwise; np.sum of the first points is the
// pairwise sum), written to tmp then copied back.
template <typename R>
__global__ void k_smooth(R *__restrict__ P, u64 rows, u64 nb, long long smooth, R *__restrict__ tmp) {
    for (u64 r = (u64)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (u64)gridDim.x * blockDim.x) {
        R *x = P + r * nb, *o = tmp + r * nb;
        const long long half = smooth / 2;
        long long npts = half < (long long)nb ? half : (long long)nb;
        R run = np_pairwise<R>(0, (u64)npts, [&](u64 i) { return x[i]; });
        for (long long i = 0; i < (long long)nb; i++) {
            if (i + half < (long long)nb) { run += x[i + half]; npts += 1; }
            if (i - half > 0) { run -= x[i - half]; npts -= 1; }
            o[i] = run / (R)npts;
        }
        for (u64 i = 0; i < nb; i++) x[i] = o[i];
    }
}

// spec *= S / (S + N + 1e-9), the filter in the spectra's precision
// (wiener_optimal_filter, :124-129).
template <typename R>
__global__ void k_wiener(R *__restrict__ spec, const R *__restrict__ S, const R *__restrict__ N, u64 n) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const R f = S[i] / ((S[i] + N[i]) + (R)1e-9);
        spec[2 * i] = mul_rn(spec[2 * i], f);
        spec[2 * i + 1] = mul_rn(spec[2 * i + 1], f);
    }
}

// ------------------------------------------------------------------ ZCA

// mask[c][s] = 1 when some |v[c][s + k]| > 0.9 thr[c] for |k| <= cushion
// (np.rint(fftconvolve(|v| > thr, ones(2 cushion + 1), 'same')) > 0): a
// block takes a tile of one channel, prefix-counts the exceedances over the
// tile and its halo (block scan), and reads each window's count.
constexpr u32 kMaskThreads = 256, kMaskTile = 2048;
template <typename T>
__global__ void k_zca_mask(const T *__restrict__ v, u32 C, u64 n, const double *__restrict__ thr, int cushion,
                           u8 *__restrict__ mask) {
    extern __shared__ u32 pre[];                     // [span + 1] prefix counts
    const u64 tiles = (n + kMaskTile - 1) / kMaskTile;
    const u32 span = kMaskTile + 2 * (u32)cushion;
    const u32 per = (span + kMaskThreads - 1) / kMaskThreads;
    for (u64 t = blockIdx.x; t < tiles * C; t += gridDim.x) {
        const u32 c = (u32)(t / tiles);
        const long long s0 = (long long)(t % tiles) * kMaskTile;
        const double th = thr[c] * 0.90;
        const u32 q0 = threadIdx.x * per;
        u32 local = 0;
        for (u32 k = 0; k < per; k++) {
            const u32 q = q0 + k;
            const long long s = s0 - cushion + (long long)q;
            u32 f = 0;
            if (q < span && s >= 0 && s < (long long)n) f = fabs((double)v[(u64)c * n + (u64)s]) > th;
            if (q < span) pre[q + 1] = f;
            local += f;
        }
        const u32 ex = fbp::block_excl_scan(local, nullptr);
        u32 run = ex;
        for (u32 k = 0; k < per; k++) {
            const u32 q = q0 + k;
            if (q < span) { run += pre[q + 1]; pre[q + 1] = run; }
        }
        if (threadIdx.x == 0) pre[0] = 0;
        __syncthreads();
        for (u32 q = threadIdx.x; q < kMaskTile; q += kMaskThreads) {
            const long long s = s0 + q;
            if (s < (long long)n) mask[(u64)c * n + (u64)s] = (pre[q + 2 * cushion + 1] - pre[q]) > 0;
        }
        __syncthreads();
    }
}

// Per channel: count and sum (pass 0) or centred sum of squares (pass 1) of
// unmasked samples; blocks (channel, sample range) add their parts.  Bound by
// reading v and the mask; with one block per channel, 32 channels x 1.2 M
// samples took 4.1 ms a pass on 32 of the SMs.
template <typename T>
__global__ void k_zca_diag(const T *__restrict__ v, const u8 *__restrict__ mask, u32 C, u64 n, u64 chunk,
                           double *__restrict__ cnt, double *__restrict__ sum, int pass, double *__restrict__ ssq) {
    __shared__ double red[2][32];
    const u32 c = blockIdx.x;
    const u64 sb = blockIdx.y * chunk, se = min(n, sb + chunk);
    double a = 0.0, b = 0.0;
    const double mu = pass ? sum[c] / cnt[c] : 0.0;
    for (u64 s0 = sb + threadIdx.x; s0 < se; s0 += 4ull * blockDim.x) {
        T x[4];
        u8 mk[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const u64 s = s0 + (u64)u * blockDim.x;
            mk[u] = s < se ? mask[(u64)c * n + s] : (u8)1;
            x[u] = s < se ? v[(u64)c * n + s] : (T)0;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (mk[u]) continue;
            const double d = (double)x[u];
            if (pass) { a += (d - mu) * (d - mu); } else { a += 1.0; b += d; }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = a; red[1][threadIdx.x >> 5] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double A = 0, B = 0;
        for (u32 w = 0; w < blockDim.x / 32; w++) { A += red[0][w]; B += red[1][w]; }
        if (pass) {
            atomicAdd(&ssq[c], A);
        } else {
            atomicAdd(&cnt[c], A);
            atomicAdd(&sum[c], B);
        }
    }
}

// Off-diagonal: G[i][j] = sum of v_i v_j and P[i][j] = count over samples
// that neither channel masks; 32x32 channel tiles of the upper triangle, 2x2
// pairs per thread, samples split over blocks.  Masked samples are staged as
// 0 and the masks as 64-bit words, so that the inner step is one product and
// the count one population count per 64 samples; a stretch with a value that
// is not finite takes the loop that tests the masks (0 times it is not 0).
// Bound by shared-memory reads (four 8-byte reads per four products); one pair
// per thread over 16x16 tiles on 57 blocks took 8.8 ms for 32 channels x
// 1.2 M samples.
constexpr u32 kGramTile = 32, kGramStep = 64;
template <typename T>
__global__ void __launch_bounds__(256)
k_zca_gram(const T *__restrict__ v, const u8 *__restrict__ mask, u32 C, u64 n, u64 chunk, double *__restrict__ G,
           double *__restrict__ P) {
    __shared__ double sh[2][kGramTile][kGramStep + 1];
    __shared__ u32 okw[2][kGramTile][2];             // unmasked samples, one bit each
    const u32 tc = ceil_div(C, kGramTile);
    const u32 ti = blockIdx.x / tc, tj = blockIdx.x % tc;
    if (tj < ti) return;                             // upper triangle of tiles
    const u32 li = threadIdx.x / 16, lj = threadIdx.x % 16, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 sides = ti == tj ? 1u : 2u, yb = sides - 1;
    double g[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    u32 p[2][2] = {{0, 0}, {0, 0}};                  // at most `chunk` samples
    const u64 sb = (u64)blockIdx.y * chunk, se = min(n, sb + chunk);
    for (u64 s0 = sb; s0 < se; s0 += kGramStep) {
        bool odd = false;
#pragma unroll 4
        for (u32 q = warp; q < sides * kGramTile * 2; q += 8) {      // (side, row, half of the step)
            const u32 side = q / (kGramTile * 2), row = (q / 2) % kGramTile, half = q & 1u;
            const u32 c = (side ? tj : ti) * kGramTile + row;
            const u64 s = s0 + half * 32 + lane;
            const bool in = s < se && c < C;
            const bool ok = in && !mask[(u64)c * n + s];
            const double x = ok ? (double)v[(u64)c * n + s] : 0.0;
            odd |= !(fabs(x) <= 1.7976931348623157e308);
            sh[side][row][half * 32 + lane] = x;
            const u32 w = __ballot_sync(0xffffffffu, ok);
            if (lane == 0) okw[side][row][half] = w;
        }
        const bool masked_loop = __syncthreads_or(odd);
        u32 wx[2][2], wy[2][2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            wx[k][0] = okw[0][li + 16 * k][0]; wx[k][1] = okw[0][li + 16 * k][1];
            wy[k][0] = okw[yb][lj + 16 * k][0]; wy[k][1] = okw[yb][lj + 16 * k][1];
        }
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 2; b++) p[a][b] += __popc(wx[a][0] & wy[b][0]) + __popc(wx[a][1] & wy[b][1]);
        if (!masked_loop) {
#pragma unroll 8
            for (u32 k = 0; k < kGramStep; k++) {
                const double x0 = sh[0][li][k], x1 = sh[0][li + 16][k], y0 = sh[yb][lj][k], y1 = sh[yb][lj + 16][k];
                g[0][0] = fma(x0, y0, g[0][0]);
                g[0][1] = fma(x0, y1, g[0][1]);
                g[1][0] = fma(x1, y0, g[1][0]);
                g[1][1] = fma(x1, y1, g[1][1]);
            }
        } else {
            for (u32 k = 0; k < kGramStep; k++)
                for (int a = 0; a < 2; a++)
                    for (int b = 0; b < 2; b++)
                        if ((wx[a][k >> 5] & wy[b][k >> 5]) >> (k & 31) & 1u)
                            g[a][b] = fma(sh[0][li + 16 * a][k], sh[yb][lj + 16 * b][k], g[a][b]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const u32 ci = ti * kGramTile + li + 16 * a, cj = tj * kGramTile + lj + 16 * b;
            if (ci < C && cj < C && cj > ci) {
                atomicAdd(&G[(u64)ci * C + cj], g[a][b]);
                atomicAdd(&P[(u64)ci * C + cj], (double)p[a][b]);
            }
        }
}

__global__ void k_zca_sigma(u32 C, const double *__restrict__ G, const double *__restrict__ P,
                            const double *__restrict__ cnt, const double *__restrict__ ssq, double *__restrict__ sigma) {
    for (u32 q = blockIdx.x * blockDim.x + threadIdx.x; q < C * C; q += gridDim.x * blockDim.x) {
        const u32 i = q / C, j = q % C;
        double val;
        if (i == j) val = ssq[i] / (cnt[i] - 1.0);
        else if (i < j) val = G[q] / (P[q] - 1.0);
        else val = G[(u64)j * C + i] / (P[(u64)j * C + i] - 1.0);
        sigma[q] = val;
    }
}

template <typename T> __device__ __forceinline__ T cast_out(double x);
template <> __device__ __forceinline__ float cast_out<float>(double x) { return (float)x; }
template <> __device__ __forceinline__ short cast_out<short>(double x) { return (short)(int)__double2ll_rz(x); }

// out = Z @ v tile by tile: a block computes 32 output channels x 256
// samples, the channel sum in ascending order in float64 (16 channels of
// the voltage staged at a time).  A thread holds 8 outputs x 4 samples, so
// that 32 products take 8 shared-memory reads (32 outputs x 1 sample took 33
// and were bound by them: 435 us for 32 channels x 1.2 M samples).
template <typename T>
__global__ void __launch_bounds__(256)
k_zca_apply(const double *__restrict__ Z, const T *__restrict__ v, u32 C, u64 n, T *__restrict__ out) {
    __shared__ __align__(16) double zs[16][32];      // [channel][output]
    __shared__ double vs[16][256];
    const u32 tio = ceil_div(C, 32);
    const u64 tis = (n + 255) / 256;
    const u32 og = (threadIdx.x >> 6) * 8, sx = threadIdx.x & 63;
    for (u64 t = blockIdx.x; t < tio * tis; t += gridDim.x) {
        const u32 i0 = (u32)(t % tio) * 32;
        const u64 s0 = (t / tio) * 256;
        double acc[8][4];
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
            for (int x = 0; x < 4; x++) acc[r][x] = 0.0;
        for (u32 c0 = 0; c0 < C; c0 += 16) {
            for (u32 q = threadIdx.x; q < 32 * 16; q += blockDim.x) {
                const u32 r = q / 16, k = q % 16;
                zs[k][r] = (i0 + r < C && c0 + k < C) ? Z[(u64)(i0 + r) * C + c0 + k] : 0.0;
            }
#pragma unroll
            for (u32 k = 0; k < 16; k++)
                vs[k][threadIdx.x] = (c0 + k < C && s0 + threadIdx.x < n)
                                         ? (double)v[(u64)(c0 + k) * n + s0 + threadIdx.x] : 0.0;
            __syncthreads();
            const u32 kmax = min(16u, C - c0);
            for (u32 k = 0; k < kmax; k++) {
                double x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = vs[k][sx + 64 * i];
#pragma unroll
                for (int r = 0; r < 8; r += 2) {
                    const double2 z = *reinterpret_cast<const double2 *>(&zs[k][og + r]);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        acc[r][i] = fma(z.x, x[i], acc[r][i]);
                        acc[r + 1][i] = fma(z.y, x[i], acc[r + 1][i]);
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const u64 s = s0 + sx + 64 * i;
                if (i0 + og + r < C && s < n) out[(u64)(i0 + og + r) * n + s] = cast_out<T>(acc[r][i]);
            }
    }
}

// ------------------------------------------------------------------ separability metrics

// compute_separability_metrics + set_bp_threshold (neuron_separability.py:
// 88-152, 251-261), one block per template: template_SS as numpy's float32
// pairwise sum of the squares (the value the pursuit's -0.5 * SS comes
// from), the same sum in float64, the variance sum_c t_c^T Sigma_c t_c in
// float64, the lower confidence bound and the noise threshold in float64.
__global__ void k_separability(const float *__restrict__ T, u32 K, u32 C, u32 L, const double *__restrict__ cov,
                               double sigma_noise, double sigma_ci, float *__restrict__ ss32,
                               double *__restrict__ ss64, double *__restrict__ var, double *__restrict__ lower_ci,
                               double *__restrict__ thr_raw, double *__restrict__ thr) {
    __shared__ double red[2][32];
    const u32 D = C * L;
    for (u32 k = blockIdx.x; k < K; k += gridDim.x) {
        const float *t = T + (u64)k * D;
        double a = 0.0, b = 0.0;
        for (u32 q = threadIdx.x; q < C * L * L; q += blockDim.x) {
            const u32 c = q / (L * L), ij = q % (L * L), i = ij / L, j = ij % L;
            a += (double)t[c * L + i] * cov[(u64)c * L * L + ij] * (double)t[c * L + j];
        }
        for (u32 q = threadIdx.x; q < D; q += blockDim.x) b += (double)t[q] * (double)t[q];
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = a; red[1][threadIdx.x >> 5] = b; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double v = 0.0, s = 0.0;
            for (u32 w = 0; w < blockDim.x / 32; w++) { v += red[0][w]; s += red[1][w]; }
            const float s32 = np_pairwise<float>(0, D, [&](u64 q) { return mul_rn(t[q], t[q]); });
            // numpy: 0.5 * float32 -> float32; the bounds then in float64
            const float e32 = __fmul_rn(0.5f, s32);
            const double sd = sqrt(v);
            const double ci = (double)e32 - sigma_ci * sd;
            const double tr = -(double)e32 + sigma_noise * sd;
            ss32[k] = s32;
            ss64[k] = s;
            var[k] = v;
            lower_ci[k] = ci;
            thr_raw[k] = tr;
            thr[k] = fmax(fmax(tr, 0.0), ci);
        }
        __syncthreads();
    }
}

}  // namespace

// ================================================================== C ABI

extern "C" {

int fbp_get_clips(const void *voltage, int dtype, uint64_t n, uint32_t C, const int64_t *neighbors,
                  uint32_t nch, const int64_t *events, uint32_t first, uint32_t count, int32_t win0, int32_t win1,
                  void *clips, void *stream) {
    fbp::set_last_error(0, "");
    if (count == 0 || nch == 0) return FBP_OK;
    if (!voltage || !neighbors || !events || !clips || win1 <= win0)
        return fail(FBP_ERR_BAD_ARG, "fbp_get_clips: bad arguments");
    (void)C;
    const u32 W = (u32)(win1 - win0);
    u32 lg = 0;
    while (lg < 5 && (1u << lg) < W) lg++;
    const u64 total = ((u64)count * nch) << lg;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == FBP_F32) {
        auto k = lg == 5 ? k_gather_clips<float, true> : k_gather_clips<float, false>;
        k<<<grid_of(total, 256), 256, 0, st>>>((const float *)voltage, n, (const long long *)neighbors, nch,
                                               (const long long *)events, first, count, win0, W, lg, (float *)clips);
    } else if (dtype == FBP_I16) {
        auto k = lg == 5 ? k_gather_clips<short, true> : k_gather_clips<short, false>;
        k<<<grid_of(total, 256), 256, 0, st>>>((const short *)voltage, n, (const long long *)neighbors, nch,
                                               (const long long *)events, first, count, win0, W, lg, (short *)clips);
    }
    else
        return fail(FBP_ERR_BAD_ARG, "fbp_get_clips: dtype must be FBP_F32 or FBP_I16");
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

size_t fbp_robust_scratch_bytes(uint32_t n_rows, uint32_t dim, int dtype) {
    return (size_t)n_rows * dim * (dtype == FBP_I16 ? 2 : 4);
}

int fbp_robust_templates(const void *clips, int dtype, uint32_t n_rows, uint32_t dim, const uint32_t *off,
                         uint32_t n_units, void *templates, void *scratch, size_t scratch_bytes, void *stream) {
    fbp::set_last_error(0, "");
    if (n_units == 0 || dim == 0) return FBP_OK;
    if (!clips || !off || !templates || !scratch)
        return fail(FBP_ERR_BAD_ARG, "fbp_robust_templates: null pointer argument");
    if (dtype != FBP_F32 && dtype != FBP_I16)
        return fail(FBP_ERR_BAD_ARG, "fbp_robust_templates: dtype must be FBP_F32 or FBP_I16");
    if (scratch_bytes < fbp_robust_scratch_bytes(n_rows, dim, dtype))
        return fail(FBP_ERR_BAD_ARG, "fbp_robust_templates: scratch too small");
    cudaStream_t st = (cudaStream_t)stream;
    const u64 tiles = (u64)ceil_div(n_rows, 32) * ceil_div(dim, 32);
    const int tgrid = (int)std::min<u64>(tiles, 148ull * 32);
    const u64 items = (u64)n_units * dim;
    const int rgrid = (int)std::min<u64>((items + 7) / 8, 148ull * 64);
    if (n_rows == 0) return FBP_OK;
    if (dtype == FBP_F32) {
        k_transpose<float><<<tgrid, dim3(32, 8), 0, st>>>((const float *)clips, n_rows, dim, (float *)scratch);
        k_robust_template<float><<<rgrid, 256, 0, st>>>((const float *)scratch, n_rows, dim, off, n_units,
                                                        (float *)templates);
    } else {
        k_transpose<short><<<tgrid, dim3(32, 8), 0, st>>>((const short *)clips, n_rows, dim, (short *)scratch);
        k_robust_template<short><<<rgrid, 256, 0, st>>>((const short *)scratch, n_rows, dim, off, n_units,
                                                        (short *)templates);
    }
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

size_t fbp_noise_cov_scratch_bytes(uint32_t C, uint32_t L) { return (size_t)C * L * sizeof(double); }

int fbp_clip_noise_covariance(const void *clips, int dtype, const uint32_t *row_unit, const void *templates,
                              const int64_t *rows, uint32_t n_sel, uint32_t C, uint32_t L, double *cov,
                              void *scratch, size_t scratch_bytes, void *stream) {
    fbp::set_last_error(0, "");
    if (!clips || !row_unit || !templates || !rows || !cov || !scratch)
        return fail(FBP_ERR_BAD_ARG, "fbp_clip_noise_covariance: null pointer argument");
    if (C == 0 || L == 0 || n_sel == 0) return fail(FBP_ERR_BAD_ARG, "fbp_clip_noise_covariance: empty input");
    if (L * L > kCovMaxLL)
        return fail(FBP_ERR_BAD_ARG, "fbp_clip_noise_covariance: L = %u above 110", L);
    if (scratch_bytes < fbp_noise_cov_scratch_bytes(C, L))
        return fail(FBP_ERR_BAD_ARG, "fbp_clip_noise_covariance: scratch too small");
    cudaStream_t st = (cudaStream_t)stream;
    double *sums = (double *)scratch;
    const u32 dim = C * L;
    PP_CUDA(cudaMemsetAsync(sums, 0, (size_t)dim * 8, st));
    PP_CUDA(cudaMemsetAsync(cov, 0, (size_t)C * L * L * 8, st));
    const dim3 mb(32, 8), mg(ceil_div(dim, 32), std::min<u32>(64, ceil_div(n_sel, 8)));
    const u32 parts = std::max<u32>(1, std::min<u32>(ceil_div(n_sel, 256), ceil_div(148 * 4, C)));
    const size_t smem = cov_smem_bytes(L);
    const bool grouped = cov_groups(cov_tiles(L)) > 1;
    if (dtype == FBP_F32) {
        k_resid_mean<float><<<mg, mb, 0, st>>>((const float *)clips, (const float *)templates, row_unit,
                                               (const long long *)rows, n_sel, dim, sums);
        auto k = grouped ? k_resid_cov<float, true> : k_resid_cov<float, false>;
        k<<<dim3(C, parts), cov_threads(L), smem, st>>>((const float *)clips, (const float *)templates, row_unit,
                                                        (const long long *)rows, n_sel, C, L, sums, cov);
    } else if (dtype == FBP_I16) {
        k_resid_mean<short><<<mg, mb, 0, st>>>((const short *)clips, (const short *)templates, row_unit,
                                               (const long long *)rows, n_sel, dim, sums);
        auto k = grouped ? k_resid_cov<short, true> : k_resid_cov<short, false>;
        k<<<dim3(C, parts), cov_threads(L), smem, st>>>((const short *)clips, (const short *)templates, row_unit,
                                                        (const long long *)rows, n_sel, C, L, sums, cov);
    } else {
        return fail(FBP_ERR_BAD_ARG, "fbp_clip_noise_covariance: dtype must be FBP_F32 or FBP_I16");
    }
    k_scale<<<grid_of((u64)C * L * L, 256), 256, 0, st>>>(cov, (u64)C * L * L, 1.0 / (double)n_sel);
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_remove_duplicates(int mode, const int64_t *events, const uint8_t *bp_bool, const float *clips,
                          const void *templates, int tdtype, uint32_t dim, const uint32_t *off, uint32_t n_units,
                          uint32_t n_events, int64_t tol, double *sse, uint8_t *keep, void *stream) {
    fbp::set_last_error(0, "");
    if (n_events == 0 || n_units == 0) return FBP_OK;
    if (mode < 0 || mode > 2) return fail(FBP_ERR_BAD_ARG, "fbp_remove_duplicates: mode must be 0, 1 or 2");
    if (!events || !off || !keep || (mode != 2 && !bp_bool) || (mode != 1 && (!clips || !templates || !sse)))
        return fail(FBP_ERR_BAD_ARG, "fbp_remove_duplicates: null pointer argument");
    cudaStream_t st = (cudaStream_t)stream;
    if (mode != 1) {
        if (tdtype == FBP_F32)
            k_event_sse<float, float><<<grid_of(n_events, 128), 128, 0, st>>>(clips, (const float *)templates, dim,
                                                                                off, n_units, n_events, sse);
        else if (tdtype == FBP_F64)
            k_event_sse<double, double><<<grid_of(n_events, 128), 128, 0, st>>>(clips, (const double *)templates, dim,
                                                                                  off, n_units, n_events, sse);
        else
            return fail(FBP_ERR_BAD_ARG, "fbp_remove_duplicates: template dtype must be FBP_F32 or FBP_F64");
    }
    k_dup_scan<<<grid_of(n_units, 64), 64, 0, st>>>(mode, (const long long *)events, bp_bool, sse, off, n_units,
                                                    (long long)tol, keep);
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_unit_mean_templates(const float *clips, uint32_t dim, const uint32_t *off, uint32_t n_units,
                            float *templates, void *stream) {
    fbp::set_last_error(0, "");
    if (n_units == 0 || dim == 0) return FBP_OK;
    if (!clips || !off || !templates) return fail(FBP_ERR_BAD_ARG, "fbp_unit_mean_templates: null pointer argument");
    k_unit_mean<<<grid_of((u64)n_units * dim, 256), 256, 0, (cudaStream_t)stream>>>(clips, dim, off, n_units,
                                                                                     templates);
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

size_t fbp_overlap_template_scratch_bytes(uint32_t n_items, int32_t n_pre, int32_t n_post) {
    const size_t S = (size_t)(n_pre + n_post + 1);
    return (size_t)n_items * S * 12;
}

int fbp_overlap_template_search(const float *templates, uint32_t K, uint32_t C, uint32_t L, int32_t n_pre,
                                int32_t n_post, const uint32_t *items, uint32_t n_items, double *best_ss,
                                int32_t *best_shift, void *scratch, size_t scratch_bytes, void *stream) {
    fbp::set_last_error(0, "");
    if (n_items == 0) return FBP_OK;
    if (!templates || !items || !best_ss || !best_shift || !scratch || n_pre < 0 || n_post < 0 || L == 0 || C == 0)
        return fail(FBP_ERR_BAD_ARG, "fbp_overlap_template_search: bad arguments");
    if (scratch_bytes < fbp_overlap_template_scratch_bytes(n_items, n_pre, n_post))
        return fail(FBP_ERR_BAD_ARG, "fbp_overlap_template_search: scratch too small");
    (void)K;
    cudaStream_t st = (cudaStream_t)stream;
    const u32 S = (u32)(n_pre + n_post + 1);
    double *part_ss = (double *)scratch;
    int *part_s2 = (int *)(part_ss + (size_t)n_items * S);
    const u64 warps = (u64)n_items * S;
    k_overlap_tpl<<<grid_of(warps * 32, 256, 148 * 64), 256, 0, st>>>(templates, C, L, n_pre, n_post, items, n_items,
                                                                      part_ss, part_s2);
    k_overlap_tpl_pick<<<grid_of(n_items, 128), 128, 0, st>>>(part_ss, part_s2, n_items, S, n_pre, best_ss,
                                                               best_shift);
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_power_spectrum(const void *spec, int dtype, uint64_t rows, uint64_t nb, void *power, void *stream) {
    fbp::set_last_error(0, "");
    if (!spec || !power) return fail(FBP_ERR_BAD_ARG, "fbp_power_spectrum: null pointer argument");
    const u64 n = rows * nb;
    if (n == 0) return FBP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == FBP_F32) k_power<float><<<grid_of(n, 256), 256, 0, st>>>((const float *)spec, n, (float *)power);
    else if (dtype == FBP_F64) k_power<double><<<grid_of(n, 256), 256, 0, st>>>((const double *)spec, n, (double *)power);
    else return fail(FBP_ERR_BAD_ARG, "fbp_power_spectrum: dtype must be FBP_F32 or FBP_F64");
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_wiener_smooth(void *power, int dtype, uint64_t rows, uint64_t nb, int64_t smooth, void *scratch,
                      void *stream) {
    fbp::set_last_error(0, "");
    if (smooth <= 1 || rows == 0 || nb == 0) return FBP_OK;
    if (!power || !scratch) return fail(FBP_ERR_BAD_ARG, "fbp_wiener_smooth: null pointer argument");
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == FBP_F32)
        k_smooth<float><<<grid_of(rows, 32), 32, 0, st>>>((float *)power, rows, nb, (long long)smooth, (float *)scratch);
    else if (dtype == FBP_F64)
        k_smooth<double><<<grid_of(rows, 32), 32, 0, st>>>((double *)power, rows, nb, (long long)smooth,
                                                           (double *)scratch);
    else return fail(FBP_ERR_BAD_ARG, "fbp_wiener_smooth: dtype must be FBP_F32 or FBP_F64");
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_wiener_apply(void *spec, const void *S, const void *N, int dtype, uint64_t rows, uint64_t nb, void *stream) {
    fbp::set_last_error(0, "");
    if (!spec || !S || !N) return fail(FBP_ERR_BAD_ARG, "fbp_wiener_apply: null pointer argument");
    const u64 n = rows * nb;
    if (n == 0) return FBP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == FBP_F32)
        k_wiener<float><<<grid_of(n, 256), 256, 0, st>>>((float *)spec, (const float *)S, (const float *)N, n);
    else if (dtype == FBP_F64)
        k_wiener<double><<<grid_of(n, 256), 256, 0, st>>>((double *)spec, (const double *)S, (const double *)N, n);
    else return fail(FBP_ERR_BAD_ARG, "fbp_wiener_apply: dtype must be FBP_F32 or FBP_F64");
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

size_t fbp_zca_scratch_bytes(uint32_t C) { return ((size_t)2 * C * C + 3 * (size_t)C) * sizeof(double); }

int fbp_zca_covariance(const void *voltage, int dtype, uint32_t C, uint64_t n, const double *thr, int32_t cushion,
                       uint8_t *mask, double *sigma, void *scratch, size_t scratch_bytes, void *stream) {
    fbp::set_last_error(0, "");
    if (!voltage || !thr || !mask || !sigma || !scratch)
        return fail(FBP_ERR_BAD_ARG, "fbp_zca_covariance: null pointer argument");
    if (C == 0 || n == 0 || cushion < 0) return fail(FBP_ERR_BAD_ARG, "fbp_zca_covariance: bad sizes");
    if (scratch_bytes < fbp_zca_scratch_bytes(C)) return fail(FBP_ERR_BAD_ARG, "fbp_zca_covariance: scratch too small");
    cudaStream_t st = (cudaStream_t)stream;
    double *G = (double *)scratch, *P = G + (size_t)C * C, *cnt = P + (size_t)C * C, *sum = cnt + C, *ssq = sum + C;
    PP_CUDA(cudaMemsetAsync(G, 0, fbp_zca_scratch_bytes(C), st));
    const u32 mthreads = kMaskThreads;
    const size_t msmem = ((size_t)kMaskTile + 2 * (size_t)cushion + 2) * 4;
    if (msmem > 200 * 1024) return fail(FBP_ERR_BAD_ARG, "fbp_zca_covariance: cushion too large");
    const u64 mtiles = (n + kMaskTile - 1) / kMaskTile * C;
    // sample ranges of the sums: about four blocks per SM of the gram tiles
    // that do work (a multiple of its step, at most 2^30 samples, at most
    // 65535 ranges), and eight of the channels
    const u32 tcs = ceil_div(C, kGramTile);
    auto range = [n](u64 want) {
        const u64 c = std::max<u64>((n + want - 1) / std::max<u64>(want, 1), 4096);
        return std::min<u64>((std::max<u64>(c, (n + 65534) / 65535) + 63) / 64 * 64, 1ull << 30);
    };
    const u64 chunk = range(std::max<u64>(1, 148 * 4 / std::max(1u, tcs * (tcs + 1) / 2)));
    const u64 dchunk = range(std::max<u64>(1, 148 * 8 / C));
    const dim3 gg(tcs * tcs, (u32)((n + chunk - 1) / chunk)), dg(C, (u32)((n + dchunk - 1) / dchunk));
    if (dtype == FBP_F32) {
        const float *v = (const float *)voltage;
        if (msmem > 48 * 1024) PP_CUDA(cudaFuncSetAttribute(k_zca_mask<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem));
        k_zca_mask<float><<<(int)std::min<u64>(mtiles, 148 * 8), mthreads, msmem, st>>>(v, C, n, thr, cushion, mask);
        k_zca_diag<float><<<dg, 256, 0, st>>>(v, mask, C, n, dchunk, cnt, sum, 0, ssq);
        k_zca_diag<float><<<dg, 256, 0, st>>>(v, mask, C, n, dchunk, cnt, sum, 1, ssq);
        k_zca_gram<float><<<gg, 256, 0, st>>>(v, mask, C, n, chunk, G, P);
    } else if (dtype == FBP_I16) {
        const short *v = (const short *)voltage;
        if (msmem > 48 * 1024) PP_CUDA(cudaFuncSetAttribute(k_zca_mask<short>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem));
        k_zca_mask<short><<<(int)std::min<u64>(mtiles, 148 * 8), mthreads, msmem, st>>>(v, C, n, thr, cushion, mask);
        k_zca_diag<short><<<dg, 256, 0, st>>>(v, mask, C, n, dchunk, cnt, sum, 0, ssq);
        k_zca_diag<short><<<dg, 256, 0, st>>>(v, mask, C, n, dchunk, cnt, sum, 1, ssq);
        k_zca_gram<short><<<gg, 256, 0, st>>>(v, mask, C, n, chunk, G, P);
    } else {
        return fail(FBP_ERR_BAD_ARG, "fbp_zca_covariance: dtype must be FBP_F32 or FBP_I16");
    }
    k_zca_sigma<<<grid_of((u64)C * C, 256), 256, 0, st>>>(C, G, P, cnt, ssq, sigma);
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_zca_apply(const double *zca, const void *voltage, int dtype, uint32_t C, uint64_t n, void *out, void *stream) {
    fbp::set_last_error(0, "");
    if (!zca || !voltage || !out) return fail(FBP_ERR_BAD_ARG, "fbp_zca_apply: null pointer argument");
    if (C == 0 || n == 0) return FBP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const u64 tiles = (u64)ceil_div(C, 32) * ((n + 255) / 256);
    const int grid = (int)std::min<u64>(tiles, 148ull * 4);
    if (dtype == FBP_F32) {
        k_zca_apply<float><<<grid, 256, 0, st>>>(zca, (const float *)voltage, C, n, (float *)out);
    } else if (dtype == FBP_I16) {
        k_zca_apply<short><<<grid, 256, 0, st>>>(zca, (const short *)voltage, C, n, (short *)out);
    } else {
        return fail(FBP_ERR_BAD_ARG, "fbp_zca_apply: dtype must be FBP_F32 or FBP_I16");
    }
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

int fbp_separability_metrics(const float *templates, uint32_t K, uint32_t C, uint32_t L, const double *cov,
                             double sigma_noise, double sigma_ci, float *ss32, double *ss64, double *var,
                             double *lower_ci, double *thr_raw, double *thr, void *stream) {
    fbp::set_last_error(0, "");
    if (K == 0) return FBP_OK;
    if (!templates || !cov || !ss32 || !ss64 || !var || !lower_ci || !thr_raw || !thr || C == 0 || L == 0)
        return fail(FBP_ERR_BAD_ARG, "fbp_separability_metrics: bad arguments");
    k_separability<<<std::min<u32>(K, 148 * 8), 256, 0, (cudaStream_t)stream>>>(
        templates, K, C, L, cov, sigma_noise, sigma_ci, ss32, ss64, var, lower_ci, thr_raw, thr);
    PP_LAUNCH_CHECK();
    return FBP_OK;
}

}  // extern "C"
