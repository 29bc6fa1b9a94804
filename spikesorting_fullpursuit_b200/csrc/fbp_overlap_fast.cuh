// Fast overlap recheck with exact refinement (sm_100a).
//
// The reference's overlap_recheck_indices (binary_pursuit.cl:444-654)
// evaluates, for each candidate window and every (a, b, t) item, the
// likelihood of the clipped sum of the best template k0 shifted by
// da = a - n_max and template t shifted by db = b - n_max, over the window
// [i0, i0+L), with C*L multiply-adds per item.  In exact arithmetic that
// value splits into
//
//     LL(t,a,b) = G(a) + H(t,b) - X(k0,t,a,b)
//     H(t,b)    = <t_t shifted by db, window>  - 0.5 * ||t_t clipped||^2   (G(a) = H(k0,a))
//     X         = <t_k0 shifted by da, t_t shifted by db>, both clipped to the window
//
// H is a small per-candidate correlation; X depends only on the templates
// and is read from prefix sums Q[k0][t][r][m] of the channel-summed product
// t_k0[m] * t_t[m+r] (r = da - db):  X = Q[hi] - Q[lo] with
// lo = max(0, -r, -da), hi = min(L, L-r, L-da).
//
// Each item gets an interval [lo, hi] guaranteed to contain the
// reference's IEEE-binary32 value: the reference's own rounding is bounded by
// gamma_n * (sum |s_j v_j| + sum s_j^2) with n the number of non-zero terms,
// and sum |s_j v_j| <= (||F_a|| + ||T_b||) * ||window||,
// sum s_j^2 <= ||F_a||^2 + ||T_b||^2 + 2|X|; kappa below covers twice that
// (the reference's error plus this approximation's).  Only items whose
// interval can reach the best one are re-evaluated exactly, in the
// reference's order; the parse kernel's strict-greater scan over single-item
// groups (.cl:699-706) then picks the same item as the reference.
#pragma once
#include "fbp_kernels.cuh"

namespace fbp {

// Contenders of all candidates of a pass share one pool of (slot, item)
// pairs; a candidate whose contenders do not fit goes to the exact kernel.
constexpr float kUnitRoundoff = 5.9604644775390625e-08f;   // 2^-24

// Constants of one chunk (computed on the device once per call).
struct OvConst {
    float kappa_ref;      // bound of the reference's rounding, per unit of sum|terms|
    float kappa_mine;     // bound of this approximation's rounding
    float kappa_rows;     // bound of the rounding of the best template's own rows (k_ov_rows)
    u32 cnz_max;          // max non-zero channels of a template
};

struct OvArgs {
    u32 n, C, K, L, nmax, S;
    const float *v, *T, *thr;
    float *Lk;
    const float *NT, *sNT, *tnorm;   // [K][S], [K][S], [K]
    const float *Q;                  // [K][K][2L-1][L+1]
    const float *XMr;                // [K][K][2L+1] upper bound of -X + kx|X| per lag r = a - b
    const float *XMw;                // [K][K][2L+32] XMr's largest value over the 32 lags from i - L - 31
                                     //               (NULL: XM stands for it)
    const float *XM;                 // [K][K]       its largest value over the lags
    const OvConst *oc;
    const u32 *cand, *n_cand;
    u32 *best_idx, *best_lab, *ov_idx, *ov_lab;
    float *best_ll;
    u8 *ovr;
    float *H;                        // [slot][K][S]
    float *vn;                       // [slot]     ||window|| over all channels (FP32 path)
    u8 *cskip;                       // [slot]
    float *cand_lb;                  // [slot]     largest lower bound of an item (atomic max, >= 0)
    float *ga_lo, *ga_hi;            // [slot][S]  interval of G(a) = H[k0][a]
    u32 *ga_bits;                    // [slot][ceil(S/32)] rows a with L[k0][afix] not <= 0
    float *ga_max, *ga_abs;          // [slot]     largest in-bounds hi(a), largest |hi(a)|
    unsigned long long *scan_next;   // next (candidate, template) pair of the scan
    u32 *seed_a1;                    // [slot]     in-bounds row a of largest lower bound
    float *pair_mb, *pair_mabs;      // [slot][K]  per (candidate, template): largest in-bounds upper
                                     //            bound of a row b and of its magnitude (from the seed;
                                     //            NULL with k_ov_tcw's tables, which keep the first)
    float *pair_v1;                  // [slot][K]  k_ov_tcw: largest lower bound of an in-bounds row b
    u16 *pair_b1;                    // [slot][K]  and its row
    uint4 *slot_tab;                 // [slot]     k_ov_tcw: window start (~0: skipped), fp16 scale exponent,
                                     //            ||k0|| (float bits)
    const float *vwmax;              // [W + 2]    bound on |v| of each window (k_ov_tcw's scale)
    const u32 *tsup;                 // [K][2] non-zero channel range of each template (may be NULL)
    u32 *pool_total;                 // appended entries this pass
    u32 pool_cap;
    u32 *pool_slot;                  // [pool_cap]
    u32 *pool_item;                  // [pool_cap]
    float *pool_hi;                  // [pool_cap] upper bound of the contender
    u32 *refined;                    // contenders evaluated exactly this pass
    u64 *best_key;                   // [slot] packed (value, ~item) of the best refined contender
    u8 *fallback;                    // [slot]
    u64 *items_evaluated;
    // H from the tensor cores: its rounding bound replaces kappa_mine, plus
    // the fp16 subnormal terms (see fbp_lik_tc.cuh)
    float km_override;               // > 0: bound of the tensor-core tables
    const float *tabs;               // [K] ||t||_1
    const int *texp;                 // [K] template scale exponents
    const int *kexp_tile;            // [group][slot][stiles] window scale exponents of k_lik_tc<1>'s tables
    const u32 *tgrp;                 // [K] template group of the tensor-core tables (NULL: one group)
    u32 kt_slots;                    // slots per group in kexp_tile
    u32 stiles;
    LazyLk lazy;                     // approximate likelihood entries (tensor-core path)
};

__device__ __forceinline__ float warp_max_f(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// ---------------------------------------------------------------- per chunk

// NT[t][b] = sum_c sum_{j in J(db)} T[t][c][j-db]^2 (clipped energy), sNT its
// square root, tnorm[t] = ||t||, and the widest count of non-zero channels.
// One block per template: the energy of every lag over the template's
// channels once, in shared memory, then each shift adds its own lags (a
// thread per (template, shift) that read every channel and lag again took
// 4.6 ms for 300 templates on 384 channels, 0.03 ms now).
constexpr int kChunkTabThreads = 128;
__global__ void __launch_bounds__(kChunkTabThreads)
k_ov_chunk_tables(const float *__restrict__ T, u32 K, u32 C, u32 L, u32 nmax, float *__restrict__ NT,
                  float *__restrict__ sNT, float *__restrict__ tnorm, OvConst *oc, const u32 *__restrict__ tsup) {
    extern __shared__ double lag_e[];                // [L]
    __shared__ u32 nz;
    const u32 S = 2 * nmax + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (u32 t = blockIdx.x; t < K; t += gridDim.x) {
        const u32 clo = tsup ? tsup[2 * t] : 0u, chi = tsup ? tsup[2 * t + 1] : C;
        const float *tt = T + (size_t)t * C * L;
        __syncthreads();                             // the previous template's readers are done
        if (threadIdx.x == 0) nz = 0;
        for (u32 m = threadIdx.x; m < L; m += blockDim.x) {
            double e = 0.0;
            for (u32 c = clo; c < chi; c++) {
                const double x = tt[(size_t)c * L + m];
                e += x * x;
            }
            lag_e[m] = e;
        }
        __syncthreads();
        for (u32 c = clo + warp; c < chi; c += blockDim.x >> 5) {
            bool any = false;
            for (u32 m = lane; m < L; m += 32) any |= tt[(size_t)c * L + m] != 0.0f;
            if (__any_sync(0xffffffffu, any) && lane == 0) atomicAdd(&nz, 1u);
        }
        for (u32 b = threadIdx.x; b <= S; b += blockDim.x) {   // b == S: the whole template
            const int d = b < S ? (int)b - (int)nmax : 0;
            const int m0 = max(0, -d), m1 = min((int)L, (int)L - d);
            double acc = 0.0;
            for (int m = m0; m < m1; m++) acc += lag_e[m];
            if (b < S) {
                NT[(size_t)t * S + b] = (float)(acc * (1.0 + 1e-6));
                sNT[(size_t)t * S + b] = (float)(sqrt(acc) * (1.0 + 1e-6));
            } else {
                tnorm[t] = (float)(sqrt(acc) * (1.0 + 1e-6));
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) atomicMax(&oc->cnz_max, nz);
    }
}

// The rounding bounds from the widest template (cnz_max, k_ov_chunk_tables).
__global__ void k_ov_const(u32 C, u32 L, OvConst *oc) {
    // gamma_n with n the reference's non-zero terms: products of two
    // templates' channels, the per-channel subtractions and sums of
    // squares, each product carrying two roundings
    const u32 cmax = oc->cnz_max;
    const double u = (double)kUnitRoundoff;
    const double n_ref = 2.0 * cmax * L + C + 2.0 * L + 16.0;
    const double n_mine = (double)cmax * L + 8.0;
    oc->kappa_ref = (float)(1.05 * n_ref * u / (1.0 - n_ref * u));
    oc->kappa_mine = (float)(1.05 * n_mine * u / (1.0 - n_mine * u));
    oc->kappa_rows = (float)(1.05 * ((double)L + cmax + 8.0) * u);   // a channel's lags, then the channels
}

// Whether no channel lies in both templates' supports: their cross term is 0
// for every shift, and the pair has no entry in Q and XMr.
__device__ __forceinline__ bool ov_disjoint(const u32 *__restrict__ tsup, u32 a, u32 b) {
    return tsup && max(tsup[2 * a], tsup[2 * b]) >= min(tsup[2 * a + 1], tsup[2 * b + 1]);
}

// ---------------------------------------------------------------- per pass

// Skip rules of .cl:518-527 and the per-candidate state.  The norms of the
// candidate's window come from the tensor-core likelihood, per template group
// (ov_window_norms); the FP32 path, which keeps none, sums the window over all
// channels (one warp per candidate).
__global__ void k_ov_prep(OvArgs A, u32 slots, u32 *__restrict__ fb_count) {
    const u32 nc = *A.n_cand;
    if (blockIdx.x == 0 && threadIdx.x == 0) {       // the pass's counters
        *A.pool_total = 0;
        *A.refined = 0;
        *A.scan_next = 0;
        *fb_count = 0;
    }
    for (u32 g = blockIdx.x * blockDim.x + threadIdx.x; g < slots; g += gridDim.x * blockDim.x) A.fallback[g] = 0;
    const bool sum = A.lazy.wn == nullptr;
    const u32 lane = sum ? threadIdx.x & 31 : 0u, per = sum ? 32u : 1u;
    for (u32 g = (blockIdx.x * blockDim.x + threadIdx.x) / per; g < nc; g += gridDim.x * blockDim.x / per) {
        const u32 id = A.cand[g];
        const u32 lab = A.best_lab[id], bidx = A.best_idx[id];
        const float bll = A.Lk[(size_t)lab * A.n + bidx];
        const bool skip = (bll < A.thr[lab]) || (bidx >= A.n - A.L);
        if (sum) {
            double e = 0.0;
            if (!skip)
                for (u32 q = lane; q < A.C * A.L; q += 32) {
                    const double x = A.v[(size_t)(q / A.L) * A.n + bidx + q % A.L];
                    e += x * x;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if (lane == 0) A.vn[g] = (float)(sqrt(e) * (1.0 + 1e-6));
        }
        if (lane == 0) {
            A.cskip[g] = skip;
            A.best_key[g] = 0ull;
            A.cand_lb[g] = 0.0f;
            if (A.slot_tab) {
                // the window's samples lie in its recording window and the next
                const float mm = fmaxf(A.vwmax[id], A.vwmax[id + 1]);
                int kexp = 0;
                if (mm > 0.0f) {
                    int e;
                    frexpf(mm, &e);                  // mm < 2^e
                    kexp = max(-126, min(126, 14 - e));      // scaled magnitudes < 2^14
                }
                A.slot_tab[g] = make_uint4(skip ? 0xffffffffu : bidx, (u32)kexp, __float_as_uint(A.tnorm[lab]), 0u);
            }
        }
    }
}

// H[g][t][b] for every template t and shift b of candidate g: correlation of
// t shifted by db with the window voltage (zero outside [i0, i0+L)), minus
// half the clipped energy.  FP32 FMA; its error is inside kappa.
// Thread tile: 8 shifts x 8 templates; per channel the window strip and the
// templates' channel slab ([m][t], t contiguous, `pad` floats between rows) are
// staged in shared memory, the slab by asynchronous copies along a template's
// samples: read template by template, a warp's load touched 32 sectors.  Blocks
// of 128 threads where that many tiles cover the table (more blocks an SM, no
// idle warps).  Bound by the FP32 pipe: 64 templates of 16 channels x 101
// samples, 26 passes, 14.0 ms, 15.5 ms before.
constexpr int kTabThreads = 256;
__global__ void __launch_bounds__(kTabThreads)
k_ov_tables(OvArgs A, u32 pad) {
    extern __shared__ __align__(16) float sm[];
    const u32 S = A.S, K = A.K, L = A.L, C = A.C, nmax = A.nmax;
    const u32 Lp = (L + 7) & ~7u;                  // lags padded to 8
    const u32 Sg = (S + 7) / 8, Kg = (K + 7) / 8;  // output groups
    const u32 Sp = Sg * 8, Kp = Kg * 8;
    const u32 strip_len = Sp + Lp + 8;
    float *strip = sm;                             // [strip_len]
    const u32 Kq = Kp + pad, lane = threadIdx.x & 31;
    float *slab = sm + strip_len;                  // [Lp][Kq]
    const u32 nc = *A.n_cand;
    const u32 groups = Sg * Kg;
    for (u32 g = blockIdx.x; g < nc; g += gridDim.x) {
        if (A.cskip[g]) continue;
        const u32 id = A.cand[g];
        const u32 bidx = A.best_idx[id];
        for (u32 gb = 0; gb < groups; gb += blockDim.x) {
            const u32 my = gb + threadIdx.x;
            const bool active = my < groups;
            const u32 sg = active ? my % Sg : 0, kg = active ? my / Sg : 0;
            float acc[8][8];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
            for (u32 c = 0; c < C; c++) {
                __syncthreads();
                // strip[x] = window voltage at position i0 - nmax + x (zero outside [i0, i0+L))
                for (u32 x = threadIdx.x; x < strip_len; x += blockDim.x) {
                    const int rel = (int)x - (int)nmax;   // position relative to i0
                    strip[x] = (rel >= 0 && rel < (int)L) ? A.v[(size_t)c * A.n + bidx + rel] : 0.0f;
                }
                for (u32 t = threadIdx.x >> 5; t < Kp; t += blockDim.x >> 5)
                    for (u32 m = lane; m < Lp; m += 32) {
                        float *dst = slab + m * Kq + t;
                        if (m < L && t < K)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                             (u32)__cvta_generic_to_shared(dst)),
                                         "l"(A.T + ((size_t)t * C + c) * L + m)
                                         : "memory");
                        else
                            *dst = 0.0f;
                    }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                if (!active) continue;
                const float *sp = strip + sg * 8;
                const float *tp = slab + kg * 8;
                for (u32 m0 = 0; m0 < Lp; m0 += 8) {
                    float w[16];
#pragma unroll
                    for (int q = 0; q < 16; q++) w[q] = sp[m0 + q];
#pragma unroll
                    for (int mm = 0; mm < 8; mm++) {
                        const float4 t0 = *reinterpret_cast<const float4 *>(tp + (m0 + mm) * Kq);
                        const float4 t1 = *reinterpret_cast<const float4 *>(tp + (m0 + mm) * Kq + 4);
                        const float tv[8] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y, t1.z, t1.w};
#pragma unroll
                        for (int i = 0; i < 8; i++)
#pragma unroll
                            for (int j = 0; j < 8; j++) acc[i][j] = fmaf(tv[j], w[i + mm], acc[i][j]);
                    }
                }
            }
            if (active) {
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const u32 t = kg * 8 + j;
                    if (t >= K) continue;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const u32 b = sg * 8 + i;
                        if (b < S)
                            A.H[((size_t)g * K + t) * S + b] = acc[i][j] - 0.5f * A.NT[(size_t)t * S + b];
                    }
                }
            }
        }
    }
}

// H[g][t][b] for masked templates (each non-zero on a narrow channel range):
// block = (candidate, group of 32 templates in support order); the group's
// channels of the window, zero-padded by n_max on both sides, are staged in
// chunks; warp w takes slots 4w..4w+3 of the group, lane l the shifts
// b = l + 32k, and each (channel, lag) step is one broadcast template value
// times a contiguous row of the window.  Only the templates' own channels
// are summed (the others add zero).  FP32 FMA in any order: the error bound
// of the tables covers it.
constexpr int kTabMThreads = 256;
constexpr int kTabMGroup = 32;
constexpr int kTabMChan = 16;            // staged channels per chunk
constexpr int kTabMShiftChunks = 16;     // S <= 512
__host__ __device__ inline size_t tables_m_smem_bytes(u32 S, u32 L) {
    return (size_t)kTabMChan * (S + L - 1) * 4;
}
__global__ void __launch_bounds__(kTabMThreads)
k_ov_tables_m(OvArgs A, const u32 *__restrict__ tperm, const u32 *__restrict__ tsup,
              const u32 *__restrict__ grange32) {
    extern __shared__ float wp[];                   // [kTabMChan][S + L - 1]
    const u32 S = A.S, K = A.K, L = A.L, nmax = A.nmax;
    const u32 P = S + L - 1;
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 nk = (S + 31) / 32;
    const u32 ng = (K + kTabMGroup - 1) / kTabMGroup;
    const u32 nc = *A.n_cand;
    for (u64 item = blockIdx.x; item < (u64)nc * ng; item += gridDim.x) {
        const u32 g = (u32)(item / ng), tg = (u32)(item % ng);
        if (A.cskip[g]) continue;
        const u32 i0 = A.best_idx[A.cand[g]];
        const u32 glo = grange32[2 * tg], ghi = grange32[2 * tg + 1];
        u32 tq[4], lo[4], hi[4];
        u32 wlo = 0xffffffffu, whi = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const u32 sl = tg * kTabMGroup + warp * 4 + q;
            tq[q] = sl < K ? tperm[sl] : 0u;
            lo[q] = sl < K ? tsup[2 * tq[q]] : 0u;
            hi[q] = sl < K ? tsup[2 * tq[q] + 1] : 0u;
            if (hi[q] > lo[q]) { wlo = min(wlo, lo[q]); whi = max(whi, hi[q]); }
        }
        float acc[4][kTabMShiftChunks];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int k = 0; k < kTabMShiftChunks; k++) acc[q][k] = 0.0f;
        for (u32 c0 = glo; c0 < ghi; c0 += kTabMChan) {
            const u32 cc = min((u32)kTabMChan, ghi - c0);
            __syncthreads();
            for (u32 e = threadIdx.x; e < cc * P; e += blockDim.x) {
                const u32 c = e / P, x = e % P;
                const int rel = (int)x - (int)nmax;          // position relative to i0
                wp[e] = (rel >= 0 && rel < (int)L) ? A.v[(size_t)(c0 + c) * A.n + i0 + rel] : 0.0f;
            }
            __syncthreads();
            const u32 cb = max(c0, wlo), ce = min(c0 + cc, whi);
            for (u32 c = cb; c < ce; c++) {
                const float *row = wp + (size_t)(c - c0) * P + lane;
                const float *tp[4];
                bool on[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    on[q] = c >= lo[q] && c < hi[q];
                    tp[q] = A.T + ((size_t)tq[q] * A.C + c) * L;
                }
                for (u32 m = 0; m < L; m++) {
                    float tv[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) tv[q] = on[q] ? __ldg(tp[q] + m) : 0.0f;
#pragma unroll
                    for (int k = 0; k < kTabMShiftChunks; k++) {
                        if ((u32)k >= nk) break;
                        // m + b <= P - 1 for every b < S; lanes past S read nothing
                        const float wv = (lane + 32u * k < S) ? row[m + 32 * k] : 0.0f;
#pragma unroll
                        for (int q = 0; q < 4; q++) acc[q][k] = fmaf(tv[q], wv, acc[q][k]);
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const u32 sl = tg * kTabMGroup + warp * 4 + q;
            if (sl >= K) continue;
            const u32 t = tq[q];
#pragma unroll
            for (int k = 0; k < kTabMShiftChunks; k++) {
                const u32 b = lane + 32 * k;
                if ((u32)k < nk && b < S)
                    A.H[((size_t)g * K + t) * S + b] = acc[q][k] - 0.5f * A.NT[(size_t)t * S + b];
            }
        }
    }
}

constexpr int kScanThreads = 256;
// Per-warp scratch of the scan: hb_lo, hb_hi (S floats each), per block of 32
// rows b the bits of rows with L[t][ashift] not <= 0 and the largest upper
// bound, the rows a's bits and upper bounds (blocks of 32), the lag bounds of
// a block of rows a against one of rows b by their distance, the pair's lag
// bounds, and a queue of items.
__host__ __device__ inline size_t sweep_warp_bytes(u32 S, u32 L) {
    const size_t NB = (S + 31) / 32;
    return align_up((size_t)8 * S + NB * 12 + NB * 128 + 2 * NB * 128 + (size_t)(2 * L + 1) * 4 + 64 * 4, 16);
}
__host__ __device__ inline size_t scan_smem_bytes(u32 S, u32 L) {
    return (size_t)(kScanThreads / 32) * sweep_warp_bytes(S, L);
}
__host__ __device__ inline size_t tables_smem_bytes(u32 S, u32 K, u32 L) {
    const size_t Lp = (L + 7) & ~7u, Sp = (size_t)(S + 7) / 8 * 8, Kp = (size_t)(K + 7) / 8 * 8;
    return (Sp + Lp + 8 + Lp * Kp) * 4;
}
constexpr int kSeedThreads = 256;

// Cross term X of one item from the pair's prefix table.
__device__ __forceinline__ float ov_x(const float *__restrict__ q, u32 L, int a_minus_nmax, int r) {
    float X = 0.0f;
    if (r > -(int)L && r < (int)L) {
        const int lo_m = max(max(0, -r), -a_minus_nmax);
        const int hi_m = min(min((int)L, (int)L - r), (int)L - a_minus_nmax);
        if (lo_m < hi_m) {
            const float *qr = q + (size_t)(r + (int)L - 1) * (L + 1);
            X = qr[hi_m] - qr[lo_m];
        }
    }
    return X;
}
// L2 (and, for tensor-core tables, L1) norm of a candidate's window over
// channels that hold template t's support: the likelihood's own norms of the
// sample the window starts at, over t's template group (written this pass: a
// candidate's window is listed), or the FP32 path's over all channels.  On
// the 384-channel probe the group's norm is about a third of the whole.
__device__ __forceinline__ void ov_window_norms(const OvArgs &A, u32 g, u32 bidx, u32 t, float &l2, float &l1) {
    if (A.lazy.wn) {
        const size_t i = (A.lazy.tgrp ? (size_t)A.lazy.tgrp[t] * A.lazy.gstride : 0) + bidx;
        l2 = A.lazy.wn[i];
        l1 = A.lazy.wa ? A.lazy.wa[i] : A.lazy.wa_f * l2;
    } else {
        l2 = A.vn[g];
        l1 = 0.0f;
    }
}

// Interval of a row term H[t][b], the rounding of the cross term (eqt)
// included, with the fp16 subnormal terms of tensor-core tables (sub0 / sub1
// scaled by the tile's voltage exponent).
struct OvRowB {
    float vn, krm, eqt, sub0, sub1;
};
__device__ __forceinline__ OvRowB ov_row_b(const OvArgs &A, u32 g, u32 bidx, u32 k0, u32 t, float krm) {
    OvRowB r;
    float l1;
    ov_window_norms(A, g, bidx, t, r.vn, l1);
    r.krm = krm;
    r.eqt = 4.0f * kUnitRoundoff * A.tnorm[k0] * A.tnorm[t];
    r.sub0 = r.sub1 = 0.0f;
    if (A.texp) {
        r.sub1 = 2.98023224e-08f * 1.001f * ldexpf(l1, -A.texp[t]);
        r.sub0 = 2.98023224e-08f * 1.001f * A.tabs[t];
        if (A.slot_tab) r.sub1 += ldexpf(r.sub0, -(int)A.slot_tab[g].y);   // one scale per candidate
    }
    return r;
}
__device__ __forceinline__ void ov_row_interval(const OvArgs &A, u32 g, u32 tmpl, u32 x, float Hv, float snt,
                                                const OvRowB &r, float &lo, float &hi) {
    // the clipped energy as the square of its root: the roundings are far inside the tables' bound
    float sx = r.sub1;
    if (A.kexp_tile) {
        // scale exponent of the table tile: per template group, candidate, tile of 128 shifts
        const size_t grp = A.tgrp ? (size_t)A.tgrp[tmpl] * A.kt_slots : 0;
        sx += r.sub0 * ldexpf(1.0f, -A.kexp_tile[(grp + g) * A.stiles + x / 128]);
    }
    const float e = r.krm * (snt * r.vn + snt * snt) + 4.0f * kUnitRoundoff * fabsf(Hv) + r.eqt + sx;
    lo = Hv - e;
    hi = Hv + e;
}

// Per-candidate constants of the row intervals.
struct OvCand {
    u32 id, k0, bidx, xlo, xhi_ex;
    float lbest;
};
__device__ __forceinline__ OvCand ov_cand(const OvArgs &A, u32 g) {
    OvCand c;
    c.id = A.cand[g];
    c.k0 = A.best_lab[c.id];
    c.bidx = A.best_idx[c.id];
    c.lbest = A.best_ll[c.id];
    c.xlo = c.bidx >= A.nmax ? 0u : A.nmax - c.bidx;          // in-bounds shifts (.cl:534-541)
    c.xhi_ex = A.n - A.L + A.nmax - c.bidx;                    // first out-of-bounds shift
    return c;
}
__device__ __forceinline__ float ov_kx(const OvArgs &A) { return 2.0f * A.oc->kappa_ref + 4.0f * kUnitRoundoff; }
__device__ __forceinline__ float ov_krm(const OvArgs &A) {
    return A.oc->kappa_ref + (A.km_override > 0.0f ? A.km_override : A.oc->kappa_mine);
}
// Slack for the float roundings of the pruning sums (2^-18 relative).
constexpr float kPruneSlack = 3.814697265625e-06f;

// Per chunk and template pair (k0, t) with a channel in common:
//   Q[k0][t][ri][m] = sum_{m' < m} sum_c T[k0][c][m'] * T[t][c][m'+r], r = ri-(L-1),
//     accumulated in double, stored in float;
//   XMr[k0][t][r + L] = an upper bound of -X + kx|X| over every shift a of an
//     item with lag r = a - b (X = 0 where the clipped templates do not
//     overlap), and XM[k0][t] = its maximum over r.  Then
//         hi(a, b) <= hiA(a) + hiB(b) + XMr[a - b]
//     bounds every item's interval without its cross term;
//   XMw[k0][t][i] = the maximum of XMr over the lags i - L - 31 .. i - L, for the
//     32 rows b of a block against one row a.
// Pairs without a common channel only get XM = 0; readers take X = 0 and
// XMr = 0 for them (ov_disjoint).  One block per pair: the shared channels of
// both templates in shared memory as doubles (stage_ch of them at most,
// otherwise global reads), one thread per lag accumulating down its row of Q
// in shared memory, the bounds from there (a warp per lag, lanes over the
// shifts), and one coalesced copy of Q to global memory.  Bound by double
// conversions and the accumulation; a thread per row writing Q with a stride
// of L + 1 and a second kernel reading it back took 13.6 ms for 300 templates
// on 384 channels (92 % of the pairs disjoint) and 1.9 ms for 64 on 16.
constexpr int kPairThreads = 256;
__host__ __device__ inline size_t pair_smem_bytes(u32 L, u32 stage_ch) {
    return align_up((size_t)(2 * L - 1) * (L + 1) * 4, 8) + (size_t)2 * stage_ch * L * 8;
}
__global__ void __launch_bounds__(kPairThreads)
k_ov_pairs(const float *__restrict__ T, u32 K, u32 C, u32 L, u32 nmax, const u32 *__restrict__ tsup, u32 stage_ch,
           const OvConst *__restrict__ oc, float *__restrict__ Q, float *XMr, float *__restrict__ XMw,
           float *__restrict__ XM) {
    extern __shared__ __align__(16) unsigned char psm[];
    const u32 R = 2 * L - 1, S = 2 * nmax + 1, NR = 2 * L + 1;
    float *qs = (float *)psm;                        // [R][L+1]
    double *sk = (double *)(psm + align_up((size_t)R * (L + 1) * 4, 8)), *st = sk + (size_t)stage_ch * L;
    const float kx = 2.0f * oc->kappa_ref + 4.0f * kUnitRoundoff;
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    __shared__ float red[kPairThreads / 32];
    for (u32 pair = blockIdx.x; pair < K * K; pair += gridDim.x) {
        const u32 k0 = pair / K, t = pair % K;
        const u32 clo = tsup ? max(tsup[2 * k0], tsup[2 * t]) : 0u;
        const u32 chi = tsup ? min(tsup[2 * k0 + 1], tsup[2 * t + 1]) : C;
        if (clo >= chi) {
            if (threadIdx.x == 0) XM[pair] = 0.0f;
            continue;
        }
        const u32 nch = chi - clo;
        const bool staged = nch <= stage_ch;
        const float *ta = T + ((size_t)k0 * C + clo) * L, *tb = T + ((size_t)t * C + clo) * L;
        __syncthreads();                             // the previous pair's readers are done
        if (staged) {
            for (u32 e = threadIdx.x; e < nch * L; e += blockDim.x) {
                sk[e] = (double)ta[e];
                st[e] = (double)tb[e];
            }
        }
        __syncthreads();
        for (u32 ri = threadIdx.x; ri < R; ri += blockDim.x) {
            const int r = (int)ri - (int)(L - 1);
            float *q = qs + (size_t)ri * (L + 1);
            double acc = 0.0;
            q[0] = 0.0f;
            for (u32 m = 0; m < L; m++) {
                const int mt = (int)m + r;
                if (mt >= 0 && mt < (int)L) {
                    if (staged) {
                        for (u32 c = 0; c < nch; c++) acc += sk[c * L + m] * st[c * L + mt];
                    } else {
                        for (u32 c = 0; c < nch; c++)
                            acc += (double)__ldg(ta + (size_t)c * L + m) * (double)__ldg(tb + (size_t)c * L + mt);
                    }
                }
                q[m + 1] = (float)acc;
            }
        }
        __syncthreads();
        float pm = -INFINITY;
        for (u32 ri = warp; ri < NR; ri += nwarp) {
            const int r = (int)ri - (int)L;
            float m = -INFINITY;
            for (u32 a = lane; a < S; a += 32) {
                const float X = ov_x(qs, L, (int)a - (int)nmax, r);
                m = fmaxf(m, -X + kx * fabsf(X));
            }
            m = warp_max_f(m);
            m += kPruneSlack * fabsf(m);
            if (lane == 0) XMr[(size_t)pair * NR + ri] = m;
            pm = fmaxf(pm, m);
        }
        if (lane == 0) red[warp] = pm;
        __syncthreads();
        for (u32 i = threadIdx.x; XMw && i < 2 * L + 32; i += blockDim.x) {
            float m = -INFINITY;                     // XMr index of lag r: r + L
            for (int q = max(0, (int)i - 31); q <= min((int)i, (int)(NR - 1)); q++) m = fmaxf(m, XMr[(size_t)pair * NR + q]);
            XMw[(size_t)pair * (2 * L + 32) + i] = m;
        }
        float *qg = Q + (size_t)pair * R * (L + 1);
        for (u32 e = threadIdx.x; e < R * (L + 1); e += blockDim.x) qg[e] = qs[e];
        __syncthreads();
        if (threadIdx.x == 0) {
            float v = red[0];
            for (u32 w = 1; w < nwarp; w++) v = fmaxf(v, red[w]);
            XM[pair] = v;
        }
    }
}

// Warp argmax: larger value, then lower index.
__device__ __forceinline__ void warp_argmax(float &v, u32 &i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const u32 oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
    }
}

// Rows a of each candidate (one block per candidate): G(a) = H[k0][a] in
// FP32, the intervals, the L[k0][afix] > 0 bits, the largest in-bounds upper
// bound and |upper bound|, and the row of largest lower bound (a1), for the
// seed and the scan.  Every item of a candidate carries the error of its row
// a, and the best template's rows have the largest: from the 16-bit tables it
// was several times the reference's own rounding, and items whose second
// template is nearly clipped away (b near the ends) could not be told apart
// -- 566 contenders per candidate on 17 channels with 23 templates.  Warps
// take the template's channels in turn; a lane holds 8 consecutive shifts and
// 8 lags of the window at a time, so 64 FMAs take four 16-byte shared reads.
// Channels are summed apart and then together: the rounding is that of
// L + channels terms.
constexpr int kRowsThreads = 128, kRowsWarps = kRowsThreads / 32;
constexpr u32 kRowsShifts = 256;                 // shifts of a block's pass (8 per lane)
__host__ __device__ inline u32 rows_warp_floats(u32 L) {
    const u32 Lp = (L + 7) & ~7u;
    return kRowsShifts + Lp + 8 + Lp;            // window strip, template row
}
__host__ __device__ inline size_t rows_smem_bytes(u32 L) {
    return (size_t)kRowsWarps * (rows_warp_floats(L) + kRowsShifts) * 4;
}
__global__ void __launch_bounds__(kRowsThreads)
k_ov_rows(OvArgs A) {
    extern __shared__ __align__(16) float rsm_rows[];
    __shared__ float red_v[kRowsWarps], red_m[kRowsWarps], red_abs[kRowsWarps];
    __shared__ u32 red_i[kRowsWarps];
    const u32 nc = *A.n_cand;
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 S = A.S, n = A.n, nmax = A.nmax, L = A.L, Lp = (L + 7) & ~7u, NB = (S + 31) / 32;
    float *strip = rsm_rows + (size_t)warp * rows_warp_floats(L), *trow = strip + kRowsShifts + Lp + 8;
    float *part = rsm_rows + (size_t)kRowsWarps * rows_warp_floats(L);   // [warp][kRowsShifts]
    const float ka = A.oc->kappa_ref + A.oc->kappa_rows;
    for (u32 g = blockIdx.x; g < nc; g += gridDim.x) {
        if (A.cskip[g]) continue;
        const OvCand c = ov_cand(A, g);
        float vn, l1;
        ov_window_norms(A, g, c.bidx, c.k0, vn, l1);
        const u32 clo = A.tsup ? A.tsup[2 * c.k0] : 0u, chi = A.tsup ? A.tsup[2 * c.k0 + 1] : A.C;
        float va = -INFINITY, mA = -INFINITY, mabs = 0.0f;
        u32 a1 = 0;
        for (u32 x0 = 0; x0 < S; x0 += kRowsShifts) {
            float tot[8];
#pragma unroll
            for (int i = 0; i < 8; i++) tot[i] = 0.0f;
            __syncwarp();
            for (u32 x = lane; x < kRowsShifts + Lp + 8; x += 32) strip[x] = 0.0f;
            for (u32 ch = clo + warp; ch < chi; ch += kRowsWarps) {
                __syncwarp();
                // strip[x]: the window at lag x0 + x - n_max (zero outside [0, L));
                // four loads of each row in flight
                const float *v = A.v + (size_t)ch * n + c.bidx, *tp = A.T + ((size_t)c.k0 * A.C + ch) * L;
                for (u32 m0 = lane; m0 < Lp; m0 += 128) {
                    float f[4], tv[4];
#pragma unroll
                    for (u32 i = 0; i < 4; i++) {
                        const u32 m = min(m0 + 32 * i, L - 1);
                        f[i] = __ldg(v + m);
                        tv[i] = __ldg(tp + m);
                    }
#pragma unroll
                    for (u32 i = 0; i < 4; i++) {
                        const u32 m = m0 + 32 * i, x = m + nmax - x0;
                        if (m < L && x < kRowsShifts + Lp + 8) strip[x] = f[i];
                        if (m < Lp) trow[m] = m < L ? tv[i] : 0.0f;
                    }
                }
                __syncwarp();
                float acc[8], w[16];
#pragma unroll
                for (int i = 0; i < 8; i++) acc[i] = 0.0f;
                if (x0 + 8 * lane < S) {
                    const float *sp = strip + 8 * lane;
                    *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(sp);
                    *reinterpret_cast<float4 *>(w + 4) = *reinterpret_cast<const float4 *>(sp + 4);
                    for (u32 m = 0; m < Lp; m += 8) {
                        float t[8];
                        *reinterpret_cast<float4 *>(w + 8) = *reinterpret_cast<const float4 *>(sp + m + 8);
                        *reinterpret_cast<float4 *>(w + 12) = *reinterpret_cast<const float4 *>(sp + m + 12);
                        *reinterpret_cast<float4 *>(t) = *reinterpret_cast<const float4 *>(trow + m);
                        *reinterpret_cast<float4 *>(t + 4) = *reinterpret_cast<const float4 *>(trow + m + 4);
#pragma unroll
                        for (int mm = 0; mm < 8; mm++)
#pragma unroll
                            for (int i = 0; i < 8; i++) acc[i] = fmaf(t[mm], w[i + mm], acc[i]);
#pragma unroll
                        for (int i = 0; i < 8; i++) w[i] = w[i + 8];
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; i++) tot[i] += acc[i];
            }
            __syncthreads();                         // the previous shifts' readers of part are done
#pragma unroll
            for (int i = 0; i < 8; i++) part[warp * kRowsShifts + 8 * lane + i] = tot[i];
            __syncthreads();
            for (u32 y = 32 * warp; y < kRowsShifts && x0 + y < S; y += kRowsThreads) {
                const u32 x = x0 + y + lane;
                bool ap = false;
                if (x < S) {
                    float h = 0.0f;
#pragma unroll
                    for (int w8 = 0; w8 < kRowsWarps; w8++) h += part[w8 * kRowsShifts + y + lane];
                    const float nt = A.NT[(size_t)c.k0 * S + x], snt = A.sNT[(size_t)c.k0 * S + x];
                    h -= 0.5f * nt;
                    const float e = ka * (snt * vn + nt) + 4.0f * kUnitRoundoff * fabsf(h);
                    const float lo = h - e, hi = h + e;
                    A.ga_lo[(size_t)g * S + x] = lo;
                    A.ga_hi[(size_t)g * S + x] = hi;
                    if (x >= c.xlo && x < c.xhi_ex) {
                        ap = !(A.Lk[(size_t)c.k0 * n + c.bidx + x - nmax] <= 0.0f);
                        if (lo > va) { va = lo; a1 = x; }
                        mA = fmaxf(mA, hi);
                        mabs = fmaxf(mabs, fabsf(hi));
                    }
                }
                const u32 m = __ballot_sync(0xffffffffu, ap);
                if (lane == 0) A.ga_bits[(size_t)g * NB + (x0 + y) / 32] = m;
            }
        }
        warp_argmax(va, a1);
        mA = warp_max_f(mA);
        mabs = warp_max_f(mabs);
        if (lane == 0) { red_v[warp] = va; red_i[warp] = a1; red_m[warp] = mA; red_abs[warp] = mabs; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w8 = 1; w8 < kRowsWarps; w8++) {
                if (red_v[w8] > va || (red_v[w8] == va && red_i[w8] < a1)) { va = red_v[w8]; a1 = red_i[w8]; }
                mA = fmaxf(mA, red_m[w8]);
                mabs = fmaxf(mabs, red_abs[w8]);
            }
            A.ga_max[g] = mA;
            A.ga_abs[g] = mabs;
            A.seed_a1[g] = a1;
        }
        __syncthreads();                             // red_* are read before the next candidate writes them
    }
}

// Seed of each candidate's best lower bound, one warp per (candidate,
// template t): the items (a1, b1), (a1, b2), (a3, b1) with b1 the row b of
// largest lower bound, b2 the best row b within L of a1 and a3 the best row a
// within L of b1.  Any item's lower bound is a valid lower bound of the best
// item, and these are close to the largest one, so the scan can prune
// against it from the start.
__global__ void __launch_bounds__(kSeedThreads)
k_ov_seed(OvArgs A) {
    const u32 nc = *A.n_cand;
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 S = A.S, K = A.K, L = A.L, nmax = A.nmax, n = A.n, R = 2 * L - 1, NB = (S + 31) / 32;
    const float krm = ov_krm(A), kx = ov_kx(A);
    const u64 total = (u64)nc * K;
    const u64 nwarps = (u64)gridDim.x * (kSeedThreads / 32);
    for (u64 e = (u64)blockIdx.x * (kSeedThreads / 32) + warp; e < total; e += nwarps) {
        const u32 g = (u32)(e / K), t = (u32)(e % K);
        if (A.cskip[g] || A.ga_max[g] == -INFINITY) continue;   // skipped, or no in-bounds row
        const OvCand c = ov_cand(A, g);
        const u32 a1 = A.seed_a1[g];
        const float *ga_lo = A.ga_lo + (size_t)g * S;
        const float va = ga_lo[a1];
        const float *Hg = A.H + ((size_t)g * K + t) * S;
        const OvRowB rb = ov_row_b(A, g, c.bidx, c.k0, t, krm);
        const u32 xend = min(S, c.xhi_ex);
        float v1 = -INFINITY, v2 = -INFINITY, mB = -INFINITY, mabs = 0.0f;
        u32 b1 = 0, b2 = 0;
        for (u32 x = c.xlo + lane; x < xend; x += 32) {
            float lo, hi;
            ov_row_interval(A, g, t, x, Hg[x], A.sNT[(size_t)t * S + x], rb, lo, hi);
            if (lo > v1) { v1 = lo; b1 = x; }
            if ((x > a1 ? x - a1 : a1 - x) <= L && lo > v2) { v2 = lo; b2 = x; }
            mB = fmaxf(mB, hi);
            mabs = fmaxf(mabs, fabsf(hi));
        }
        warp_argmax(v1, b1);
        warp_argmax(v2, b2);
        mB = warp_max_f(mB);
        mabs = warp_max_f(mabs);
        if (lane == 0) {                                 // the scan's pair test, before its row pass
            A.pair_mb[e] = mB;
            A.pair_mabs[e] = mabs;
        }
        float v3 = -INFINITY;
        u32 a3 = 0;
        for (u32 x = c.xlo + lane; x < xend; x += 32)
            if ((x > b1 ? x - b1 : b1 - x) <= L && ga_lo[x] > v3) { v3 = ga_lo[x]; a3 = x; }
        warp_argmax(v3, a3);
        float seed = 0.0f;
        if (lane < 3) {
            const u32 a = lane == 2 ? a3 : a1, b = lane == 1 ? b2 : b1;
            const float lb_b = lane == 1 ? v2 : v1;
            const float lb_a = lane == 2 ? v3 : va;
            if ((a > b ? a - b : b - a) <= L && lb_a > -INFINITY && lb_b > -INFINITY) {
                const bool fp = (A.ga_bits[(size_t)g * NB + (a >> 5)] >> (a & 31)) & 1u;
                const bool sp = !(A.Lk[(size_t)t * n + c.bidx + b - nmax] <= 0.0f);
                if (fp || sp) {                          // .cl:572-576
                    const float *q = A.Q + ((size_t)c.k0 * K + t) * R * (L + 1);
                    const float X = ov_disjoint(A.tsup, c.k0, t) ? 0.0f
                                                                 : ov_x(q, L, (int)a - (int)nmax, (int)a - (int)b);
                    seed = lb_a + lb_b - X - kx * fabsf(X);
                }
            }
        }
        seed = warp_max_f(seed);
        if (lane == 0 && seed > 0.0f) atomicMax(reinterpret_cast<int *>(A.cand_lb) + g, __float_as_int(seed));
    }
}

// One warp per (candidate, template t): every item (a, b, t) the reference
// evaluates (.cl:534-576) either gets its interval here or is shown to have
// hi < TH, TH = max(best lower bound so far, current best likelihood):
//   - the whole pair is skipped when max hiA + max hiB + XM < TH;
//   - a row a against a block of 32 rows b is skipped when
//     hiA + max hiB of the block + XMw of its lags < TH (lanes over the rows a);
//   - of a row and a block that remain, lanes over the rows b, the items that
//     pass the skip rules and hiA + hiB + XMr[a-b] >= TH are queued, and 32 of
//     them at a time, one per lane, get their interval from the prefix table.
// An item that is never enumerated can neither be the best item (whose value
// is >= every lower bound) nor beat the current best.  Items with
// hi >= TH and hi > current best go to the contender pool with their hi;
// their lower bounds raise the candidate's best lower bound, and TH with it
// (the block of largest upper bound goes first).  Testing rows against blocks
// leaves about 50 warp steps of a pair with 201 shifts; lists of single rows
// a and b were crossed pair by pair, up to 1,250 steps.  What is left is bound
// by latency, so everything a pair needs is loaded before it is used and kept
// in shared memory.
__global__ void __launch_bounds__(kScanThreads, 4)
k_ov_scan(OvArgs A) {
    extern __shared__ float sm[];
    const u32 S = A.S, K = A.K, L = A.L, nmax = A.nmax, n = A.n;
    const u32 R = 2 * L - 1, NR = 2 * L + 1, NW = 2 * L + 32, NB = (S + 31) / 32;
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *hb_lo = (float *)((char *)sm + (size_t)warp * sweep_warp_bytes(S, L)), *hb_hi = hb_lo + S;
    u32 *bbits = (u32 *)(hb_hi + S), *abits = bbits + NB;
    float *bmax = (float *)(abits + NB);             // largest in-bounds upper bound of each block of rows b
    float *ua = bmax + NB, *xw = ua + 32 * NB;       // rows a; lag bounds: block distance (ka - kb + NB - 1), lane
    float *xr = xw + 64 * NB;                        // the pair's lag bounds, slack added
    u32 *queue = (u32 *)(xr + NR);                   // items a | b << 16 that passed every bound
    const u32 nc = *A.n_cand;
    const u64 total = (u64)nc * K;
    // a warp's share of a small pass is spread over two turns at least
    const u32 per = (u32)max(1ull, min(32ull, total / ((u64)gridDim.x * (kScanThreads / 32) * 2)));
    const float krm = ov_krm(A), kx = ov_kx(A);
    u32 evaluated = 0;
    for (;;) {
        // pairs are taken dynamically, up to 32 at a time: their cost varies by
        // orders of magnitude, and most fail the pair test (lanes over pairs)
        u64 e32 = 0;
        if (lane == 0) e32 = atomicAdd(A.scan_next, (unsigned long long)per);
        e32 = __shfl_sync(0xffffffffu, e32, 0);
        if (e32 >= total) break;
        // the pair test with the seed's row maxima: a pair that fails it needs no row pass
        bool go = false;
        if (lane < per && e32 + lane < total) {
            const u64 e = e32 + lane;
            const u32 g = (u32)(e / K), t = (u32)(e - (u64)g * K);
            const float mA = A.cskip[g] ? -INFINITY : A.ga_max[g];
            if (mA != -INFINITY) {                   // else skipped, or no in-bounds row
                const u32 id = A.cand[g], k0 = A.best_lab[id];
                const float TH = fmaxf(*(volatile const float *)(A.cand_lb + g), A.best_ll[id]);
                const float XM = A.XM[(size_t)k0 * K + t];
                // without the stored magnitude, a bound: |H| + its error is below 1.02 (||t|| ||window|| + ||t||^2)
                float mabs;
                if (A.pair_mabs) {
                    mabs = A.pair_mabs[e];
                } else {
                    const OvRowB rb = ov_row_b(A, g, A.best_idx[id], k0, t, krm);
                    mabs = 1.02f * A.tnorm[t] * (rb.vn + A.tnorm[t]) + rb.eqt + rb.sub1;
                }
                const float slack = kPruneSlack * (2.0f * fmaxf(A.ga_abs[g], mabs) + fabsf(TH) + fabsf(XM));
                go = mA + A.pair_mb[e] + XM + slack >= TH;
            }
        }
        u32 todo = __ballot_sync(0xffffffffu, go);
        while (todo) {
            const u64 e = e32 + (u32)(__ffs(todo) - 1);
            todo &= todo - 1;
            const u32 g = (u32)(e / K), t = (u32)(e - (u64)g * K);
            const OvCand c = ov_cand(A, g);
            const float mA = A.ga_max[g];
            float TH = fmaxf(*(volatile const float *)(A.cand_lb + g), c.lbest);
            const size_t pair = (size_t)c.k0 * K + t;
            const float XM = A.XM[pair];
            const OvRowB rb = ov_row_b(A, g, c.bidx, c.k0, t, krm);
            const float *Hg = A.H + ((size_t)g * K + t) * S;
            const float *ga_lo = A.ga_lo + (size_t)g * S, *ga_hi = A.ga_hi + (size_t)g * S;
            // rows b: intervals and the L[t][ashift] > 0 bits
            float mB = -INFINITY, mabs = A.ga_abs[g];
            u32 kbest = 0;
            __syncwarp();                            // the previous pair's readers are done
            // (every load of 256 rows before their arithmetic)
            for (u32 x1 = 0; x1 < S; x1 += 256) {
                float hv[8], nt[8], lk[8];
#pragma unroll
                for (u32 i = 0; i < 8; i++) {
                    const u32 x = min(x1 + 32 * i + lane, S - 1);
                    hv[i] = __ldg(Hg + x);
                    nt[i] = __ldg(A.sNT + (size_t)t * S + x);
                    // in-bounds rows only: the others' positions lie outside the recording
                    lk[i] = A.Lk[(size_t)t * n + c.bidx + max(c.xlo, min(x, c.xhi_ex - 1)) - nmax];
                }
#pragma unroll
                for (u32 i = 0; i < 8; i++) {
                    const u32 x = x1 + 32 * i + lane;
                    if (x1 + 32 * i >= S) break;     // uniform in the warp
                    bool bp = false;
                    float up = -INFINITY;
                    if (x < S) {
                        float lo, hi;
                        ov_row_interval(A, g, t, x, hv[i], nt[i], rb, lo, hi);
                        hb_lo[x] = lo;
                        hb_hi[x] = hi;
                        if (x >= c.xlo && x < c.xhi_ex) {
                            bp = !(lk[i] <= 0.0f);
                            up = hi;
                            mabs = fmaxf(mabs, fabsf(hi));
                        }
                    }
                    const u32 mb = __ballot_sync(0xffffffffu, bp);
                    up = warp_max_f(up);
                    if (lane == 0) { bbits[x1 / 32 + i] = mb; bmax[x1 / 32 + i] = up; }
                    if (up > mB) { mB = up; kbest = x1 / 32 + i; }
                }
            }
            mabs = warp_max_f(mabs);
            __syncwarp();
            float slack = kPruneSlack * (2.0f * mabs + fabsf(TH) + fabsf(XM));
            if (!(mA + mB + XM + slack >= TH)) continue;
            const bool apart = ov_disjoint(A.tsup, c.k0, t);   // no cross term, no table
            const float *xmr = A.XMr + pair * NR, *xmw = A.XMw ? A.XMw + pair * NW : nullptr;
            // rows a (out of bounds: below everything), and for every distance of
            // blocks the bound of the lags of a row a against 32 rows b: XMw at
            // a - 32 k + L (no lag there: below everything)
            for (u32 x = lane; x < NB; x += 32) abits[x] = A.ga_bits[(size_t)g * NB + x];
            for (u32 x0 = lane; x0 < NR; x0 += 256) {
                float y[8];
#pragma unroll
                for (u32 i = 0; i < 8; i++) y[i] = apart ? 0.0f : __ldg(xmr + min(x0 + 32 * i, NR - 1));
#pragma unroll
                for (u32 i = 0; i < 8; i++)
                    if (x0 + 32 * i < NR) xr[x0 + 32 * i] = y[i] + kPruneSlack * fabsf(y[i]);
            }
            for (u32 k = 0; k < NB; k += 4) {
                float u[4], y[8];
#pragma unroll
                for (u32 i = 0; i < 4; i++) u[i] = __ldg(ga_hi + min(32 * (k + i) + lane, S - 1));
#pragma unroll
                for (u32 i = 0; i < 8; i++) {
                    const int wi = 32 * ((int)(2 * k + i) - (int)(NB - 1)) + (int)lane + (int)L;
                    y[i] = apart ? 0.0f : !A.XMw ? XM : __ldg(xmw + max(0, min((int)NW - 1, wi)));
                    if (wi < 0 || wi >= (int)NW) y[i] = -INFINITY;
                }
#pragma unroll
                for (u32 i = 0; i < 4; i++) {
                    const u32 a = 32 * (k + i) + lane;
                    if (k + i < NB) ua[a] = a < S && a >= c.xlo && a < c.xhi_ex ? u[i] : -INFINITY;
                }
#pragma unroll
                for (u32 i = 0; i < 8; i++)
                    if (2 * k + i < 2 * NB - 1)
                        xw[32 * (2 * k + i) + lane] = y[i] > -INFINITY ? y[i] + kPruneSlack * fabsf(y[i]) : y[i];
            }
            __syncwarp();
            const float *q = A.Q + pair * R * (L + 1);
            u32 held = 0;                            // items in the queue
            // intervals of the first min(held, 32) queued items, one per lane
            auto drain = [&]() {
                __syncwarp();
                const bool valid = lane < held;
                const u32 it = valid ? queue[lane] : 0u, a = it & 0xffffu, b = it >> 16;
                float hi = -INFINITY, lo = -INFINITY;
                if (valid) {
                    const float la = __ldg(ga_lo + a);
                    const float X = apart ? 0.0f : ov_x(q, L, (int)a - (int)nmax, (int)a - (int)b);
                    const float ex = kx * fabsf(X);
                    hi = ua[a] + hb_hi[b] - X + ex;
                    lo = la + hb_lo[b] - X - ex;
                    evaluated++;
                }
                const bool keep = valid && hi >= TH && hi > c.lbest;
                const u32 mk = __ballot_sync(0xffffffffu, keep);
                if (mk) {
                    u32 base = 0;
                    if (lane == 0) base = atomicAdd(A.pool_total, (u32)__popc(mk));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (keep) {
                        const u32 pp = base + __popc(mk & ((1u << lane) - 1u));
                        if (pp < A.pool_cap) {
                            A.pool_slot[pp] = g;
                            A.pool_item[pp] = t + K * (a + S * b);
                            A.pool_hi[pp] = hi;
                        } else {
                            A.fallback[g] = 1;
                        }
                    }
                }
                lo = warp_max_f(lo);
                if (lo > TH) {
                    if (lane == 0) atomicMax(reinterpret_cast<int *>(A.cand_lb) + g, __float_as_int(lo));   // > 0
                    TH = lo;
                    slack = kPruneSlack * (2.0f * mabs + fabsf(TH) + fabsf(XM));
                }
                const u32 rest = held > 32 && lane < held - 32 ? queue[32 + lane] : 0u;
                __syncwarp();
                if (held > 32 && lane < held - 32) queue[lane] = rest;
                held = held > 32 ? held - 32 : 0;
                __syncwarp();
            };
            for (u32 kk = 0; kk < NB; kk++) {
                const u32 k = kk == 0 ? kbest : kk <= kbest ? kk - 1 : kk;   // kbest, then the others in order
                const float mBk = bmax[k];
                if (!(mA + mBk + XM + slack >= TH)) continue;                // uniform
                const u32 b = 32 * k + lane;
                const bool inb = b < S && b >= c.xlo && b < c.xhi_ex;
                const float hi_b = b < S ? hb_hi[b] : 0.0f;
                const bool bp = (bbits[k] >> lane) & 1u;
                for (u32 a0 = 0; a0 < S; a0 += 32) {
                    const float xb = xw[a0 + 32 * (NB - 1 - k) + lane], ub = ua[a0 + lane];
                    const bool ka = xb > -INFINITY && ub > -INFINITY && ub + mBk + xb + slack >= TH;
                    u32 rows = __ballot_sync(0xffffffffu, ka);
                    const u32 ap = abits[a0 / 32];
                    while (rows) {
                        const u32 r = __ffs(rows) - 1, a = a0 + r;
                        rows &= rows - 1;
                        const bool valid = inb && (a > b ? a - b : b - a) <= L &&        // .cl:543-556
                                           (bp || ((ap >> r) & 1u)) &&                   // .cl:572-576
                                           ua[a] + hi_b + xr[(int)a - (int)b + (int)L] + slack >= TH;
                        const u32 m = __ballot_sync(0xffffffffu, valid);
                        if (m == 0) continue;
                        if (valid) queue[held + __popc(m & ((1u << lane) - 1u))] = a | (b << 16);
                        held += __popc(m);
                        if (held >= 32) drain();
                    }
                }
            }
            if (held) drain();
        }
    }
    if (A.items_evaluated) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) evaluated += __shfl_xor_sync(0xffffffffu, evaluated, o);
        if (lane == 0 && evaluated) atomicAdd(A.items_evaluated, (u64)evaluated);
    }
}

// Order-preserving key: larger value first, then lower item id.
__device__ __forceinline__ u64 ov_pack(float v, u32 item) {
    u32 u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((u64)u << 32) | (u64)(0xffffffffu - item);
}
__device__ __forceinline__ float ov_unpack_value(u64 key) {
    u32 u = (u32)(key >> 32);
    u = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(u);
}

// Exact value of one item (overlap_recheck_indices, .cl:583-646), in the
// reference's order of operations; loads are issued eight lags at a time so
// the two sequential sums do not wait on each one.
__device__ float overlap_item_exact_global(const OvArgs &A, u32 lab, u32 bidx, u32 t, u32 a, u32 b) {
    const u32 L = A.L, C = A.C;
    const u32 afix = bidx + a - A.nmax, ashift = bidx + b - A.nmax;
    const int fa = (int)bidx - (int)afix, sa = (int)bidx - (int)ashift;
    // channels where either template is non-zero, in channel order: the two
    // supports as one range when they meet, else one after the other
    // (elsewhere both terms are 0 and the reference's sums do not change)
    u32 r0 = 0, r1 = C, r2 = C, r3 = C;
    if (A.tsup) {
        u32 al = A.tsup[2 * lab], ah = A.tsup[2 * lab + 1], bl = A.tsup[2 * t], bh = A.tsup[2 * t + 1];
        if (ah <= al) { al = bl; ah = bh; }
        if (bh <= bl) { bl = al; bh = ah; }
        if (bl < al) { u32 x = al; al = bl; bl = x; x = ah; ah = bh; bh = x; }
        if (bl <= ah) { r0 = al; r1 = max(ah, bh); r2 = r3 = r1; }
        else { r0 = al; r1 = ah; r2 = bl; r3 = bh; }
    }
    float cml = 0.0f;
    for (u32 c = r0; c < r3; c = (c + 1 == r1) ? r2 : c + 1) {
        const float *f = A.T + ((size_t)lab * C + c) * L;
        const float *sp = A.T + ((size_t)t * C + c) * L;
        const float *vv = A.v + (size_t)c * A.n + bidx;
        float ss = 0.0f;
        for (u32 j0 = 0; j0 < L; j0 += 8) {
            float fv[8], sv[8], wv[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int j = (int)j0 + i;
                const int jf = fa + j, js = sa + j;
                fv[i] = (j < (int)L && jf >= 0 && jf < (int)L) ? __ldg(f + jf) : 0.0f;
                sv[i] = (j < (int)L && js >= 0 && js < (int)L) ? __ldg(sp + js) : 0.0f;
                wv[i] = j < (int)L ? __ldg(vv + j) : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (j0 + i < L) {
                    const float sum = __fadd_rn(fv[i], sv[i]);
                    ss = __fadd_rn(ss, __fmul_rn(sum, sum));
                    cml = __fadd_rn(cml, __fmul_rn(sum, wv[i]));
                }
            }
        }
        if ((double)ss > 0.0) cml = __double2float_rn(__dsub_rn((double)cml, __dmul_rn(0.5, (double)ss)));
    }
    return cml;
}

constexpr int kRefineThreads = 256;
constexpr u32 kRefRows = 16;             // product rows (chunks of 32 lags) a warp stages at once
constexpr u32 kRefWarpMax = 24576;       // pool entries up to which a warp shares the terms of its contenders
constexpr u32 kRefStride = 33;           // row stride: lanes walk 32 rows without bank conflicts
struct RefItem {                         // one contender, in shared memory
    u32 lab, t, bidx, r0, n1, r2, nch, e;
    int fa, sa;
};
__host__ __device__ inline size_t ov_refine_smem_bytes() {
    return (size_t)(kRefineThreads / 32) * (2 * kRefRows * kRefStride * 4 + kRefRows * sizeof(RefItem)) +
           kRefineThreads * 4;
}

// Exact values of the pooled contenders whose upper bound reaches their
// candidate's final lower bound (overlap_recheck_indices, .cl:583-646), each
// by the reference's own sequence of operations; each candidate keeps the
// largest value above its current best, lowest item id on ties (the parse
// kernel's strict-greater scan over single-item groups, .cl:699-706).
//
// An item is two float chains (the likelihood and the channel's sum of
// squares) over channels x lags that must be added in order, of terms that
// are independent.  With many contenders one thread each hides its loads
// behind the others'.  With few (most passes: the last contenders of a
// recording take as many passes as the first) nothing hides them: 276 us a
// pass on the 384-channel probe however few contenders there were.  Up to
// kRefWarpMax pool entries a block therefore gathers the contenders still in
// question, and a warp takes up to 16 of them: its lanes form the terms of 32
// lags of one channel of one contender at a time (coalesced loads, each
// product rounded as in the reference) into a row of shared memory, then lane
// i adds contender i's rows in order; few contenders get several rows each, so
// that they wait for global memory once per eight rows (48 us a pass).  That
// costs 84 instructions per 32 terms against about 22 of a thread's: the line
// lies where both take about 250 us (17 channels x 77 lags).
__global__ void __launch_bounds__(kRefineThreads)
k_ov_refine(OvArgs A) {
    extern __shared__ float refsm[];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *pr = refsm + (size_t)warp * 2 * kRefRows * kRefStride;    // sum * voltage
    float *qr = pr + kRefRows * kRefStride;                          // sum * sum
    RefItem *items = (RefItem *)(refsm + (size_t)(kRefineThreads / 32) * 2 * kRefRows * kRefStride) + kRefRows * warp;
    const u32 L = A.L, C = A.C, K = A.K, S = A.S;
    const u32 m = min(*A.pool_total, A.pool_cap);
    if (m > kRefWarpMax) {
        for (u32 e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
            const u32 g = A.pool_slot[e];
            if (A.fallback[g] || A.pool_hi[e] < A.cand_lb[g]) continue;   // below another item's lower bound
            atomicAdd(A.refined, 1u);
            const u32 it = A.pool_item[e], id = A.cand[g];
            const float ll = overlap_item_exact_global(A, A.best_lab[id], A.best_idx[id], it % K, (it / K) % S,
                                                       it / (K * S));
            if (ll > A.best_ll[id]) atomicMax(&A.best_key[g], ov_pack(ll, it));
        }
        return;
    }
    u32 *list = (u32 *)((RefItem *)(refsm + (size_t)(kRefineThreads / 32) * 2 * kRefRows * kRefStride) +
                        kRefRows * (kRefineThreads / 32));
    __shared__ u32 cnt;
    const u32 part = (m + gridDim.x - 1) / gridDim.x;
    const u32 e0 = min(m, part * blockIdx.x), e1 = min(m, e0 + part);
    const u32 ncl = (L + 31) / 32;                   // rows of a channel
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    for (u32 eb = e0; eb < e1; eb += kRefineThreads) {
      const u32 e = eb + threadIdx.x;
      if (e < e1) {
          const u32 g = A.pool_slot[e];
          // the others lie below another item's lower bound
          if (!A.fallback[g] && !(A.pool_hi[e] < A.cand_lb[g])) list[atomicAdd(&cnt, 1u)] = e;
      }
      __syncthreads();
      const u32 held = cnt;                          // at most kRefineThreads
      if (threadIdx.x == 0 && held) atomicAdd(A.refined, held);
      const u32 per = min(kRefRows, max(1u, (held + kRefineThreads / 32 - 1) / (kRefineThreads / 32)));
      for (u32 base = warp * per; base < held; base += (kRefineThreads / 32) * per) {
        const u32 nact = min(per, held - base);
        const bool act = lane < nact;
        u32 nq = 0;                                  // this lane's contender: rows
        if (act) {
            RefItem it;
            it.e = list[base + lane];
            const u32 id = A.cand[A.pool_slot[it.e]], item = A.pool_item[it.e];
            it.lab = A.best_lab[id];
            it.bidx = A.best_idx[id];
            it.t = item % K;
            it.fa = (int)A.nmax - (int)((item / K) % S);
            it.sa = (int)A.nmax - (int)(item / (K * S));
            // channels where either template is non-zero, in channel order: the
            // two supports as one range when they meet, else one after the other
            // (elsewhere both terms are 0 and the reference's sums do not change)
            it.r0 = 0; it.n1 = C; it.r2 = C; it.nch = C;
            if (A.tsup) {
                u32 al = A.tsup[2 * it.lab], ah = A.tsup[2 * it.lab + 1], bl = A.tsup[2 * it.t], bh = A.tsup[2 * it.t + 1];
                if (ah <= al) { al = bl; ah = bh; }
                if (bh <= bl) { bl = al; bh = ah; }
                if (bl < al) { u32 x = al; al = bl; bl = x; x = ah; ah = bh; bh = x; }
                it.r0 = al;
                if (bl <= ah) { it.n1 = max(ah, bh) - al; it.r2 = al + it.n1; it.nch = it.n1; }
                else { it.n1 = ah - al; it.r2 = bl; it.nch = it.n1 + (bh - bl); }
            }
            nq = it.nch * ncl;
            items[lane] = it;
        }
        u32 nqmax = nq;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nqmax = max(nqmax, __shfl_xor_sync(0xffffffffu, nqmax, o));
        __syncwarp();
        const u32 sh = nact <= 2 ? 3u : nact <= 4 ? 2u : nact <= 8 ? 1u : 0u;   // log2(rows of a contender per stage)
        const u32 nrows = nact << sh;
        float cml = 0.0f, ss = 0.0f;
        for (u32 q0 = 0; q0 < nqmax; q0 += 1u << sh) {
            const u32 my_ci = (q0 + (lane & 7u)) / ncl;              // channel and chunk of row q0 + (lane & 7)
            const u32 my_lc = (q0 + (lane & 7u)) - my_ci * ncl;
            for (u32 rb = 0; rb < nrows; rb += 8) {
                float fv[8], sv[8], wv[8];
#pragma unroll
                for (u32 u = 0; u < 8; u++) {
                    const u32 r = rb + u, k = r & ((1u << sh) - 1u);
                    const u32 ci = __shfl_sync(0xffffffffu, my_ci, k), j = __shfl_sync(0xffffffffu, my_lc, k) * 32 + lane;
                    fv[u] = sv[u] = wv[u] = 0.0f;
                    const RefItem &it = items[min(r >> sh, nact - 1)];
                    if (r < nrows && ci < it.nch && j < L) {
                        const u32 c = ci < it.n1 ? it.r0 + ci : it.r2 + (ci - it.n1);
                        const int jf = it.fa + (int)j, js = it.sa + (int)j;
                        if (jf >= 0 && jf < (int)L) fv[u] = __ldg(A.T + ((size_t)it.lab * C + c) * L + jf);
                        if (js >= 0 && js < (int)L) sv[u] = __ldg(A.T + ((size_t)it.t * C + c) * L + js);
                        wv[u] = __ldg(A.v + (size_t)c * A.n + it.bidx + j);
                    }
                }
#pragma unroll
                for (u32 u = 0; u < 8; u++) {
                    if (rb + u >= nrows) break;      // uniform in the warp
                    const float sum = __fadd_rn(fv[u], sv[u]);
                    pr[(rb + u) * kRefStride + lane] = __fmul_rn(sum, wv[u]);
                    qr[(rb + u) * kRefStride + lane] = __fmul_rn(sum, sum);
                }
            }
            __syncwarp();
            for (u32 k = 0; k < (1u << sh); k++) {
                const u32 lc = __shfl_sync(0xffffffffu, my_lc, k);
                if (q0 + k < nq) {
                    const float *p = pr + ((lane << sh) + k) * kRefStride, *q = qr + ((lane << sh) + k) * kRefStride;
                    const u32 cnt = min(32u, L - lc * 32);
                    u32 j = 0;
                    for (; j + 8 <= cnt; j += 8) {
#pragma unroll
                        for (u32 x = 0; x < 8; x++) {
                            ss = __fadd_rn(ss, q[j + x]);
                            cml = __fadd_rn(cml, p[j + x]);
                        }
                    }
                    for (; j < cnt; j++) {
                        ss = __fadd_rn(ss, q[j]);
                        cml = __fadd_rn(cml, p[j]);
                    }
                    if (lc == ncl - 1) {             // the channel's last lag (.cl:627-630)
                        if ((double)ss > 0.0) cml = __double2float_rn(__dsub_rn((double)cml, __dmul_rn(0.5, (double)ss)));
                        ss = 0.0f;
                    }
                }
            }
            __syncwarp();
        }
        if (lane < nact) {
            const u32 pe = items[lane].e, pg = A.pool_slot[pe];
            if (cml > A.best_ll[A.cand[pg]]) atomicMax(&A.best_key[pg], ov_pack(cml, A.pool_item[pe]));
        }
        __syncwarp();
      }
      __syncthreads();
      if (threadIdx.x == 0) cnt = 0;
      __syncthreads();
    }
}

// One warp per candidate slot: the parse decision (.cl:707-814) for the
// winning contender, or "no improvement".
__global__ void __launch_bounds__(kRefineThreads)
k_ov_finalize(OvArgs A) {
    __shared__ float fbuf[kRefineThreads / 32][kWarpChunk];
    const u32 lane = threadIdx.x & 31;
    float *buf = fbuf[threadIdx.x >> 5];
    const u32 nc = *A.n_cand;
    const u32 nwarps = gridDim.x * (blockDim.x >> 5);
    for (u32 g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < nc; g += nwarps) {
        if (A.fallback[g]) continue;
        const u32 id = A.cand[g];
        const u64 key = A.best_key[g];
        float bv = A.best_ll[id];
        u64 bi = 0;
        if (key != 0ull) {
            bv = ov_unpack_value(key);
            bi = 0xffffffffu - (u32)(key & 0xffffffffu);
        }
        if (bv <= A.best_ll[id] || bv <= 0.0f) {
            if (lane == 0) A.ovr[id] = 0;
            continue;
        }
        const u32 lab = A.best_lab[id], bidx = A.best_idx[id];
        const u32 t = (u32)(bi % A.K);
        const u32 a = (u32)((bi / A.K) % A.S);
        const u32 b = (u32)((bi / ((u64)A.S * A.K)) % A.S);
        const u32 afix = bidx + a - A.nmax, ashift = bidx + b - A.nmax;
        const float lf = warp_lk_exact(A.lazy, A.Lk, A.n, lab, afix, buf);
        const float ls = warp_lk_exact(A.lazy, A.Lk, A.n, t, ashift, buf);
        if (lane == 0)
            overlap_parse_tail(id, bv, lab, t, afix, ashift, lf, ls, A.best_idx, A.best_lab, A.best_ll, A.ov_idx,
                               A.ov_lab, A.ovr, A.thr);
    }
}

}  // namespace fbp
