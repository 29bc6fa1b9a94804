// The overlap recheck's per-candidate tables on the tensor cores, wide tiles:
//     H[g][t][b] = <t shifted by b - n_max, window of candidate g> - 0.5 * ||t clipped||^2
// for every template t and shift b < S, in the contraction of the wide-tile
// likelihood (fbp_lik_tcw.cuh): M = 128 = 16 templates x 8 sample shifts,
// N = blocks of 8 positions, K = 16 lags of one channel, the same packed
// template tiles.  The position axis holds `spt` candidates, one per slot of
// ST = 8 * ncol positions: the candidate's L samples stand at n_max.. of its
// slot, zeros elsewhere, so position b of a slot is shift b and no other
// candidate's sample is within its lags (ST >= max(2 n_max + 1, n_max + L)).
//
// Persistent, one CTA per SM, 16 warps.  An item is (tile of spt candidates,
// template group); consecutive items are the groups of one tile, so that
// concurrent CTAs read the same windows.  Producer warps take whole channels
// in turn, one warp per ring stage (at most 7): the channel's samples come by coalesced 4-byte loads (16
// in flight per lane, issued before the wait for a free ring stage), are
// scaled by their candidate's power of two and written as fp16 into the stage
// beside the template tiles, which one bulk copy brings.  No barrier joins the
// producers: a stage is complete when its warp has arrived and the copy has
// landed.  Epilogue warps (two per TMEM lane quadrant, alternate slots) store
// H and keep, per (candidate, template), the largest upper bound of an
// in-bounds row and the row of largest lower bound, which the search would
// otherwise read the table again for.
//
// Sixteen templates of a 384-channel probe span 34 channels; at five MMAs a
// channel the MMA time of a tile is 11,000 cycles, and 16 candidates share
// it.  The 128-sample tiles (k_lik_tc<1>: one candidate, 16 template columns
// behind every 4 KB operand) were bound by operand fetches.
// Every wait is bounded; a wait that gives up sets err and the abort flag.
#pragma once
#include "fbp_lik_tcw.cuh"
#include "fbp_overlap_fast.cuh"

namespace fbp {

// Sixteen warps (four to a scheduler, so that a thread may hold 128 registers).
constexpr int kOvtProdWarps = 7, kOvtMmaWarp = kOvtProdWarps, kOvtEpiWarp0 = 8, kOvtEpiWarps = 8;
constexpr int kOvtThreads = 512, kOvtProdThreads = 32 * kOvtProdWarps;
constexpr u32 kOvtLoads = 16;            // voltage loads of a producer lane in flight

// Slots of a tile: columns per slot, slots, MMA N, staged positions.
struct OvtPlan {
    u32 ncol, spt, N, px, ns;
    size_t stage, smem;
};
__host__ __device__ inline OvtPlan ovt_plan(u32 L, u32 nmax) {
    OvtPlan p{};
    const u32 need = 2 * nmax + 1 > nmax + L ? 2 * nmax + 1 : nmax + L;
    p.ncol = (need + 7) / 8;
    const u32 chunk = (p.ncol + 7) / 8 * 8;          // columns an epilogue warp reads of a slot
    if (chunk > kWN || L < kWMinL) return p;         // spt 0: does not apply
    p.spt = (kWN - chunk) / p.ncol + 1;
    if (p.spt > 32) p.spt = 32;
    p.N = ((p.spt - 1) * p.ncol + chunk + 15) / 16 * 16;
    if (p.N > kWN) p.N = kWN;
    p.px = 8 * p.N + 16 * tcw_nkc(L);
    p.stage = align_up((size_t)tcw_nkc(L) * kWATile + align_up((size_t)p.px * 2, 16), 128);
    const size_t tail = 1024;                        // barriers, fill counts, flags
    for (p.ns = kOvtProdWarps; p.ns >= 2; p.ns--)     // a stage for each producer warp at most
        if (p.ns * p.stage + tail <= 227 * 1024) break;
    if (p.ns < 2) p.spt = 0;
    p.smem = p.ns * p.stage + tail;
    return p;
}

struct OvtArgs {
    OvArgs o;
    const TcwArgs *groups;           // the likelihood's wide groups (channels, templates, packed tiles)
    u32 ngroups;
    u32 ncol, spt, N, ns, stage, px;
    u32 *err;
    u32 wait_polls;
};

__global__ void __launch_bounds__(kOvtThreads, 1)
k_ov_tcw(const __grid_constant__ OvtArgs P) {
    const OvArgs &A = P.o;
    const u32 nc = *A.n_cand;
    // with few candidates, fewer to a tile: every CTA gets an item
    const u32 G = P.ngroups, ns = P.ns;
    const u32 spt = (u32)min((u64)P.spt, max((u64)1, ((u64)nc * G + gridDim.x - 1) / gridDim.x));
    const u32 N = min(P.N, ((spt - 1) * P.ncol + (P.ncol + 7) / 8 * 8 + 15) / 16 * 16);
    const u64 nitems = (u64)((nc + spt - 1) / spt) * G;
    if ((u64)blockIdx.x >= nitems) return;           // no item for this CTA: no set-up at all
    extern __shared__ __align__(128) unsigned char osm[];
    const u32 L = A.L, nkc = tcw_nkc(L), n = A.n, nmax = A.nmax, S = A.S, K = A.K;
    const u32 a_bytes = nkc * kWATile;
    u64 *bars = (u64 *)(osm + (size_t)ns * P.stage);
    u32 *fills = (u32 *)(bars + 2 * ns + 5);         // [ns] copies issued into a stage
    u32 *tmem_slot = fills + ns, *abort_flag = tmem_slot + 1;
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const u32 wlim = P.wait_polls;
    auto bar_sfull = [&](u32 s) { return smem_u32(&bars[s]); };
    auto bar_sempty = [&](u32 s) { return smem_u32(&bars[ns + s]); };
    auto bar_afull = [&](u32 b) { return smem_u32(&bars[2 * ns + b]); };
    auto bar_aempty = [&](u32 b) { return smem_u32(&bars[2 * ns + 2 + b]); };
    const u32 bar_fin = smem_u32(&bars[2 * ns + 4]);
    if (tid == 0) {
        for (u32 s = 0; s < ns; s++) {
            mbar_init(bar_sfull(s), 1);
            mbar_init(bar_sempty(s), 1);
            fills[s] = 0;
        }
        for (u32 b = 0; b < 2; b++) {
            mbar_init(bar_afull(b), 1);
            mbar_init(bar_aempty(b), kOvtEpiWarps);
        }
        mbar_init(bar_fin, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(2 * kWN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // the position streams start as zeros; only the samples of the slots are
    // written later, always at the same places
    for (u32 s = 0; s < ns; s++) {
        uint4 *z = reinterpret_cast<uint4 *>(osm + (size_t)s * P.stage + a_bytes);
        for (u32 q = tid; q < (P.px * 2 + 15) / 16; q += blockDim.x) z[q] = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const u32 tmem = *tmem_slot;

    if (warp < kOvtProdWarps) {
        // =========================== producers ===========================
        const u32 ncl = (L + 31) / 32;               // loads of a slot's channel per lane
        u32 gs0 = 0;                                 // ring uses before this item
        bool stop = false;
        for (u64 item = blockIdx.x; item < nitems && !stop; item += gridDim.x) {
            const TcwArgs &T = P.groups[(u32)(item % G)];
            const u32 g = (u32)(item / G) * spt + lane;
            // lane k: candidate of slot k (a skipped one, or none, reads nothing)
            uint4 sl = make_uint4(0xffffffffu, 0u, 0u, 0u);
            if (lane < spt && g < nc) sl = A.slot_tab[g];
            const float scale = ldexpf(1.0f, (int)sl.y);     // exact: |kexp| <= 126
            const u32 start = sl.x != 0xffffffffu ? sl.x : 0u;       // n >= 4 L
            const u32 Cg = T.Cg, nq = spt * ncl;
            const float *v = T.v;
            const unsigned char *Aw = T.Aw;
            // stage s belongs to warp s: its uses are filled in order by one warp
            for (u32 c = warp < ns ? (warp + ns - gs0 % ns) % ns : Cg; c < Cg; c += ns) {
                const u32 s = warp, u = (gs0 + c) / ns;
                const float *vc = v + (size_t)c * n;
                unsigned char *stg = osm + (size_t)s * P.stage;
                u16 *B = reinterpret_cast<u16 *>(stg + a_bytes);
                for (u32 q0 = 0; q0 < nq; q0 += kOvtLoads) {
                    float f[kOvtLoads];
                    u32 k = q0 / ncl, jc = q0 - k * ncl;
#pragma unroll
                    for (u32 i = 0; i < kOvtLoads; i++) {
                        // unconditional, so that the loads do not wait for one another
                        // (a slot without a candidate reads samples whose outputs are dropped)
                        const u32 b0 = __shfl_sync(0xffffffffu, start, min(k, 31u));
                        f[i] = __ldg(vc + b0 + min(jc * 32 + lane, L - 1));
                        if (++jc == ncl) { jc = 0; k++; }
                    }
                    if (q0 == 0) {
                        bool ok = true;
                        if (lane == 0 && u > 0 && !mbar_wait_bounded(bar_sempty(s), (u - 1) & 1u, wlim)) {
                            atomicExch(P.err, 21u);
                            atomicExch(abort_flag, 1u);
                        }
                        __syncwarp();
                        ok = *(volatile u32 *)abort_flag == 0;
                        if (!__all_sync(0xffffffffu, ok)) { stop = true; break; }
                        if (lane == 0) {
                            fills[s] = u + 1;
                            mbar_expect_tx(bar_sfull(s), a_bytes);
                            asm volatile(
                                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                ::"r"(smem_u32(stg)), "l"(Aw + (size_t)c * a_bytes), "r"(a_bytes), "r"(bar_sfull(s))
                                : "memory");
                        }
                    }
                    k = q0 / ncl;
                    jc = q0 - k * ncl;
#pragma unroll
                    for (u32 i = 0; i < kOvtLoads; i++) {
                        const float sc = __shfl_sync(0xffffffffu, scale, min(k, 31u));
                        const u32 j = jc * 32 + lane;
                        if (k < spt && j < L)
                            B[k * 8 * P.ncol + nmax + j] = half_bits_clamped(__fmul_rn(f[i], sc));
                        if (++jc == ncl) { jc = 0; k++; }
                    }
                }
                if (stop) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_sfull(s));
            }
            gs0 += Cg;
        }
        // every copy into the ring has landed before the CTA exits (a warp
        // that issued one has also arrived)
        named_bar(1, kOvtProdThreads);
        if (tid == 0) {
            for (u32 s = 0; s < ns; s++)
                if (fills[s] > 0) mbar_wait_bounded(bar_sfull(s), (fills[s] - 1) & 1u, kTcDrainPolls);
        }
    } else if (warp == kOvtMmaWarp) {
        // =========================== MMA issue ===========================
        const u32 idesc = (1u << 4) | ((N >> 3) << 17) | ((u32)(kTcM >> 4) << 24);
        const u64 a0 = umma_desc(smem_u32(osm), kWATile / 2, 128);        // K halves 2048 B apart
        const u64 b0 = umma_desc(smem_u32(osm) + a_bytes, 16, 128);       // rows 8 positions apart
        const u64 sstep = (u64)(P.stage >> 4);
        u32 gs = 0, it = 0;
        bool issued = false;
        for (u64 item = blockIdx.x; item < nitems; item += gridDim.x, it++) {
            const u32 b = it & 1u, ub = it >> 1, Cg = P.groups[(u32)(item % G)].Cg;
            u32 ok = 1;
            if (lane == 0) {
                if (ub > 0 && !mbar_wait_bounded(bar_aempty(b), (ub - 1) & 1u, wlim)) {
                    atomicExch(P.err, 22u);
                    atomicExch(abort_flag, 1u);
                }
                if (*(volatile u32 *)abort_flag) ok = 0;
                const u32 dst = tmem + b * kWN;
                for (u32 c = 0; c < Cg && ok; c++, gs++) {
                    const u32 s = gs % ns, u = gs / ns;
                    if (!mbar_wait_bounded(bar_sfull(s), u & 1u, wlim)) {
                        atomicExch(P.err, 23u);
                        atomicExch(abort_flag, 1u);
                    }
                    if (*(volatile u32 *)abort_flag) { ok = 0; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    u64 da = a0 + s * sstep, db = b0 + s * sstep;
                    for (u32 k = 0; k < nkc; k++) {
                        const u32 acc = (c | k) != 0 ? 1u : 0u;   // the first MMA overwrites
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(dst), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
                        da += (u64)(kWATile >> 4);
                        db += 2u;
                    }
                    issued = true;
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                                 ::"r"(bar_sempty(s)) : "memory");
                }
                if (ok)
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                                 ::"r"(bar_afull(b)) : "memory");
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
        }
        // every MMA issued here is done before TMEM and the ring are released
        if (lane == 0 && issued) {
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(bar_fin) : "memory");
            mbar_wait_bounded(bar_fin, 0, kTcDrainPolls);
        }
        __syncwarp();
    } else {
        // =========================== epilogue ===========================
        const u32 ew_ = warp - kOvtEpiWarp0;         // 0..7
        const u32 quad = warp & 3u;                  // TMEM lanes [32 quad, 32 quad + 32)
        const u32 half = ew_ >> 2;                   // slots half, half + 2, ...
        const u32 row = quad * 32 + lane, tl = row >> 3, d = row & 7u;
        const float krm = ov_krm(A);
        u32 it = 0;
        for (u64 item = blockIdx.x; item < nitems; item += gridDim.x, it++) {
            const u32 b = it & 1u, ub = it >> 1, gi = (u32)(item % G);
            const TcwArgs &T = P.groups[gi];
            const u32 gbase = (u32)(item / G) * spt;
            const bool real = tl < T.nt;
            const u32 gt = real ? T.trow[tl] : 0u;
            const int texp_t = A.texp[gt];
            const float tn = A.tnorm[gt], tab = A.tabs[gt];
            // clipped norms of the template at this lane's shifts, the same for
            // every slot (the clipped energy is their square: its rounding is
            // far inside the tables' bound); 32 columns in registers
            const float *sNTt = A.sNT + (size_t)gt * S;
            auto norms = [&](u32 c0, float (&sn)[8]) {
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    sn[q] = __ldg(sNTt + min(8 * (c0 + q) + d, S - 1));   // unconditional: no load waits for another
                }
            };
            float snt[4][8];
#pragma unroll
            for (int q = 0; q < 4; q++) norms(8 * q, snt[q]);
            // lane k: slot k's candidate, its window norms over this group's channels
            uint4 sl = make_uint4(0xffffffffu, 0u, 0u, 0u);
            float wn = 0.0f, wa = 0.0f;
            if (lane < spt && gbase + lane < nc) sl = A.slot_tab[gbase + lane];
            if (sl.x != 0xffffffffu) {
                wn = A.lazy.wn[(size_t)gi * A.lazy.gstride + sl.x];
                wa = A.lazy.wa_f * wn;               // at most (the wide likelihood keeps no L1 norms)
            }
            u32 ok = 1;
            if (lane == 0) {
                if (!mbar_wait_bounded(bar_afull(b), ub & 1u, wlim)) {
                    atomicExch(P.err, 24u);
                    atomicExch(abort_flag, 1u);
                }
                if (*(volatile u32 *)abort_flag) ok = 0;
            }
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            // every lane observes the completed phase itself (the accumulator is ordered after it)
            if (!mbar_wait_bounded(bar_afull(b), ub & 1u, wlim)) atomicExch(abort_flag, 1u);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const u32 acc0 = tmem + ((quad * 32u) << 16) + b * kWN;
            for (u32 k = half; k < spt; k += 2) {
                const u32 bidx = __shfl_sync(0xffffffffu, sl.x, k);
                if (bidx == 0xffffffffu) continue;               // uniform in the warp
                const int kexp = (int)__shfl_sync(0xffffffffu, sl.y, k);
                const float tn0 = __uint_as_float(__shfl_sync(0xffffffffu, sl.z, k));
                const float vn = __shfl_sync(0xffffffffu, wn, k), va = __shfl_sync(0xffffffffu, wa, k);
                const u32 g = gbase + k;
                const int ex = -(kexp + texp_t);
                const bool plain = ex >= -149 && ex <= 127;
                const float sc = plain ? ldexpf(1.0f, ex) : 0.0f;    // exact power of two
                const float cst = 4.0f * kUnitRoundoff * tn0 * tn +
                                  (2.98023224e-08f * 1.001f) * (ldexpf(tab, -kexp) + ldexpf(va, -texp_t));
                const u32 xlo = bidx >= nmax ? 0u : nmax - bidx, xhi = n - L + nmax - bidx;   // .cl:534-541
                float *Hg = A.H + ((size_t)g * K + gt) * S;
                float mb = -INFINITY, v1 = -INFINITY;
                u32 b1 = 0;
                const bool odd = __any_sync(0xffffffffu, !plain);    // a scale outside the float range
                // (no branches: the eight elements of a chunk overlap)
                auto chunk = [&](u32 c0, const float (&sn)[8]) {
                    u32 r[8];
                    __syncwarp();
                    tmem_ld<8>(r, acc0 + k * P.ncol + c0);
                    float h[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) h[q] = __fmul_rn(__uint_as_float(r[q]), sc);
                    if (odd) {
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            if (!plain) h[q] = ldexpf(__uint_as_float(r[q]), ex);
                    }
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const u32 x = 8 * (c0 + q) + d;              // past the slot's columns: x >= S
                        const float nt = sn[q] * sn[q];
                        h[q] -= 0.5f * nt;
                        const float e = krm * (sn[q] * vn + nt) + 4.0f * kUnitRoundoff * fabsf(h[q]) + cst;
                        const bool inb = x >= xlo && x < xhi && x < S;
                        const float lo = inb ? h[q] - e : -INFINITY;
                        mb = fmaxf(mb, inb ? h[q] + e : -INFINITY);
                        b1 = lo > v1 ? x : b1;
                        v1 = fmaxf(v1, lo);
                    }
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const u32 x = 8 * (c0 + q) + d;
                        if (x < S && real) Hg[x] = h[q];
                    }
                };
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (8u * q < P.ncol) chunk(8 * q, snt[q]);
                for (u32 c0 = 32; c0 < P.ncol; c0 += 8) {
                    float sn[8];
                    norms(c0, sn);
                    chunk(c0, sn);
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {            // the template's 8 sample shifts
                    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, o));
                    const float ov = __shfl_xor_sync(0xffffffffu, v1, o);
                    const u32 oi = __shfl_xor_sync(0xffffffffu, b1, o);
                    if (ov > v1 || (ov == v1 && oi < b1)) { v1 = ov; b1 = oi; }
                }
                if (d == 0 && real) {
                    const size_t e = (size_t)g * K + gt;
                    A.pair_mb[e] = mb;
                    A.pair_v1[e] = v1;
                    A.pair_b1[e] = (u16)b1;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_aempty(b));
        }
    }
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kWN));
}

// Seed of each candidate's best lower bound after k_ov_tcw, one thread per
// (candidate, template): the item of the best template's row of largest lower
// bound (a1) and the template's own (b1).
__global__ void __launch_bounds__(kSeedThreads)
k_ov_seed_pairs(OvArgs A) {
    const u32 nc = *A.n_cand;
    const u32 S = A.S, K = A.K, L = A.L, nmax = A.nmax, n = A.n, R = 2 * L - 1, NB = (S + 31) / 32;
    const float kx = ov_kx(A);
    const u64 total = (u64)nc * K, step = (u64)gridDim.x * blockDim.x;
    const u32 lane = threadIdx.x & 31;
    for (u64 e0 = (u64)blockIdx.x * blockDim.x + threadIdx.x - lane; e0 < total; e0 += step) {
        const u64 e = e0 + lane;
        float seed = 0.0f;
        u32 g = 0;
        if (e < total) {
            g = (u32)(e / K);
            const u32 t = (u32)(e - (u64)g * K);
            if (!A.cskip[g] && A.ga_max[g] != -INFINITY) {
                const OvCand c = ov_cand(A, g);
                const u32 a = A.seed_a1[g], b = A.pair_b1[e];
                const float v1 = A.pair_v1[e], va = A.ga_lo[(size_t)g * S + a];
                // (b lies in the window unless the tables gave up on a wait)
                if (v1 > -INFINITY && va > -INFINITY && (a > b ? a - b : b - a) <= L && b < S && b >= c.xlo && b < c.xhi_ex) {
                    const bool fp = (A.ga_bits[(size_t)g * NB + (a >> 5)] >> (a & 31)) & 1u;
                    if (fp || !(A.Lk[(size_t)t * n + c.bidx + b - nmax] <= 0.0f)) {          // .cl:572-576
                        const float X = ov_disjoint(A.tsup, c.k0, t)
                                            ? 0.0f : ov_x(A.Q + ((size_t)c.k0 * K + t) * R * (L + 1), L,
                                                          (int)a - (int)nmax, (int)a - (int)b);
                        seed = va + v1 - X - kx * fabsf(X);
                    }
                }
            }
        }
        // one atomic per warp when its pairs are one candidate's
        const u32 g0 = __shfl_sync(0xffffffffu, g, 0);
        if (__all_sync(0xffffffffu, g == g0)) {
            seed = warp_max_f(seed);
            if (lane == 0 && seed > 0.0f) atomicMax(reinterpret_cast<int *>(A.cand_lb) + g, __float_as_int(seed));
        } else if (seed > 0.0f) {
            atomicMax(reinterpret_cast<int *>(A.cand_lb) + g, __float_as_int(seed));
        }
    }
}

}  // namespace fbp
