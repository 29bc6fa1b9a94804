// Path (a) on the tensor cores, wide tiles: the likelihood of every listed
// window as one tcgen05 contraction per (channel, 16-lag block) with
// M = 128 = 16 templates x 8 sample shifts and N = 256 blocks of 8 samples.
//
// likelihood[t][s] = -0.5*SS_t + sum_c sum_m T[t][c][m] * v[c][s+m]
// (compute_full_likelihood, binary_pursuit.cl:216-300).  Write s = s0 + 8u + d
// (d < 8) and j = m + d.  Then
//     sum_m T[t][c][m] v[c][s+m] = sum_j A[(t,d)][j] * B[u][j],
//     A[(t,d)][j] = T[t][c][j-d]  (zero outside 0 <= j-d < L),
//     B[u][j]     = v[c][s0 + 8u + j],
// with j < 16 * nkc, nkc = ceil((L + 7) / 16).  B is the channel's voltage
// stream itself: in the K-major no-swizzle UMMA layout a row is 16 bytes
// (8 fp16 samples), so rows 16 bytes apart (SBO 128 per 8 rows) and K halves
// 16 bytes apart (LBO 16) make row u start at sample 8u and read 16 samples.
// No im2col, and one MMA does 128 x 256 x 16 products where the
// sample-major kernel (fbp_lik_tc.cuh) does 128 x (templates in a group) x 16.
// A (the shifted templates) is packed once per chunk (k_tcw_pack) and
// streamed per channel into a ring of shared-memory stages with one bulk
// asynchronous copy.  Accumulators are FP32 in tensor memory (two tiles of
// 256 columns).
//
// What a pass computes.  A window's likelihoods under a template change only
// when a spike's subtraction touches samples the window's outputs read, on the
// template's channels.  Per window, a bit per group of 16 templates says
// whether that has happened since the group's last computation (dirty;
// k_gather_spikes sets it, the window argmax clears it), and a group computes
// the listed windows with its bit set: the others hold the values a
// recomputation from the same voltage would give.  On the 384-channel probe,
// whose templates cover 16 channels, that leaves about a fifth of the (window,
// group) pairs of a pursuit.
//
// The stream.  A group's windows w of a pass (ascending) are laid end to end:
// window i of its list starts at stream position
//     pos_i = i * L + R_i * (L - 1),
// R_i = the number of runs of consecutive windows before it, so a run is
// contiguous and every run is followed by L - 1 positions that continue its
// recording samples (the lags of its last outputs).  Those positions, and
// whatever lies past the last run, compute values that are dropped.  A tile
// is 2048 consecutive stream positions; dense passes fill it with ~33
// windows of L = 61, isolated windows still use about half of it.
//
// Exactness is the argument of fbp_lik_tc.cuh: the same bound E per entry
// (fp16 operands after exact power-of-two scaling, FP32 accumulation in any
// order -- a zero product adds and rounds nothing, so the count of rounded
// terms is the template support times L -- and the reference's recursive
// sum), the same three classes of entries and the same refinement list.
// The tile's voltage scale comes from a per-window bound on |v| over all
// channels (vwmax, kept by k_residual), covering every sample a kept output
// multiplies by a non-zero template value; other staged samples are clamped
// to the fp16 range, so no inf reaches a product with a zero template value.
#pragma once
#include <cuda_fp16.h>
#include <type_traits>
#include "fbp_lik_tc.cuh"

namespace fbp {

constexpr u32 kWN = 256;                 // MMA N: blocks of 8 samples per tile
constexpr u32 kWPos = 8 * kWN;           // 2048 stream positions per tile
constexpr u32 kWTwMax = 136;             // listed windows a tile can touch (L >= kWMinL)
constexpr u32 kWMinL = 16;
constexpr u32 kWATile = 4096;            // one A tile: 128 rows x 16 lags x fp16
__host__ __device__ inline u32 tcw_nkc(u32 L) { return (L + 7 + 15) / 16; }
__host__ __device__ inline u32 tcw_px(u32 L) { return kWPos + 16 * tcw_nkc(L); }   // staged positions

// One template group (16 templates in support order).
struct TcwArgs {
    u32 Cg, nt;                      // channels of the union of its supports, templates
    const u32 *trow;                 // [nt] template of each group column
    const float *v;                  // channel clo of the recording ([Cg][n] from there)
    const unsigned char *Aw;         // [Cg][nkc] A tiles
};
struct TcwParams {
    u32 n, L, ns, G, Kall, wstride, fstride;
    const TcwArgs *groups;           // [G]
    float kappa_b, kappa_s;
    const float *tss, *tnorm, *tabs;
    const int *texp;
    const float *vwmax;              // [W + 2] largest |v| of each window over all channels
    const u32 *win, *pos;            // [G][wstride] the group's windows of this pass, their stream positions
    const u32 *first;                // [G][fstride] first window of each tile of the group's stream
    const u32 *n_win, *n_stiles;     // [G] windows, tiles of the stream
    float *Lk;                       // [Kall][n]
    u8 *apx;                         // [Kall][n]
    float *dbgE;                     // testing: when set, the bound E of every entry ([Kall][n])
    float *wn_s;                     // [G][n] window norms
    float wa_f;                      // a window's L1 norm is at most wa_f times its L2 norm
    signed char *kx_s;               // [G][n] fp16 scale exponents
    float *wlb, *umax;               // [W][G], [W][Kall]
    u8 *wpos;                        // [W][G]
    u32 *ref_t, *ref_s;
    unsigned long long *refseg;
    u32 ref_cap;
    u32 *seg_s0, *seg_base, *seg_cnt, *seg_grp;
    u32 *seg_overflow;
    u32 seg_cap;
    u32 *err;
    u32 wait_polls;
};

// Warp roles: 4 table warps (the tile's table, position map and window
// norms), up to 7 producer warps (one per ring stage), 1 MMA warp, 8 epilogue
// warps.
constexpr int kWTabWarps = 4, kWTabThreads = 32 * kWTabWarps;
constexpr int kWProdWarp0 = kWTabWarps, kWProdWarps = 7;
constexpr int kWMmaWarp = kWProdWarp0 + kWProdWarps;
constexpr int kWEpiWarp0 = kWMmaWarp + 1, kWEpiWarps = 8, kWEpiThreads = 32 * kWEpiWarps;
constexpr int kWThreads = 32 * (kWEpiWarp0 + kWEpiWarps);
static_assert(kWEpiWarp0 % 4 == 0, "epilogue warp w reads TMEM lanes 32 (w % 4)..");
// ||window||_1 <= sqrt(terms) ||window||_2: it only scales the subnormal term of
// the bound, 2^-13 of the main one at most.
__host__ __device__ inline float tcw_l1_factor(u32 Cmax, u32 L) { return 1.001f * sqrtf((float)Cmax * (float)L); }
// Windows a tile's table can hold for this L (kWTwMax at L = kWMinL).
__host__ __device__ inline u32 tcw_entries(u32 L) {
    const u32 e = tcw_px(L) / L + 3;
    return e < kWTwMax ? e : kWTwMax;
}
constexpr u32 kWMaps = 3;                // position maps in flight: built, read by producers, by the epilogue
constexpr u32 kWLoads = 24;              // voltage loads of a producer lane in flight
constexpr u32 kWPart = 32 * kWLoads;     // positions a producer warp takes at a time
constexpr u32 kWParts = 4;               // parts of the staged positions at most (px <= 3072: L <= 1016)

struct TcwInfo {                         // per map: the tile
    u32 g, Cg;
    int kexp;
    float kscale;
    u32 gt[16];                          // template of each group column
    float ck[16], cb[16], css[16], ca[16], tsc[16], tsa[16];
    int texp[16];
};
static_assert(sizeof(TcwInfo) % 16 == 0, "what follows it in a map is stored in 8 and 16 bytes");
struct TcwSmem {
    size_t ring, stage, a_bytes, map, map_bytes, smap, wrel, tw, info, tpos, twin, ep, es, nrm, um, wl, bars, misc, tcnt, total;
};
__host__ __device__ inline TcwSmem tcw_smem_layout(u32 L, u32 ns) {
    const size_t nkc = tcw_nkc(L), px = tcw_px(L), rows = px / 8;
    TcwSmem m;
    m.a_bytes = nkc * kWATile;
    m.stage = align_up(m.a_bytes + align_up(px * 2, 16), 128);
    size_t o = 0;
    m.smap = o;  o += px * 4;                             // sample of every staged position, ~0 past the recording
    m.info = o;  o += sizeof(TcwInfo);
    m.wrel = o;  o += kWPos;                              // table entry of a kept output, else 0xff (8-byte stores)
    m.tw = o;    o += (size_t)tcw_entries(L) * 4;         // window of each table entry
    m.map_bytes = align_up(o, 16);
    o = 0;
    m.ring = o;  o += ns * m.stage;                       // A tiles + voltage stream per channel
    m.map = o;   o += kWMaps * m.map_bytes;
    m.tpos = o;  o += (size_t)(tcw_entries(L) + 1) * 4;   // table warps: stream position and window of each entry
    m.twin = o;  o += (size_t)(tcw_entries(L) + 1) * 4;
    m.ep = o;    o += (size_t)ns * rows * 4;              // energies of the blocks of 8 (scaled samples), per producer
    m.es = o;    o += 2 * rows * 4;                       // and of all channels, by the tile's parity
    m.nrm = o;   o += 2 * (size_t)kWN * 4;                // epilogue: window norms per block of 8, two spans
    m.um = o;    o += (size_t)16 * tcw_entries(L) * 4;    //           upper bounds per (template, window)
    m.wl = o;    o += (size_t)tcw_entries(L) * 4;         //           lower bounds per window
    o = align_up(o, 8);
    m.bars = o;  o += (size_t)(2 * ns + 7 + 3 * kWMaps) * 8;
    m.misc = o;  o += 256;
    m.tcnt = o;  o += 16 * 4;
    m.total = o;
    return m;
}

__device__ __forceinline__ void mbar_expect_tx(u32 bar, u32 bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ u32 named_bar_popc(u32 id, u32 count, bool v) {
    u32 r;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.popc.u32 %0, %2, %3, p;\n\t}"
        : "=r"(r) : "r"((u32)v), "r"(id), "r"(count) : "memory");
    return r;
}
// Sums of squares over each group of 8 lanes, of 8 values per lane: lane l gets
// the one of z[l & 7] over its group (each step a lane keeps half of its values
// and takes its partner's for them: 4 + 2 + 1 shuffles).
__device__ __forceinline__ float octet_energy(const float *z, u32 lane) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __fmul_rn(z[i], z[i]);
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) {
        const bool hi = (lane & (u32)h) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const float send = hi ? v[i] : v[i + h], keep = hi ? v[i + h] : v[i];
            v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, h));
        }
    }
    return v[0];
}
__device__ __forceinline__ u16 half_bits_clamped(float f) {
    return __half_as_ushort(__float2half_rn(fminf(fmaxf(f, -65504.0f), 65504.0f)));
}

// Persistent, one CTA per SM, 20 warps.  The tiles of all groups' streams form
// one sequence; CTA b takes tiles b, b + gridDim, ...
//   Table warps, per tile, one tile ahead: the windows that meet it, the sample
//     of every position, the tile's fp16 scale and per-template factors; at the
//     end of a tile the energies of its blocks of 8 positions, from the
//     producers' parts.
//   Producer warp s fills ring stage s: a channel's voltage by coalesced 4-byte
//     loads (24 in flight per lane, the first ones issued before the wait for
//     the stage), scaled, rounded to fp16; one bulk copy brings the channel's A
//     tiles.  It also sums the energies of its float32 samples over blocks of 8
//     positions (seven shuffles reduce eight loads of 32 lanes to a block a
//     lane).  No barrier joins the producers.  (Energies of the fp16 samples,
//     read from the stages by the table warps, took 17.9 in place of 20.1 ms on
//     the 384-channel probe's 100 s, and as much on 16 channels; table warps
//     that load the float32 samples again took 30, since the loads are what
//     bounds a tile, and a producer that adds its sums to the one before it 20.8.)
//   The MMA warp issues nkc MMAs per channel.
//   Epilogue warps (two per TMEM lane quadrant, one half of the columns each)
//     bound every output's window norm by the blocks that hold its lags,
//     classify and store; the entries that are not certainly <= 0 update the
//     per-(window, template) and per-window bounds of the tile in shared
//     memory, which go to global memory once per tile (global atomics per
//     entry took 110,000 of 135,000 cycles a tile).
// Producers that shared every channel over 256 threads with two barriers a
// channel and built the tables and norms between tiles took 144,000 cycles a
// tile of 34 channels, against 31,000 of MMA issue.
// Barriers:
//   stage_full[s]  the producer arrived and the A copy landed (tx);
//   stage_empty[s] the MMAs that read stage s are done (tcgen05.commit);
//   acc_full[b]    the tile's MMAs are done (commit);
//   acc_empty[b]   the epilogue read accumulator b (one arrive per warp);
//   map_full[k], norm_full[k]  map k is built, its norms are (one arrive each);
//   map_empty[k]   producers and epilogue are done with map k (one arrive per warp).
// Every wait is bounded; a wait that gives up sets err and the abort flag.
__global__ void __launch_bounds__(kWThreads, 1)
k_lik_tcw(const __grid_constant__ TcwParams P) {
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const u32 G = P.G;
    u32 total = 0;                                   // tiles of all groups
    for (u32 g = lane; g < G; g += 32) total += P.n_stiles[g];
    total = __reduce_add_sync(0xffffffffu, total);
    if (blockIdx.x >= total) return;                 // no tile for this CTA: no set-up at all
    extern __shared__ __align__(128) unsigned char wsm[];
    const u32 L = P.L, ns = P.ns, n = P.n, nkc = tcw_nkc(L), px = tcw_px(L);
    const TcwSmem lay = tcw_smem_layout(L, ns);
    unsigned char *ring = wsm + lay.ring;
    auto map_of = [&](u32 k) { return wsm + lay.map + (size_t)k * lay.map_bytes; };
    u64 *bars = (u64 *)(wsm + lay.bars);
    u32 *misc = (u32 *)(wsm + lay.misc);
    u32 *tmem_slot = misc, *seg_info = misc + 1, *abort_flag = misc + 4, *fills = misc + 8;   // fills: [ns]
    float *pred = (float *)(misc + 16);              // [4] table warps' maxima
    u32 *tcnt = (u32 *)(wsm + lay.tcnt);
    const u32 wlim = P.wait_polls;
    auto bar_sfull = [&](u32 s) { return smem_u32(&bars[s]); };
    auto bar_sempty = [&](u32 s) { return smem_u32(&bars[ns + s]); };
    auto bar_afull = [&](u32 b) { return smem_u32(&bars[2 * ns + b]); };
    auto bar_aempty = [&](u32 b) { return smem_u32(&bars[2 * ns + 2 + b]); };
    auto bar_mfull = [&](u32 k) { return smem_u32(&bars[2 * ns + 4 + k]); };
    auto bar_nfull = [&](u32 k) { return smem_u32(&bars[2 * ns + 4 + kWMaps + k]); };
    auto bar_mempty = [&](u32 k) { return smem_u32(&bars[2 * ns + 4 + 2 * kWMaps + k]); };
    const u32 bar_fin = smem_u32(&bars[2 * ns + 4 + 3 * kWMaps]);
    const u32 bar_efull = smem_u32(&bars[2 * ns + 5 + 3 * kWMaps]), bar_eempty = smem_u32(&bars[2 * ns + 6 + 3 * kWMaps]);
    const u32 rows = px / 8;                         // blocks of 8 staged positions
    auto aborted = [&]() { return *(volatile u32 *)abort_flag != 0; };
    // a wait of one warp: false when it gave up or another role has
    auto wait_warp = [&](u32 bar, u32 parity, u32 code) -> bool {
        bool ok = !aborted();
        if (ok && !mbar_wait_bounded(bar, parity, wlim)) {
            if (lane == 0) atomicExch(P.err, code);
            atomicExch(abort_flag, 1u);
            ok = false;
        }
        return __all_sync(0xffffffffu, ok);
    };

    if (tid == 0) {
        for (u32 s = 0; s < ns; s++) {
            mbar_init(bar_sfull(s), 1);
            mbar_init(bar_sempty(s), 1);
            fills[s] = 0;
        }
        for (u32 b = 0; b < 2; b++) {
            mbar_init(bar_afull(b), 1);
            mbar_init(bar_aempty(b), kWEpiWarps);
        }
        for (u32 k = 0; k < kWMaps; k++) {
            mbar_init(bar_mfull(k), 1);
            mbar_init(bar_nfull(k), 1);
            mbar_init(bar_mempty(k), ns + kWEpiWarps);
        }
        mbar_init(bar_fin, 1);
        mbar_init(bar_efull, ns);
        mbar_init(bar_eempty, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(2 * kWN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid < 16) tcnt[tid] = 0;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const u32 tmem = *tmem_slot;

    if (warp < kWTabWarps) {
        // ============================ tables =============================
        const u32 tt = tid;                          // 0..127
        const u32 TW = tcw_entries(L);
        int *tpos = (int *)(wsm + lay.tpos);
        u32 *twin = (u32 *)(wsm + lay.twin);
        // waits until the tile that had the map of the CTA's it-th tile is done
        auto map_free = [&](u32 it) -> bool {
            const u32 k = it % kWMaps, use = it / kWMaps;
            const bool ok = use == 0 || wait_warp(bar_mempty(k), (use - 1) & 1u, 13u);
            return !named_bar_or(3, kWTabThreads, !ok);
        };
        // builds the map of the CTA's it-th tile; false when a role gave up
        auto build = [&](u32 f, u32 it) -> bool {
            const u32 k = it % kWMaps;
            unsigned char *mp = map_of(k);
            u32 *smap = (u32 *)(mp + lay.smap), *tw = (u32 *)(mp + lay.tw);
            u8 *wrel = mp + lay.wrel;
            TcwInfo &I = *(TcwInfo *)(mp + lay.info);
            if (!map_free(it)) return false;
            // the tile's group and its place in the group's stream.  Group after
            // group: tiles computed together write the rows of 16 templates and
            // read one group's channels (taking every group's tile 0, then tile
            // 1, ... spreads them over all rows, 1,000 pages of 2 MB on the
            // 384-channel probe: its first pass of 100 s took 1.7 times as long)
            u32 g = 0, q = f;
            for (u32 g0 = 0; g0 < G; g0 += 32) {
                const u32 t = g0 + lane < G ? P.n_stiles[g0 + lane] : 0u;
                const u32 incl = warp_incl_scan(t);
                const u32 m = __ballot_sync(0xffffffffu, q < incl);
                if (m) {
                    const u32 src = __ffs(m) - 1;
                    g = g0 + src;
                    q -= __shfl_sync(0xffffffffu, incl - t, src);
                    break;
                }
                q -= __shfl_sync(0xffffffffu, incl, 31);
            }
            const TcwArgs &T = P.groups[g];
            // the windows whose outputs or lags meet positions [Q0, Q0 + px)
            const long long Q0 = (long long)q * kWPos;
            const u32 m = P.n_win[g], i_lo = P.first[(size_t)g * P.fstride + q];
            const u32 *gpos = P.pos + (size_t)g * P.wstride, *gwin = P.win + (size_t)g * P.wstride;
            u32 nw = 0;
            float mx = 0.0f;
            for (u32 b0 = 0; b0 < TW + 1; b0 += kWTabThreads) {
                const u32 e = b0 + tt, i = i_lo + e;
                bool in = e <= TW && i < m && (long long)gpos[i] < Q0 + (long long)px;
                if (in && e == TW) {                 // cannot happen: windows start at least L positions apart
                    atomicExch(P.err, 15u);
                    atomicExch(abort_flag, 1u);
                    in = false;
                }
                if (in) {
                    const u32 w = gwin[i];
                    tpos[e] = (int)((long long)gpos[i] - Q0);
                    twin[e] = w;
                    tw[e] = w;
                    // every sample a kept output multiplies by a non-zero
                    // template value lies in its window or the next
                    mx = fmaxf(mx, fmaxf(P.vwmax[w], P.vwmax[w + 1]));
                }
                nw += named_bar_popc(3, kWTabThreads, in);          // also publishes the table
            }
            if (nw == 0 || tpos[0] > 0) {            // the list kernels guarantee an entry at or before Q0
                if (tt == 0) { atomicExch(P.err, 16u); atomicExch(abort_flag, 1u); }
                nw = 0;
            }
            mx = warp_max_float(mx);
            if (lane == 0) pred[warp] = mx;
            if (named_bar_or(3, kWTabThreads, nw == 0 || aborted())) return false;
            float mm = 0.0f;
            for (int w4 = 0; w4 < kWTabWarps; w4++) mm = fmaxf(mm, pred[w4]);
            int kexp = 0;
            if (mm > 0.0f) {
                int e;
                frexpf(mm, &e);                      // mm < 2^e
                kexp = max(-126, min(126, 14 - e));  // scaled magnitudes < 2^14
            }
            if (tt == 0) {
                I.g = g;
                I.Cg = T.Cg;
                I.kexp = kexp;
                I.kscale = ldexpf(1.0f, kexp);       // exact: |kexp| <= 126
            }
            if (tt < 16) {
                const bool real = tt < T.nt;
                const u32 gt = real ? T.trow[tt] : 0u;
                const int te = real ? P.texp[gt] : 0, ex = -(kexp + te);
                I.gt[tt] = real ? gt : 0xffffffffu;
                I.texp[tt] = te;
                I.ck[tt] = real ? P.kappa_b * P.tnorm[gt] : 0.0f;
                I.cb[tt] = real ? 2.98023223876953125e-08f * 1.001f * ldexpf(1.0f, -te) : 0.0f;
                I.css[tt] = real ? P.tss[gt] : 0.0f;
                I.ca[tt] = real ? P.kappa_s * fabsf(P.tss[gt]) : 0.0f;
                I.tsc[tt] = (real && ex >= -149 && ex <= 127) ? ldexpf(1.0f, ex) : 0.0f;   // exact power of two
                I.tsa[tt] = real ? 2.98023223876953125e-08f * 1.001f * ldexpf(P.tabs[gt], -kexp) : 0.0f;
            }
            for (u32 r = tt; r < rows; r += kWTabThreads) {          // 8 positions of a block
                const u32 x0 = 8 * r;
                u32 lo = 0, hi = nw - 1;             // last entry with tpos <= x0
                while (lo < hi) {
                    const u32 mid = (lo + hi + 1) >> 1;
                    if (tpos[mid] <= (int)x0) lo = mid; else hi = mid - 1;
                }
                u32 j = lo, sv[8], wv[2] = {0u, 0u};
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const u32 x = x0 + e;
                    while (j + 1 < nw && tpos[j + 1] <= (int)x) j++;
                    const u32 o = (u32)((int)x - tpos[j]);
                    const u32 s = twin[j] * L + o;
                    sv[e] = s < n ? s : 0xffffffffu;
                    wv[e >> 2] |= ((o < L && s < n) ? j : 0xffu) << (8 * (e & 3));
                }
                *reinterpret_cast<uint4 *>(smap + x0) = make_uint4(sv[0], sv[1], sv[2], sv[3]);
                *reinterpret_cast<uint4 *>(smap + x0 + 4) = make_uint4(sv[4], sv[5], sv[6], sv[7]);
                if (x0 < kWPos) *reinterpret_cast<uint2 *>(wrel + x0) = make_uint2(wv[0], wv[1]);
            }
            named_bar(3, kWTabThreads);
            if (tt == 0) mbar_arrive(bar_mfull(k));  // release: the barrier ordered every write
            return true;
        };
        u32 it = 0;
        bool ok = build(blockIdx.x, 0);
        for (u32 f = blockIdx.x; ok && f < total; f += gridDim.x, it++) {
            // once the tile three before the next is done, the one two before this has
            // had its energies read: their place is free
            if (f + gridDim.x < total ? !build(f + gridDim.x, it + 1) : !map_free(it + 1)) break;
            const bool full = wait_warp(bar_efull, it & 1u, 17u);
            const float *ep = (const float *)(wsm + lay.ep);
            float *es = (float *)(wsm + lay.es) + (it & 1u) * rows;
            for (u32 row = tt; full && row < rows; row += kWTabThreads) {
                float e = ep[row];
                for (u32 q = 1; q < ns; q++) e = __fadd_rn(e, ep[(size_t)q * rows + row]);
                es[row] = e;
            }
            if (named_bar_or(3, kWTabThreads, aborted())) break;
            if (tt == 0) {
                mbar_arrive(bar_eempty);
                mbar_arrive(bar_nfull(it % kWMaps));
            }
        }
    } else if (warp < kWMmaWarp) {
        // =========================== producers ===========================
        const u32 s = warp - kWProdWarp0;            // this warp's ring stage
        u32 gs0 = 0, it = 0;
        unsigned char *stg = ring + (size_t)s * lay.stage;
        u16 *B = reinterpret_cast<u16 *>(stg + lay.a_bytes);
        bool stop = s >= ns;
        for (u32 f = blockIdx.x; !stop && f < total; f += gridDim.x, it++) {
            const u32 k = it % kWMaps;
            if (!wait_warp(bar_mfull(k), (it / kWMaps) & 1u, 18u)) break;
            const unsigned char *mp = map_of(k);
            const u32 *smap = (const u32 *)(mp + lay.smap);
            const TcwInfo &I = *(const TcwInfo *)(mp + lay.info);
            const TcwArgs &T = P.groups[I.g];
            const float kscale = I.kscale;
            const float *v = T.v;
            const unsigned char *Aw = T.Aw;
            const u32 Cg = I.Cg;
            // energies of this warp's channels: the lane's block of part p, eight loads j
            float e2[kWParts][kWLoads / 8];
#pragma unroll
            for (u32 j = 0; j < kWLoads / 8; j++)
#pragma unroll
                for (u32 q = 0; q < kWParts; q++) e2[q][j] = 0.0f;
            for (u32 c = (s + ns - gs0 % ns) % ns; c < Cg; c += ns) {
                const u32 u = (gs0 + c) / ns;
                const float *vc = v + (size_t)c * n;
#pragma unroll 1
                for (u32 p = 0; p * kWPart < px; p++) {
                    const u32 x0 = p * kWPart + lane;
                    float fv[kWLoads];
#pragma unroll
                    for (u32 i = 0; i < kWLoads; i++) {
                        const u32 x = x0 + 32 * i;
                        // unconditional, so that the loads do not wait for one another; a
                        // position past the recording reads its last sample, which no
                        // output that is not in the zeroed tail multiplies
                        fv[i] = __ldg(vc + min(smap[min(x, px - 1)], n - 1));
                    }
                    if (p == 0) {                    // the first loads are in flight
                        if (u > 0 && !wait_warp(bar_sempty(s), (u - 1) & 1u, 11u)) { stop = true; break; }
                        if (lane == 0) {
                            fills[s] = u + 1;
                            mbar_expect_tx(bar_sfull(s), (u32)lay.a_bytes);
                            asm volatile(
                                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                ::"r"(smem_u32(stg)), "l"(Aw + (size_t)c * lay.a_bytes), "r"((u32)lay.a_bytes),
                                  "r"(bar_sfull(s)) : "memory");
                        }
                    }
#pragma unroll
                    for (u32 j = 0; j < kWLoads / 8; j++) {
                        if (p * kWPart + 256 * j >= px) break;       // uniform
                        float z[8];
#pragma unroll
                        for (u32 r = 0; r < 8; r++) {
                            const u32 x = x0 + 256 * j + 32 * r;
                            z[r] = fminf(fmaxf(__fmul_rn(fv[8 * j + r], kscale), -65504.0f), 65504.0f);
                            if (x < px) B[x] = __half_as_ushort(__float2half_rn(z[r]));
                        }
                        const float e = octet_energy(z, lane);
#pragma unroll
                        for (u32 q = 0; q < kWParts; q++)            // registers: no index that varies
                            e2[q][j] = __fadd_rn(e2[q][j], q == p ? e : 0.0f);
                    }
                }
                if (stop) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_sfull(s));
            }
            // to the table warps, which have long added the tile before
            if (!stop && it > 0) stop = !wait_warp(bar_eempty, (it - 1) & 1u, 25u);
            if (!stop) {
                float *ep = (float *)(wsm + lay.ep) + (size_t)s * rows;
#pragma unroll
                for (u32 q = 0; q < kWParts; q++)
#pragma unroll
                    for (u32 j = 0; j < kWLoads / 8; j++) {
                        const u32 row = q * (kWPart / 8) + 32 * j + 4 * (lane & 7) + (lane >> 3);
                        if (row < rows) ep[row] = e2[q][j];
                    }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_efull);
            }
            if (stop) break;
            gs0 += Cg;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_mempty(k));
        }
        // every copy into the ring has landed before the CTA exits (a warp
        // that issued one has also arrived)
        __syncwarp();
        if (lane == 0 && s < ns && fills[s] > 0) mbar_wait_bounded(bar_sfull(s), (fills[s] - 1) & 1u, kTcDrainPolls);
    } else if (warp == kWMmaWarp) {
        // =========================== MMA issue ===========================
        // D f32, A/B f16, both K-major, M = 128, N = 256
        const u32 idesc = (1u << 4) | ((kWN >> 3) << 17) | ((u32)(kTcM >> 4) << 24);
        const u64 a0 = umma_desc(smem_u32(ring), kWATile / 2, 128);       // K halves 2048 B apart
        const u64 b0 = umma_desc(smem_u32(ring) + (u32)lay.a_bytes, 16, 128);   // rows 8 samples apart
        const u64 sstep = (u64)(lay.stage >> 4);
        u32 gs = 0, it = 0;
        bool issued = false;
        for (u32 f = blockIdx.x; f < total; f += gridDim.x, it++) {
            const u32 b = it & 1u, ub = it >> 1, k = it % kWMaps;
            if (!wait_warp(bar_mfull(k), (it / kWMaps) & 1u, 19u)) break;
            const u32 Cg = ((const TcwInfo *)(map_of(k) + lay.info))->Cg;
            if (ub > 0 && !wait_warp(bar_aempty(b), (ub - 1) & 1u, 12u)) break;
            const u32 dst = tmem + b * kWN;
            bool ok = true;
            for (u32 c = 0; c < Cg && ok; c++, gs++) {
                const u32 s = gs % ns, u = gs / ns;
                ok = wait_warp(bar_sfull(s), u & 1u, 14u);
                if (ok && lane == 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    u64 da = a0 + s * sstep, db = b0 + s * sstep;
                    for (u32 q = 0; q < nkc; q++) {
                        const u32 acc = (c | q) != 0 ? 1u : 0u;   // the first MMA overwrites
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            ::"r"(dst), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
                        da += (u64)(kWATile >> 4);           // next A tile
                        db += 2u;                            // 16 samples (32 bytes) later
                    }
                    issued = true;
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                                 ::"r"(bar_sempty(s)) : "memory");
                }
                __syncwarp();
            }
            if (!ok) break;
            if (lane == 0)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             ::"r"(bar_afull(b)) : "memory");
            __syncwarp();
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
        const u32 ew_ = warp - kWEpiWarp0;           // 0..7
        const u32 quad = warp & 3u;                  // TMEM lanes [32 quad, 32 quad + 32)
        const u32 half = ew_ >> 2;                   // columns [128 half, 128 half + 128)
        const u32 row = quad * 32 + lane;
        const u32 tl = row >> 3, d = row & 7u;       // template column, sample shift
        const u32 span = d + (L - 1) % 8 >= 8 ? kWN : 0u;    // which of the two norm spans
        const u32 et = tid - 32 * kWEpiWarp0;        // 0..255
        const u32 TW = tcw_entries(L);
        float *nrm_all = (float *)(wsm + lay.nrm);
        int *um = (int *)(wsm + lay.um), *wl = (int *)(wsm + lay.wl);    // [16][TW], [TW]
        for (u32 q = et; q < 16 * TW; q += kWEpiThreads) um[q] = 0;
        for (u32 q = et; q < TW; q += kWEpiThreads) wl[q] = 0;
        u32 it = 0;
        for (u32 f = blockIdx.x; f < total; f += gridDim.x, it++) {
            const u32 b = it & 1u, ub = it >> 1, k3 = it % kWMaps;
            bool ok = wait_warp(bar_mfull(k3), (it / kWMaps) & 1u, 20u) &&
                      wait_warp(bar_nfull(k3), (it / kWMaps) & 1u, 20u) && wait_warp(bar_afull(b), ub & 1u, 10u);
            if (named_bar_or(2, kWEpiThreads, !ok || aborted())) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned char *mp = map_of(k3);
            const u32 *smap = (const u32 *)(mp + lay.smap), *tw = (const u32 *)(mp + lay.tw);
            const u8 *wrel = mp + lay.wrel;
            const TcwInfo &I = *(const TcwInfo *)(mp + lay.info);
            const u32 gi = I.g;
            {
                // norms of the blocks that hold an output's lags: output 8 u + d
                // reads blocks u .. u + (L - 1) / 8, one more when d + (L - 1) % 8
                // reaches 8.  A block's energy took a product, three adds over
                // the lanes and one for every channel and warp, each rounded to
                // float32 (what the products lose below the normal range, 2^-150
                // each, the added 2^-60 of the scaled samples covers); the blocks
                // are added in float64.
                const float *es = (const float *)(wsm + lay.es) + (it & 1u) * rows;
                const float up = 1.0f + 6.6e-8f * (float)(I.Cg + 32);
                const float add = ldexpf(8.7e-19f, -I.kexp) + 1e-30f;
                double e = 0.0;
                const u32 nb = (L - 1) / 8 + 1;
                for (u32 q = 0; q < nb; q++) e += (double)es[et + q];
                nrm_all[et] = ldexpf(sqrtf((float)e) * up, -I.kexp) + add;
                nrm_all[kWN + et] = ldexpf(sqrtf((float)(e + (double)es[et + nb])) * up, -I.kexp) + add;
            }
            named_bar(2, kWEpiThreads);
            const float *nrm = nrm_all + span;
            // interval data of the kept outputs (read by later kernels)
            for (u32 x = et; x < kWPos; x += kWEpiThreads) {
                if (wrel[x] == 0xffu) continue;
                const size_t o = (size_t)gi * n + smap[x];
                P.wn_s[o] = nrm_all[(x >> 3) + ((x & 7u) + (L - 1) % 8 >= 8 ? kWN : 0u)];
                P.kx_s[o] = (signed char)I.kexp;
            }
            const bool real = I.gt[tl] != 0xffffffffu;
            const u32 gt = real ? I.gt[tl] : 0u;
            const float ck = fmaf(I.cb[tl], P.wa_f, I.ck[tl]), css = I.css[tl], tsc = I.tsc[tl];
            const float cst = I.tsa[tl] + I.ca[tl];
            const int ex = -(I.kexp + I.texp[tl]);
            // this lane's template row of the likelihood and flag buffers
            float *const Lk_t = P.Lk + (size_t)gt * n;
            u8 *const apx_t = P.apx + (size_t)gt * n;
            float *const dbg_t = P.dbgE ? P.dbgE + (size_t)gt * n : nullptr;
            const u32 acc0 = tmem + ((quad * 32u) << 16) + b * kWN;
            // the rare cases (a scale outside the float range, the testing
            // output of E) take a separate, warp-uniform copy of the loop
            const bool rare = __any_sync(0xffffffffu, real && tsc == 0.0f) || dbg_t != nullptr;
            u32 curw = 0xffu;                        // table entry the lane's running bounds belong to
            float mu = 0.0f, ml = 0.0f;
            auto flush = [&]() {
                if (mu > 0.0f) atomicMax(um + tl * TW + curw, __float_as_int(mu));
                if (ml > 0.0f) atomicMax(wl + curw, __float_as_int(ml));
            };
            u32 want[4];                             // bit 8 (k & 3) + j of word k / 4: column 8 k + j of this half
#pragma unroll
            for (int q = 0; q < 4; q++) want[q] = 0;
            // one 8-column chunk: classify and store its entries.  Every shared
            // read first, then the arithmetic, then the stores, so that a column
            // does not wait for the one before it; the few entries that are not
            // certainly <= 0 afterwards, column by column.
            auto chunk = [&](const int k, auto RARE) {
                constexpr bool kRare = decltype(RARE)::value;
                const u32 c0 = 128 * half + 8 * k;
                u32 r[8], sm[8], wr[8];
                float ap[8], E[8];
                float nw[8];
                __syncwarp();
                tmem_ld<8>(r, acc0 + c0);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    sm[j] = smap[8 * (c0 + j) + d];
                    wr[j] = wrel[8 * (c0 + j) + d];
                    nw[j] = nrm[c0 + j];
                }
                u32 hot = 0, pos = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float a = __uint_as_float(r[j]);
                    float sa = __fmul_rn(a, tsc);
                    if (kRare && tsc == 0.0f) sa = ldexpf(a, ex);
                    ap[j] = __fadd_rn(sa, css);
                    // E = kappa ||t|| ||w|| + 2^-25 (|t|_1 / s_v + |w|_1 / s_t) * 1.001
                    //     + kappa_s |SS/2| + 2^-22 |approx|
                    E[j] = fmaf(ck, nw[j], cst + 2.384185791015625e-07f * fabsf(ap[j]));
                    const bool kept = real && wr[j] != 0xffu;
                    const bool tail = sm[j] + L >= n;                // .cl:231-234 (kept outputs: s < n < 2^31)
                    const bool live = kept && !tail;
                    const bool p = live && ap[j] - E[j] > 0.0f;      // certainly > 0: refined when a decision needs it
                    hot |= live && !(ap[j] + E[j] <= 0.0f) ? 1u << j : 0u;   // not certainly <= 0
                    pos |= p ? 1u << j : 0u;
                    if (kept) {
                        Lk_t[sm[j]] = tail ? 0.0f : ap[j];
                        apx_t[sm[j]] = p ? (u8)1 : (u8)0;
                        if (kRare && dbg_t) dbg_t[sm[j]] = tail ? 0.0f : E[j];
                    }
                }
                want[k >> 2] |= (hot & ~pos) << (8 * (k & 3));
                // bounds per (window, template) and per window: a lane's columns
                // pass through the windows in order, so it keeps the running
                // maxima of one window and hands them over when it leaves it
                if (!__any_sync(0xffffffffu, hot != 0)) return;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (!((hot >> j) & 1u)) continue;
                    if (wr[j] != curw) {
                        flush();
                        curw = wr[j];
                        mu = ml = 0.0f;
                    }
                    mu = fmaxf(mu, ap[j] + E[j]);
                    if ((pos >> j) & 1u) ml = fmaxf(ml, ap[j] - E[j]);
                }
            };
            if (rare) {
#pragma unroll
                for (int k = 0; k < 16; k++) chunk(k, std::true_type{});
            } else {
#pragma unroll
                for (int k = 0; k < 16; k++) chunk(k, std::false_type{});
            }
            flush();
            // accumulator b is no longer needed
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_aempty(b));
            u32 nwant = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) nwant += __popc(want[q]);
            const bool queue = named_bar_or(2, kWEpiThreads, nwant != 0);   // also orders the bounds in shared memory
            // the tile's bounds to global memory (a window may lie in two tiles)
            for (u32 q = et; q < 16 * TW; q += kWEpiThreads) {
                const int v = um[q];
                if (v == 0) continue;
                um[q] = 0;
                atomicMax(reinterpret_cast<int *>(P.umax) + (size_t)tw[q % TW] * P.Kall + I.gt[q / TW], v);
            }
            for (u32 q = et; q < TW; q += kWEpiThreads) {
                const int v = wl[q];
                if (v == 0) continue;
                wl[q] = 0;
                atomicMax(reinterpret_cast<int *>(P.wlb) + (size_t)tw[q] * G + gi, v);
                P.wpos[(size_t)tw[q] * G + gi] = 1;
            }
            if (queue) {
                // one contiguous segment of (template, sample) entries per
                // tile, ordered by template (tcnt is zero here)
                if (nwant) atomicAdd(&tcnt[tl], nwant);
                named_bar(2, kWEpiThreads);
                if (ew_ == 0) {
                    const u32 cnt_t = lane < 16 ? tcnt[lane] : 0u;
                    const u32 incl = warp_incl_scan(cnt_t);
                    if (lane < 16) tcnt[lane] = incl - cnt_t;
                    const u32 tot = __shfl_sync(0xffffffffu, incl, 31);
                    if (lane == 0) {
                        const unsigned long long old = atomicAdd(P.refseg, ((unsigned long long)tot << 32) | 1ull);
                        const u32 base = (u32)(old >> 32), si = (u32)old;
                        seg_info[0] = base;
                        seg_info[2] = 0;
                        if (base + tot <= P.ref_cap && si < P.seg_cap) {
                            P.seg_s0[si] = 0;                // entries carry their absolute samples
                            P.seg_base[si] = base;
                            P.seg_cnt[si] = tot;
                            P.seg_grp[si] = gi;
                            seg_info[2] = 1;
                        } else {
                            atomicExch(P.seg_overflow, 1u);
                        }
                    }
                }
                named_bar(2, kWEpiThreads);
                const u32 seg_base = seg_info[0];
                if (seg_info[2] && nwant) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        u32 bits = want[q];
                        while (bits) {
                            const u32 j = __ffs(bits) - 1;
                            bits &= bits - 1;
                            const u32 x = 8 * (128 * half + 32 * q + j) + d;
                            const u32 p = seg_base + atomicAdd(&tcnt[tl], 1u);
                            P.ref_t[p] = tl;
                            P.ref_s[p] = smap[x];
                        }
                    }
                }
                named_bar(2, kWEpiThreads);          // tcnt / seg_info are done with
                if (ew_ == 0 && lane < 16) tcnt[lane] = 0;
            }
            // the tile's map is no longer needed
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_mempty(k3));
        }
    }
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kWN));
}

// A tiles of one template group: Aw[c][k] = 128 rows (template tl = row / 8,
// shift d = row % 8) x 16 lags j = 16k + jj, holding T[trow[tl]][clo + c][j - d]
// scaled by 2^texp (zero outside 0 <= j - d < L and for tl >= nt), in the
// K-major no-swizzle layout: K half (jj / 8) 2048 bytes apart, 8-row groups
// 128 bytes apart, rows 16 bytes apart.
__global__ void k_tcw_pack(const float *__restrict__ T, u32 Call, u32 L, u32 nkc, const u32 *__restrict__ trow,
                           u32 nt, u32 clo, u32 Cg, const int *__restrict__ texp, u16 *__restrict__ Aw) {
    const u64 total = (u64)Cg * nkc * (kWATile / 2);
    for (u64 e = (u64)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (u64)gridDim.x * blockDim.x) {
        const u32 within = (u32)(e % (kWATile / 2)), tile = (u32)(e / (kWATile / 2));
        const u32 c = tile / nkc, k = tile % nkc;
        const u32 h = within >> 10, tl = (within >> 6) & 15u, d = (within >> 3) & 7u, el = within & 7u;
        const int lag = (int)(16 * k + 8 * h + el) - (int)d;
        float f = 0.0f;
        if (tl < nt && lag >= 0 && lag < (int)L) {
            const u32 t = trow[tl];
            f = ldexpf(T[((size_t)t * Call + clo + c) * L + (u32)lag], texp[t]);
        }
        Aw[e] = __half_as_ushort(__float2half_rn(f));
    }
}

// Largest |v| of each window over all channels; two zero pads past the end.  And
// whether a sample is not finite or above kSafeV.
__global__ void k_window_vmax(const float *__restrict__ v, u32 n, u32 C, u32 L, u32 W, float *__restrict__ vwmax,
                              u32 *__restrict__ no_bounds) {
    const u32 lane = threadIdx.x & 31;
    const u32 nwarps = (gridDim.x * blockDim.x) >> 5;
    for (u32 w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < W + 2; w += nwarps) {
        u32 m = 0;                                   // as bits: in the order of the values, NaN above all
        if (w < W) {
            for (u32 c = 0; c < C; c++) {
                const float *vc = v + (size_t)c * n + (size_t)w * L;
                for (u32 i = lane; i < L; i += 32)
                    if ((size_t)w * L + i < n) m = max(m, __float_as_uint(vc[i]) & 0x7fffffffu);
            }
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) {
            vwmax[w] = __uint_as_float(min(m, 0x7f800000u));
            if (m > __float_as_uint(kSafeV)) *no_bounds = 1;
        }
    }
}

// The groups' window lists and streams of a pass: a group's windows are those
// listed (active) with the group's dirty bit set.  Two launches over (tile of
// kCompactTile windows, group): counts of windows and of runs of consecutive
// windows, then the lists with their stream positions, the first window of
// every tile of the stream (the one whose stretch of positions holds the
// tile's start: a window's own L, and after the last window of a run L - 1
// more), and the totals.
__device__ __forceinline__ u32 tcw_selected(const u8 *__restrict__ active, const u32 *__restrict__ dirty, u32 GW, u32 g,
                                            u32 W, u32 w) {
    return w < W && active[w] && ((dirty[(size_t)w * GW + (g >> 5)] >> (g & 31)) & 1u) ? 1u : 0u;
}
// this thread's kCompactPerThread windows and their two neighbours: bit k + 1
// is window base + k
__device__ __forceinline__ u32 tcw_selection(const u8 *active, const u32 *dirty, u32 GW, u32 g, u32 W, u32 base) {
    u32 m = base > 0 ? tcw_selected(active, dirty, GW, g, W, base - 1) : 0u;
#pragma unroll
    for (u32 k = 0; k <= kCompactPerThread; k++) m |= tcw_selected(active, dirty, GW, g, W, base + k) << (k + 1);
    return m;
}
static_assert(kCompactPerThread + 2 <= 32, "a thread's windows and neighbours fit a word");
__device__ __forceinline__ u32 tcw_counts(u32 m) {   // windows, runs started << 16
    const u32 own = (m >> 1) & ((1u << kCompactPerThread) - 1u), prev = m & ((1u << kCompactPerThread) - 1u);
    return __popc(own) | (__popc(own & ~prev) << 16);
}
__global__ void __launch_bounds__(kCompactThreads)
k_tcw_count(const u8 *__restrict__ active, const u32 *__restrict__ dirty, u32 GW, u32 W, u32 *__restrict__ counts,
            Counters *cnt) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {   // the pass's refinement list
        cnt->tc_refseg = 0;
        cnt->tc_overflow = 0;                        // set by the tiles when the list overflows
    }
    const u32 g = blockIdx.y, base = blockIdx.x * kCompactTile + threadIdx.x * kCompactPerThread;
    u32 tot;
    block_excl_scan(tcw_counts(tcw_selection(active, dirty, GW, g, W, base)), &tot);
    if (threadIdx.x == 0) counts[(size_t)g * gridDim.x + blockIdx.x] = tot;
}
__global__ void __launch_bounds__(kCompactThreads)
k_tcw_lists(const u8 *__restrict__ active, const u32 *__restrict__ dirty, u32 GW, u32 W, u32 L,
            const u32 *__restrict__ counts, u32 wstride, u32 fstride, u32 *__restrict__ win, u32 *__restrict__ pos,
            u32 *__restrict__ first, u32 *__restrict__ n_win, u32 *__restrict__ n_stiles) {
    const u32 g = blockIdx.y, base = blockIdx.x * kCompactTile + threadIdx.x * kCompactPerThread;
    // windows and runs of the tiles before this one
    u32 bm = 0, br = 0, tot;
    for (u32 t = threadIdx.x; t < blockIdx.x; t += blockDim.x) {
        const u32 c = counts[(size_t)g * gridDim.x + t];
        bm += c & 0xffffu;
        br += c >> 16;
    }
    block_excl_scan(bm, &tot);
    bm = tot;
    __syncthreads();
    block_excl_scan(br, &tot);
    br = tot;
    __syncthreads();
    const u32 sel = tcw_selection(active, dirty, GW, g, W, base);
    const u32 before = block_excl_scan(tcw_counts(sel), &tot);
    u32 i = bm + (before & 0xffffu), runs = br + (before >> 16);
    u32 *gw = win + (size_t)g * wstride, *gp = pos + (size_t)g * wstride, *gf = first + (size_t)g * fstride;
#pragma unroll
    for (u32 k = 0; k < kCompactPerThread; k++) {
        if (!((sel >> (k + 1)) & 1u)) continue;
        if (!((sel >> k) & 1u)) runs++;
        const u32 p = i * L + (runs - 1) * (L - 1);
        gw[i] = base + k;
        gp[i] = p;
        const u32 nxt = p + L + (((sel >> (k + 2)) & 1u) ? 0u : L - 1);
        const u32 qt = (p + kWPos - 1) / kWPos;      // the one tile start that [p, nxt) can hold
        if (qt * kWPos < nxt) gf[qt] = i;
        i++;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        const u32 m = bm + (tot & 0xffffu), r = br + (tot >> 16);
        n_win[g] = m;
        n_stiles[g] = m ? ((m - 1) * L + (r - 1) * (L - 1) + L + kWPos - 1) / kWPos : 0u;
    }
}

}  // namespace fbp
