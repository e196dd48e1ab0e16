// Batched dequant-GEMM for 2 .. 16 (small matrices 32) activation columns a launch on the tensor cores, every quantized format (core: pb_hmma.cuh).  (Two columns of a
// small matrix in a format with a long decode stay on the dp4a kernel: pb_gemvq.cu.)
//
//   y[b][yoff_s + r] (+)= sum_c W_s[r][c] * act(x)[b][c]        b = 0 .. t-1
//
// Used where one weight matrix meets several tokens at once (batched decode, verify windows): the weights are streamed and decoded ONCE for
// all columns, instead of once per column as in the dp4a GEMV.  Persistent CTAs, one per SM; the 16-row tiles of all segments are dealt to the
// CTAs in contiguous runs.  A CTA prepares the activations (none / RMSNorm / per-head gated norm, f16 high + low parts) in its shared memory
// while its warps already load their first weights, then every warp takes whole tiles on its own: no barrier in the loop.  What is left of
// a run after whole rounds of one tile per warp -- or all of a small matrix -- is cut along the contraction: 2, 4, .. warps share a tile, each
// takes a run of its blocks, and their sums meet in shared memory.  Without that cut a 12352-row matrix keeps a third of the warps busy, and a
// 151936-row one (64.2 tiles per CTA) waits a fifth of its time for the last round.
// Rows of 4096 columns, and rows of 2048 where a CTA has at most a round of tiles and the tokens are more than four, are cut along the contraction
// over a cluster of CTAs as well: each prepares
// and keeps only its part of the activations (the preparation of 8 tokens x 4096 columns in every CTA took longer than the product: 23 us a
// launch against 7), and the parts' sums are read from the partners' shared memory, in rank order.
// Replaces the reference's batched GEMV / prefill GEMM (k_gemv4*, k_gemm_pf / k_gemm_tc, src/model/qn_cube.rs:71-233, 293-1159).
#include "pb_hmma.cuh"
#include "pb_internal.h"

#include <stdio.h>
#include <stdlib.h>

#define GH_WARPS 16
#define GH_MAXBLK 16         // blocks of 256 columns per row at most
#define GH_MAXNT 8           // n-tiles of four tokens at most
#define GH_HEAD (4 * GH_MAXNT * GH_MAXBLK * 4)   // bytes in front of the tables: partial sums of squares [tokens][blocks]

struct PbGemmHParams {
    PbGemvQParams q;         // seg[].chunk0 = first 16-row tile of the segment, nchunks = tiles in all
    PbHGeom g;
    int stages;              // weight stages of a warp
    int ks;                  // CTAs of a cluster; each takes bpr / ks blocks of every row
    uint32_t off_act, off_red, off_stage;
};

__device__ __forceinline__ void gh_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float gh_remote(uint32_t saddr, int rank) {
    uint32_t a; float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

template <int FMT, int NT>
__global__ void __launch_bounds__(GH_WARPS * 32, 1) pb_gemmh_kernel(const PbGemmHParams h) {
    const PbGemvQParams& p = h.q;
    extern __shared__ __align__(128) uint8_t smem[];
    float* ssq = reinterpret_cast<float*>(smem);
    uint8_t* tab = smem + GH_HEAD;
    uint8_t* act = smem + h.off_act;
    float* red = reinterpret_cast<float*>(smem + h.off_red);          // [GH_WARPS][4 NT tokens][16 rows]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, nw = (int)blockDim.x >> 5;
    const int ks = h.ks, rank = ks > 1 ? (int)blockIdx.x % ks : 0, cl = (int)blockIdx.x / ks, ncl = (int)gridDim.x / ks;   // (clusters are consecutive CTAs)
    const int bpr = p.bpr / ks, kb = rank * bpr;                       // this CTA's blocks of a row: kb .. kb + bpr
    const uint32_t tokb = (uint32_t)pb_h_tok_bytes<FMT>(256 * bpr);
    pb_pdl_trigger();
    const int tile0 = (int)((int64_t)p.nchunks * cl / ncl), tile1 = (int)((int64_t)p.nchunks * (cl + 1) / ncl);
    // whole rounds: every warp a tile; then one round of `share` warps per tile
    const int rounds = (tile1 - tile0) / nw, nfull = rounds * nw, nrest = tile1 - tile0 - nfull;
    int share = 1;
    while (nrest > 0 && 2 * share <= bpr && 2 * share * nrest <= nw) share *= 2;
    const int pieces = rounds + (nrest > 0 ? 1 : 0);
    // piece i of this warp: its tile (-1: none) and blocks [b0, b1)
    auto piece = [&](int i, int& b0, int& b1) -> int {
        if (i < rounds) { b0 = 0; b1 = bpr; return tile0 + i * nw + warp; }
        const int k = warp / share, part = warp - k * share;
        b0 = part * (bpr / share); b1 = b0 + bpr / share;
        return k < nrest ? tile0 + nfull + k : -1;
    };
    auto locate = [&](int tile, int& r0) -> int { int s = 0; while (s + 1 < p.nseg && tile >= p.seg[s + 1].chunk0) s++; r0 = (tile - p.seg[s].chunk0) * 16; return s; };

    // ---- weights: the blocks of the warp's pieces go round its ring of stages; the first are requested before anything of the previous
    //      kernel is awaited
    const uint32_t ring = pb_smem_u32(smem + h.off_stage) + (uint32_t)(warp * h.stages * h.g.stage_bytes);
    PbHTile pt; pt.a = pt.b = nullptr; pt.la = pt.lb = 7;
    int pi = 0, pb0 = 0, pb1 = 0, ptile = -1, pblk = 0, ps = 0;
    auto tile_of = [&](int tile, PbHTile& t) {
        int r0;
        const int s = locate(tile, r0), rows = p.seg[s].rows;
        const uint8_t* w = p.seg[s].w + (size_t)r0 * p.row_bytes;
        t.a = w; t.la = min(7, rows - 1 - r0);
        const bool two = r0 + 8 < rows;                                // (else the second half repeats the first and is not stored)
        t.b = two ? w + 8 * (size_t)p.row_bytes : w; t.lb = two ? min(7, rows - 9 - r0) : t.la;
    };
    auto open = [&]() { ptile = pi < pieces ? piece(pi, pb0, pb1) : -1; if (ptile >= 0) { tile_of(ptile, pt); pblk = pb0; } };
    auto issue = [&]() {
        if (ptile >= 0) {
            pb_h_stage<FMT>(ring + (uint32_t)(ps * h.g.stage_bytes), pt, h.g, kb + pblk, lane);
            if (++pblk == pb1) { pi++; open(); }
        } else asm volatile("cp.async.commit_group;" ::: "memory");
        ps = ps + 1 == h.stages ? 0 : ps + 1;
    };
    open();
    for (int i = 0; i + 1 < h.stages; i++) issue();
    PbQTabs T = {0u, 0u, 0u};
    if constexpr (pb_h_mode<FMT>() != PB_H_DIRECT) T = pb_h_fill_tabs<FMT>(tab, p.rep, tid, (int)blockDim.x, lane);

    // ---- activations: a block of a token per warp
    pb_pdl_wait();
    const int c0 = pb_h_c0<FMT>(lane), c1 = pb_h_c1<FMT>(lane);
    if (p.mode == PB_ACT_NORM) {
        for (int i = warp; i < p.t * p.bpr; i += nw) {
            const int b = i / p.bpr, blk = i - b * p.bpr;
            const float* x = p.x + (size_t)b * p.ldx + 256 * blk;
            const float4 u = *reinterpret_cast<const float4*>(x + 4 * lane), v = *reinterpret_cast<const float4*>(x + 128 + 4 * lane);
            const float ss = pb_warp_sum((u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w) + (v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w));
            if (lane == 0) ssq[b * GH_MAXBLK + blk] = ss;
        }
        __syncthreads();
    }
#pragma unroll 2
    for (int i = warp; i < p.t * bpr; i += nw) {
        const int b = i / bpr, blk = i - b * bpr;
        const int col = 256 * (kb + blk);
        const float* x = p.x + (size_t)b * p.ldx + col;
        const float4 u = *reinterpret_cast<const float4*>(x + c0), v = *reinterpret_cast<const float4*>(x + c1);
        float a[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
        if (p.mode == PB_ACT_NORM) {          // rms(): x * s * w  (qwen4exp_gguf.rs:209)
            float ss = 0.f;
            for (int k = 0; k < p.bpr; k++) ss += ssq[b * GH_MAXBLK + k];
            const float s = 1.0f / sqrtf(ss / (float)(256 * p.bpr) + p.eps);
            const float4 n0 = *reinterpret_cast<const float4*>(p.norm_w + col + c0), n1 = *reinterpret_cast<const float4*>(p.norm_w + col + c1);
            const float n[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
            for (int c = 0; c < 8; c++) a[c] = a[c] * s * n[c];
        } else if (p.mode == PB_ACT_GNORM) {  // per head of 128 (two quarters): rms(x) * w * sigmoid(z)  (linear_core, qwen4exp_gguf.rs:1667)
            const float* z = p.z + (size_t)b * p.ldz + col;
            const float4 z0 = *reinterpret_cast<const float4*>(z + c0), z1 = *reinterpret_cast<const float4*>(z + c1);
            float ss = 0.f;
#pragma unroll
            for (int c = 0; c < 8; c++) ss += a[c] * a[c];
            ss += __shfl_xor_sync(0xffffffffu, ss, 1); ss += __shfl_xor_sync(0xffffffffu, ss, 4); ss += __shfl_xor_sync(0xffffffffu, ss, 8); ss += __shfl_xor_sync(0xffffffffu, ss, 16);
            const float s = 1.0f / sqrtf(ss / 128.0f + p.eps);
            const float4 n0 = *reinterpret_cast<const float4*>(p.norm_w + (c0 & 127)), n1 = *reinterpret_cast<const float4*>(p.norm_w + (c1 & 127));
            const float n[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w}, zz[8] = {z0.x, z0.y, z0.z, z0.w, z1.x, z1.y, z1.z, z1.w};
#pragma unroll
            for (int c = 0; c < 8; c++) a[c] = a[c] * (s * n[c]) * pb_sigm(zz[c]);
        }
        pb_h_put<FMT>(act + (size_t)b * tokb, bpr, blk, lane, a);   // (columns past the tokens read whatever their slots hold and are dropped)
    }
    __syncthreads();

    const PbHLane L = pb_h_lane<FMT>(pb_smem_u32(act), bpr, lane);
    int cs = 0;
    for (int i = 0; i < pieces; i++) {
        int b0, b1, r0 = 0, s = 0;
        const int tile = piece(i, b0, b1);
        PbHTile ct; ct.a = ct.b = nullptr; ct.la = ct.lb = 7;
        if (tile >= 0) { s = locate(tile, r0); if constexpr (pb_h_mode<FMT>() != PB_H_DIRECT) tile_of(tile, ct); }
        float tot[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) tot[nt][0] = tot[nt][1] = 0.f;
        if (tile >= 0)
            for (int blk = b0; blk < b1; blk++) {
                if (h.stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory"); else asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncwarp();   // this block has landed for all lanes, and all have left the stage that is refilled now
                issue();
                pb_h_block<FMT, NT>(ring + (uint32_t)(cs * h.g.stage_bytes), ct, h.g, T, kb + blk, blk, lane, L, tot);
                cs = cs + 1 == h.stages ? 0 : cs + 1;
            }
        const int shr = i < rounds ? 1 : share;
        if (shr == 1 && ks == 1) {
            if (tile >= 0) {
                const int rows = p.seg[s].rows;
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    const int b = 4 * nt + q;
                    if (b < p.t) {
                        float* dst = p.y + (size_t)b * p.ldy + p.seg[s].yoff + r0 + g;
                        if (r0 + g < rows) dst[0] = p.accumulate ? dst[0] + tot[nt][0] : tot[nt][0];
                        if (r0 + 8 + g < rows) dst[8] = p.accumulate ? dst[8] + tot[nt][1] : tot[nt][1];
                    }
                }
            }
        } else {
            // the sums of a tile's parts meet in shared memory and are added in block order; a CTA of a cluster adds a share of the round's outputs
            float* mine = red + (size_t)warp * (4 * NT * 16);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) { mine[(4 * nt + q) * 16 + g] = tot[nt][0]; mine[(4 * nt + q) * 16 + g + 8] = tot[nt][1]; }
            if (ks > 1) gh_cluster_sync(); else __syncthreads();
            const int first = tile0 + i * nw, nout = (i < rounds ? nw : nrest) * 16 * p.t;
            for (int o = nout * rank / ks + tid; o < nout * (rank + 1) / ks; o += (int)blockDim.x) {
                const int k = o / (16 * p.t), e = o - k * 16 * p.t, b = e >> 4, r = e & 15;
                int rr;
                const int sg = locate(first + k, rr);
                if (rr + r >= p.seg[sg].rows) continue;
                const uint32_t src = pb_smem_u32(red) + (uint32_t)((k * shr * (4 * NT * 16) + b * 16 + r) * 4);
                float v = 0.f;
                for (int c = 0; c < ks; c++)
                    for (int w = 0; w < shr; w++) v += ks > 1 ? gh_remote(src + (uint32_t)(w * 4 * NT * 16 * 4), c) : red[(size_t)(k * shr + w) * (4 * NT * 16) + b * 16 + r];
                float* dst = p.y + (size_t)b * p.ldy + p.seg[sg].yoff + rr + r;
                *dst = p.accumulate ? *dst + v : v;
            }
            if (ks > 1) gh_cluster_sync(); else if (i + 1 < pieces) __syncthreads();   // the buffer is rewritten (or, at the end, given up) only when all have read it
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Tokens of one launch and warps per CTA that fit shared memory
template <int FMT>
static bool gh_layout(pb_ctx* ctx, int cols, int t, int ks, int& nt, int& nw, PbGemmHParams& h, size_t& smem) {
    constexpr int rep = pb_tab_rep_max<FMT>();
    h.g = pb_h_geom<FMT>(cols);
    for (nt = t > 4 * GH_MAXNT ? GH_MAXNT : ((t + 3) / 4 > 4 ? ((t + 3) / 4 + 1) & ~1 : (t + 3) / 4); nt >= 1; nt -= nt > 4 ? 2 : 1)   // (forms are built for 1, 2, 3, 4, 6 and 8)
        for (nw = GH_WARPS; nw >= 8; nw /= 2)
            for (h.stages = 3; h.stages >= 2; h.stages--)
                for (h.q.rep = rep > 8 ? 8 : rep; h.q.rep >= 1; h.q.rep /= 2) {   // copies of the codebook: as many as fit
                    const uint32_t tabb = pb_h_tab_bytes<FMT>(h.q.rep);
                    h.off_act = GH_HEAD + ((tabb + 127) & ~127u);
                    h.off_red = h.off_act + (uint32_t)(4 * nt) * (uint32_t)pb_h_tok_bytes<FMT>(cols / ks);
                    h.off_stage = h.off_red + (uint32_t)nw * 4 * nt * 16 * 4;
                    smem = h.off_stage + (size_t)nw * h.stages * h.g.stage_bytes + 64;   // the decoders read whole words: a few bytes past the last row
                    if (smem <= (size_t)ctx->max_smem_optin) return true;
                }
    return false;
}

template <int FMT>
static const void* gh_kernel(int nt) {
    const void* k[] = {(const void*)pb_gemmh_kernel<FMT, 1>, (const void*)pb_gemmh_kernel<FMT, 2>, (const void*)pb_gemmh_kernel<FMT, 3>, (const void*)pb_gemmh_kernel<FMT, 4>, (const void*)pb_gemmh_kernel<FMT, 6>, (const void*)pb_gemmh_kernel<FMT, 8>};
    return k[nt <= 4 ? nt - 1 : nt / 2 + 1];
}
// Tiles of a round: one per warp of every cluster that is resident at a time (148 SMs hold 74 clusters of two CTAs, but 33 of four and 15 of eight)
template <int FMT>
static int gh_round(pb_ctx* ctx, int nt, int nw, size_t smem, int ks, int* tiles) {
    PB_TRY(pb_ensure_smem_fn(ctx, gh_kernel<FMT>(nt), smem));
    *tiles = nw * pb_max_clusters(ctx, gh_kernel<FMT>(nt), nw * 32, smem, ks);
    return PB_OK;
}

// Whether r tokens, 17 to 32, go in one launch, on clusters of ks32 CTAs of 512 columns (32 tokens' activations fit beside the weights), or in launches of
// sixteen.  One launch is the shorter one for every format, 17 to 31 tokens and 512 to 4096 columns while a CTA has at most one round of tiles (us, two launches /
// one, 24 tokens: 2048 x 512 IQ3_S 12.3 / 9.9, 4096 x 2048 20.5 / 15.7, 8448 x 2048 24.2 / 18.5, Q6_K 39.0 / 27.1, 3584 x 4096 IQ2_XS 34.8 / 24.6;
// 31 tokens: 8448 x 2048 IQ3_S 26.7 / 22.6, Q5_K 45.0 / 33.2), where the round counts the warps that fit: Q8_0 has eight with 25 and more tokens (31 tokens of
// 4096 x 2048, 0.97 rounds, 28.7 / 24.6; of 4096 x 4096, 2.1 rounds, 41.0 / 51.2).  With more, the parts' sums are exchanged in every round.  A little more than a
// round still pays where two launches have no second warp for a tile (4608 x 4096 24 tokens: Q4_K 32.9 / 28.9, Q6_K 51.2 / 38.7), for the formats of the
// longest decodes (31 tokens of 4096 x 4096 IQ3_XXS 47.2 / 43.2, 9472 x 2048 IQ1_M 45.4 / 41.0), for 18 to 24 tokens (9472 x 2048 Q8_0 36.9 / 32.8) except
// for short decodes in clusters of eight (4096 x 4096, 20 tokens: IQ3_S 23.8 / 24.6, Q4_K 26.9 / 28.7), and from 29 on but for the two shortest (31 tokens of
// 9472 x 2048 Q6_K 45.1 / 42.9, IQ3_S 27.7 / 28.7); not for a single seventeenth token, which the dp4a kernel takes (9472 x 2048 Q4_0 28.7 / 30.8), nor
// for 25 to 28 (25 tokens of 4096 x 4096 Q4_0 36.9 / 39.0).  Several rounds are shorter in two launches (24 tokens of 151936 x 2048 IQ3_S 138 / 221); at one and a
// half the formats differ (12351 x 2048, 17 tokens IQ3_S 24.6 / 26.7, Q4_K 30.8 / 30.7; 24 tokens IQ3_S 26.9 / 26.7, IQ2_XS 41.0 / 32.8, Q8_0 47.2 / 38.9; 25
// tokens IQ3_S 28.7 / 32.7, Q8_0 49.2 / 57.4, IQ3_XXS 55.3 / 49.2) and two launches are kept for all.
template <int FMT>
static int gh_one_launch(pb_ctx* ctx, int cols, int all, int r, int ks16, int ks32, bool* one) {
    *one = false;
    if (all > GH_WARPS * (ctx->sm_count / ks32)) return PB_OK;
    PbGemmHParams h;
    int nt, nw, nt16, nw16, round, round16; size_t smem, smem16;
    memset(&h, 0, sizeof h);
    if (!gh_layout<FMT>(ctx, cols, r, ks32, nt, nw, h, smem) || nt <= 4) return PB_OK;
    PB_TRY((gh_round<FMT>(ctx, nt, nw, smem, ks32, &round)));
    if (all <= round) { *one = true; return PB_OK; }
    if (4 * all > 5 * round || !gh_layout<FMT>(ctx, cols, 16, ks16, nt16, nw16, h, smem16)) return PB_OK;
    PB_TRY((gh_round<FMT>(ctx, nt16, nw16, smem16, ks16, &round16)));
    constexpr bool longest = FMT == PB_T_IQ3_XXS || FMT == PB_T_IQ2_XXS || FMT == PB_T_IQ1_M || FMT == PB_T_IQ2_XS;
    constexpr bool brief = FMT == PB_T_IQ3S_N4 || FMT == PB_T_Q4_K || FMT == PB_T_IQ2_S;
    *one = 2 * all > round16 || longest || (nt <= 6 ? r > 17 && !(brief && ks32 == 8) : r > 28 && nw == GH_WARPS && (!brief || FMT == PB_T_Q4_K));
    return PB_OK;
}

// CTAs of a cluster.  Launches of up to sixteen tokens: 1024 columns each above 2048; half a row each where a CTA has at most a round of tiles and the
// activations of several tokens would take as long to prepare as the product
static int gh_ks16(pb_ctx* ctx, int cols, int all, int t) { return cols > 2048 ? cols / 1024 : (cols == 2048 && all <= 16 * ctx->sm_count && t > 4 ? 2 : 1); }
static int gh_ks32(int cols) { return cols > 512 ? cols / 512 : 1; }

template <int FMT>
static int launch_fmt(pb_ctx* ctx, const PbGemvQArgs& a, bool recoded) {
    int el, bs;
    pb_geom(FMT, &el, &bs);
    int all = 0;
    for (int s = 0; s < a.nseg; s++) all += (int)((a.seg[s].rows + 15) / 16);
    const int ks16 = gh_ks16(ctx, a.cols, all, a.t), ks32 = gh_ks32(a.cols);
    for (int t0 = 0, n = 0; t0 < a.t; t0 += n) {
        PbGemmHParams h;
        memset(&h, 0, sizeof h);
        int nt, nw, r = a.t - t0 < 4 * GH_MAXNT ? a.t - t0 : 4 * GH_MAXNT; size_t smem;
        bool one = true;
        if (r > 16) { PB_TRY((gh_one_launch<FMT>(ctx, a.cols, all, r, ks16, ks32, &one))); if (!one) r = 16; }
        const int ks = r > 16 ? ks32 : ks16;
        h.ks = ks;
        if (!gh_layout<FMT>(ctx, a.cols, r, ks, nt, nw, h, smem)) PB_FAIL(ctx, PB_UNSUPPORTED, "gemm: %d columns do not fit shared memory", a.cols);
        n = r < 4 * nt ? r : 4 * nt;
        PbGemvQParams& p = h.q;
        p.row_bytes = a.cols / el * bs; p.bpr = a.cols / 256; p.nseg = a.nseg;
        p.x = a.x + (int64_t)t0 * a.ldx; p.ldx = a.ldx; p.t = n; p.y = a.y + (int64_t)t0 * a.ldy; p.ldy = a.ldy; p.status = ctx->dev_status;
        p.mode = a.mode; p.norm_w = a.norm_w; p.z = a.z ? a.z + (int64_t)t0 * a.ldz : nullptr; p.ldz = a.ldz; p.head_dim = a.head_dim; p.eps = a.eps; p.accumulate = a.accumulate;
        int ntiles = 0;
        for (int s = 0; s < a.nseg; s++) {
            p.seg[s].w = recoded ? a.seg[s].wr : a.seg[s].w; p.seg[s].rows = (int)a.seg[s].rows; p.seg[s].yoff = (int)a.seg[s].yoff; p.seg[s].chunk0 = ntiles;
            ntiles += (int)((a.seg[s].rows + 15) / 16);
        }
        p.nchunks = ntiles;
        if (ntiles == 0) return PB_OK;
#define GO(N) { auto kern = pb_gemmh_kernel<FMT, N>; PB_TRY(pb_ensure_smem(ctx, kern, smem)); const int ncl = pb_max_clusters(ctx, reinterpret_cast<const void*>(kern), nw * 32, smem, ks), grid = (ntiles < ncl ? ntiles : ncl) * ks; pb_launch_kc(ctx, kern, dim3(grid), dim3(nw * 32), smem, ks, h); }
        if (nt == 1) GO(1) else if (nt == 2) GO(2) else if (nt == 3) GO(3) else if (nt == 4) GO(4) else if (nt == 6) GO(6) else GO(8)
#undef GO
        ctx->kernels_launched++;
        PB_CUDA(ctx, cudaGetLastError());
    }
    return PB_OK;
}

template <int FMT>
static int tokens_fmt(pb_ctx* ctx, int64_t rows, int cols, int t, int* n) {
    const int all = (int)((rows + 15) / 16), r = t < 4 * GH_MAXNT ? t : 4 * GH_MAXNT;
    bool one = false;
    PB_TRY((gh_one_launch<FMT>(ctx, cols, all, r, gh_ks16(ctx, cols, all, t), gh_ks32(cols), &one)));
    *n = one ? r : 16;
    return PB_OK;
}
int pb_gemmh_tokens(pb_ctx* ctx, int type, bool recoded, int64_t rows, int cols, int t, int* n) {
    static const bool use_mma = !(getenv("PYRE_B200_MMA") && atoi(getenv("PYRE_B200_MMA")) == 0);
    *n = t < 16 ? t : 16;
    if (t <= 16 || !use_mma || !pb_gemvq_supported(type, cols)) return PB_OK;
#define GO(F) case F: return tokens_fmt<F>(ctx, rows, cols, t, n)
    switch (type) {
        case PB_T_IQ3_S: return recoded ? tokens_fmt<PB_T_IQ3S_N4>(ctx, rows, cols, t, n) : tokens_fmt<PB_T_IQ3_S>(ctx, rows, cols, t, n);
        GO(PB_T_IQ3S_N4); GO(PB_T_IQ2_XS); GO(PB_T_Q4_K); GO(PB_T_Q8_0); GO(PB_T_IQ3_XXS); GO(PB_T_IQ2_S); GO(PB_T_IQ4_NL); GO(PB_T_IQ4_XS);
        GO(PB_T_Q2_0); GO(PB_T_IQ2_XXS); GO(PB_T_Q6_K); GO(PB_T_IQ1_M); GO(PB_T_Q4_0); GO(PB_T_Q5_0); GO(PB_T_Q3_K); GO(PB_T_Q5_K);
        default: return PB_OK;
    }
#undef GO
}
bool pb_gemmh_supported(int type, int cols, int t) { return t >= 2 && pb_gemvq_supported(type, cols); }

int pb_launch_gemmh(pb_ctx* ctx, const PbGemvQArgs& a) {
    if (!pb_gemmh_supported(a.type, a.cols, a.t)) PB_FAIL(ctx, PB_UNSUPPORTED, "gemm: type %d cols %d t %d", a.type, a.cols, a.t);
    if (a.nseg < 1 || a.nseg > 4) PB_FAIL(ctx, PB_ERR_ARG, "gemm: %d segments", a.nseg);
    if (a.mode == PB_ACT_PREQ) PB_FAIL(ctx, PB_UNSUPPORTED, "gemm: pre-split activations are not accepted");
    if (a.mode == PB_ACT_GNORM && a.head_dim != 128) PB_FAIL(ctx, PB_UNSUPPORTED, "gemm: gated norm over heads of %d (128 is built)", a.head_dim);
    if (((uintptr_t)a.x & 15) || (a.ldx & 3)) PB_FAIL(ctx, PB_ERR_ARG, "gemm: activations must be 16-byte aligned");
    bool recoded = a.type == PB_T_IQ3_S;   // every segment has a re-coded copy
    for (int sg = 0; sg < a.nseg; sg++) { recoded = recoded && a.seg[sg].wr != nullptr; if ((uintptr_t)a.seg[sg].w & 15) PB_FAIL(ctx, PB_ERR_ARG, "gemm: weight pointer must be 16-byte aligned"); }
#define GO(F) case F: return launch_fmt<F>(ctx, a, false)
    switch (a.type) {
        case PB_T_IQ3_S: return recoded ? launch_fmt<PB_T_IQ3S_N4>(ctx, a, true) : launch_fmt<PB_T_IQ3_S>(ctx, a, false);
        GO(PB_T_IQ3S_N4); GO(PB_T_IQ2_XS); GO(PB_T_Q4_K); GO(PB_T_Q8_0); GO(PB_T_IQ3_XXS); GO(PB_T_IQ2_S); GO(PB_T_IQ4_NL); GO(PB_T_IQ4_XS);
        GO(PB_T_Q2_0); GO(PB_T_IQ2_XXS); GO(PB_T_Q6_K); GO(PB_T_IQ1_M); GO(PB_T_Q4_0); GO(PB_T_Q5_0); GO(PB_T_Q3_K); GO(PB_T_Q5_K);
        default: PB_FAIL(ctx, PB_UNSUPPORTED, "gemm: type %d", a.type);
    }
#undef GO
}
