// Grouped expert SwiGLU for two and more tokens on the tensor cores (core: pb_hmma.cuh).
//
// The router lists the distinct selected experts in groups of up to eight or twelve of their (token, slot) entries (pb_route_lists; which: expert_many in pb_engine.cu);
// the shared expert adds groups of as many tokens.  Unit of work: eight rows of gate and the same eight rows of up of one group (GU: the two halves of one mma
// tile, so a lane ends up with both products and forms the hidden value itself), or sixteen output rows (DOWN).  The units, ordered by group, are
// cut into runs of equal cost, one per CTA (one CTA of sixteen warps per SM; with runs of as many units the CTAs that got the shared expert's full
// groups ended 20 to 30 % after the mean); inside a CTA the warps take the units of a run in turn.  The CTA first
// prepares the activations of as many groups as its shared memory holds (one token per warp), then runs their units without any
// further barrier; a run that spans more groups repeats this.  An expert of several groups streams its weights again, from L2.
//
// What bounds it: for a few entries per expert the weight stream, beyond that the decode (about two instructions per weight).  An earlier
// form split the contraction over the warps and added the partial sums in shared memory behind a barrier per 32 rows: the barrier kept the issue slots
// 44 % busy (143 / 77 us for gate-up / down at 32 tokens of the 2048 x 512 x 512-expert block, the dp4a kernels 132 / 105).
// Now 512 experts of 2048 x 512: 67 / 38 us at 32 tokens, 134 / 76 at 128, 216 / 120 at 256 (the mean CTA; dp4a 132 / 105 at 32).  The form of three
// n-tiles spills a few registers of 128, that of two none to speak of: one kernel for both made the decode of 10 Q4_K sequences 8 % longer.
// Replaces the reference's k_xgu* / k_xdown* (src/model/qn_cube.rs:3482-5419) for several tokens.
#include "pb_hmma.cuh"
#include "pb_internal.h"

#include <stdio.h>

#define MH_WARPS 16
#define MH_THREADS (MH_WARPS * 32)
#define MH_MAXV 32          // groups of one phase
#define MH_STAGES 3         // weight stages of a warp: two blocks on their way while one is used
#define MH_HEAD (MH_MAXV * 16 + 512)

// NT: n-tiles of four entries a group holds at most
template <int FMT, bool DOWN, int NT>
__global__ void __launch_bounds__(MH_THREADS, 1) pb_moeh_kernel(const PbExpertParams p, const PbHGeom h) {
    extern __shared__ __align__(128) uint8_t smem[];
    int4* vtab = reinterpret_cast<int4*>(smem);                        // [MH_MAXV] {expert or -1 (shared), first entry / token, entries, first slot}
    int* stok = reinterpret_cast<int*>(smem + MH_MAXV * 16);           // [slots] group of the slot
    __shared__ int nphase, nslots_used, bound[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const uint32_t ring = pb_smem_u32(smem + MH_HEAD) + (uint32_t)(warp * MH_STAGES * h.stage_bytes);
    uint8_t* act = smem + MH_HEAD + (size_t)MH_WARPS * MH_STAGES * h.stage_bytes;
    const int bpr = p.bpr, cols = 256 * bpr;
    const uint32_t tokb = (uint32_t)pb_h_tok_bytes<FMT>(cols);
    constexpr int VG = 4 * NT;
    const PbQTabs T = {0u, 0u, 0u};
    pb_pdl_trigger();
    pb_pdl_wait();          // lists, activations / hidden vectors come from earlier kernels
    const int nv = *p.n_virt, nsh = p.has_shared ? (p.sh_ntok + VG - 1) / VG : 0;
    const int upg = p.rows_e / (DOWN ? 16 : 8);                          // units per group
    // the CTA's run: the cost in front of a group stands in its list entry; the thread whose group holds a boundary finds its unit
    if (tid < 2) bound[tid] = (nv + nsh) * upg;
    const int4 lv = nv > 0 ? p.virt[nv - 1] : make_int4(0, 0, 0, 0);
    const int croute = lv.w + pb_vgroup_cost(lv.z), zlast = p.sh_ntok - (nsh - 1) * VG;
    const int64_t total = ((int64_t)croute + (nsh > 0 ? (nsh - 1) * pb_vgroup_cost(VG) + pb_vgroup_cost(zlast) : 0)) * upg;
    const int64_t at0 = total * blockIdx.x / gridDim.x, at1 = total * (blockIdx.x + 1) / gridDim.x;
    __syncthreads();
    for (int v = tid; v < nv + nsh; v += MH_THREADS) {
        const int4 e = v < nv ? p.virt[v] : make_int4(0, 0, v == nv + nsh - 1 ? zlast : VG, croute + (v - nv) * pb_vgroup_cost(VG));
        const int c = pb_vgroup_cost(e.z);
        const int64_t lo = (int64_t)e.w * upg, hi = lo + (int64_t)c * upg;
        if (at0 >= lo && at0 < hi) bound[0] = v * upg + (int)(at0 - lo) / c;
        if (at1 >= lo && at1 < hi) bound[1] = v * upg + (int)(at1 - lo) / c;
    }
    __syncthreads();
    const int u1 = bound[1];
    int u0 = bound[0];
    while (u0 < u1) {
        // ---- groups of this phase: as many as the slots hold
        const int v0 = u0 / upg;
        if (warp == 0) {
            const int v = v0 + lane;
            int4 e = make_int4(-1, 0, 0, 0);
            if (v <= (u1 - 1) / upg) {
                if (v < nv) {
                    e = p.virt[v];
                    if (e.x < 0 || e.x >= p.n_exp || e.y < 0 || e.z < 1 || e.z > VG || e.y + e.z > p.t * p.top_k) { atomicExch(p.status, PB_DEV_BAD_INDEX); e = make_int4(-1, 0, 0, 0); }
                } else { const int t0 = (v - nv) * VG; e = make_int4(-1, t0, min(VG, p.sh_ntok - t0), 0); }
            }
            int s = e.z, incl = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int a = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += a; }
            e.w = incl - s;
            const bool in = v <= (u1 - 1) / upg && incl - s + ((s + 3) & ~3) <= p.nslots;   // the columns past a group's entries read the slots behind it (and are dropped)
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int n = m == 0xffffffffu ? 32 : __ffs(~m) - 1;         // leading groups that fit (at least one: nslots >= VG)
            vtab[lane] = e;
            if (lane < n) for (int i = 0; i < s; i++) stok[e.w + i] = lane;
            if (lane == n - 1) { nphase = n; nslots_used = incl; }
        }
        __syncthreads();
        const int ue = min(u1, (v0 + nphase) * upg);
        // ---- weights: warp w takes units u0 + w, u0 + w + 16, ..; its blocks go round the ring of stages
        PbHTile pt; pt.la = pt.lb = 7;
        int pu = u0 + warp, pblk = 0, ps = 0;
        auto issue = [&]() {
            if (pu < ue) {
                if (pblk == 0) {
                    const int vi = pu / upg - v0, j = pu - (v0 + vi) * upg, ex = vtab[vi].x;
                    const size_t off = ex < 0 ? 0 : (size_t)(ex - p.e_base) * p.rows_e * p.row_bytes;
                    const uint8_t* a = (ex < 0 ? p.sh_a : p.w_a) + off;
                    if (DOWN) { pt.a = a + (size_t)(16 * j) * p.row_bytes; pt.b = pt.a + 8 * (size_t)p.row_bytes; }
                    else { pt.a = a + (size_t)(8 * j) * p.row_bytes; pt.b = (ex < 0 ? p.sh_b : p.w_b) + off + (size_t)(8 * j) * p.row_bytes; }
                }
                pb_h_stage<FMT>(ring + (uint32_t)(ps * h.stage_bytes), pt, h, pblk, lane);
                if (++pblk == bpr) { pblk = 0; pu += MH_WARPS; }
            } else asm volatile("cp.async.commit_group;" ::: "memory");
            ps = ps + 1 == MH_STAGES ? 0 : ps + 1;
        };
#pragma unroll
        for (int i = 0; i < MH_STAGES - 1; i++) issue();
        // ---- activations of the phase's tokens, a block of a token per warp
        const int c0 = pb_h_c0<FMT>(lane), c1 = pb_h_c1<FMT>(lane);
#pragma unroll 2
        for (int i = warp; i < nslots_used * bpr; i += MH_WARPS) {
            const int sl = i / bpr, blk = i - sl * bpr;
            const int4 e = vtab[stok[sl]];
            const int k = sl - e.w;
            const float* src; float sc = 1.0f; bool norm = false;
            if (DOWN) src = (e.x < 0 ? p.h_sh + (size_t)(p.sh_tok0 + e.y + k) * cols : p.h + (size_t)(e.y + k) * cols) + 256 * blk;
            else {
                int tok = e.x < 0 ? p.sh_tok0 + e.y + k : p.ent_tok[e.y + k];
                if (tok < 0 || tok >= p.t) { atomicExch(p.status, PB_DEV_BAD_INDEX); tok = 0; }
                src = p.x + (size_t)tok * p.ldx + 256 * blk;
                norm = p.norm_w != nullptr;
                if (norm) sc = p.tok_scale[tok];
            }
            const float4 a = *reinterpret_cast<const float4*>(src + c0), b = *reinterpret_cast<const float4*>(src + c1);
            float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            if (norm) {
                const float4 na = *reinterpret_cast<const float4*>(p.norm_w + 256 * blk + c0), nb = *reinterpret_cast<const float4*>(p.norm_w + 256 * blk + c1);
                const float n[8] = {na.x, na.y, na.z, na.w, nb.x, nb.y, nb.z, nb.w};
#pragma unroll
                for (int c = 0; c < 8; c++) x[c] = x[c] * sc * n[c];
            }
            pb_h_put<FMT>(act + (size_t)sl * tokb, bpr, blk, lane, x);
        }
        __syncthreads();
        int cs = 0;
        for (int u = u0 + warp; u < ue; u += MH_WARPS) {
            const int vi = u / upg - v0, j = u - (v0 + vi) * upg;
            const int4 e = vtab[vi];
            const PbHLane L = pb_h_lane<FMT>(pb_smem_u32(act) + (uint32_t)e.w * tokb, bpr, lane);
            float tot[NT][2];
#pragma unroll
            for (int nt = 0; nt < NT; nt++) tot[nt][0] = tot[nt][1] = 0.f;
            for (int blk = 0; blk < bpr; blk++) {
                asm volatile("cp.async.wait_group %0;" ::"n"(MH_STAGES - 2) : "memory");
                __syncwarp();   // this block has landed for all lanes, and all have left the stage that is refilled now
                issue();
                const uint32_t st = ring + (uint32_t)(cs * h.stage_bytes);
                if (e.z <= 4) pb_h_block<FMT, 1>(st, pt, h, T, blk, blk, lane, L, reinterpret_cast<float (&)[1][2]>(tot));
                else if (NT == 2 || e.z <= 8) pb_h_block<FMT, 2>(st, pt, h, T, blk, blk, lane, L, reinterpret_cast<float (&)[2][2]>(tot));
                else pb_h_block<FMT, NT>(st, pt, h, T, blk, blk, lane, L, tot);
                cs = cs + 1 == MH_STAGES ? 0 : cs + 1;
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const int k = 4 * nt + q;
                if (k < e.z) {
                    const float a = tot[nt][0], b = tot[nt][1];
                    if (!DOWN) {
                        // hidden = silu(gate . x) * (up . x)   (routed :1781-1783, ffn :1680)
                        float* dst = e.x < 0 ? p.h_sh + (size_t)(p.sh_tok0 + e.y + k) * p.rows_e : p.h + (size_t)(e.y + k) * p.rows_e;
                        dst[8 * j + g] = pb_silu(a) * b;
                    } else if (e.x < 0) {
                        float* dst = p.part_sh + (size_t)(p.sh_tok0 + e.y + k) * p.rows_e + 16 * j + g;
                        dst[0] = a; dst[8] = b;
                    } else {
                        const int en = e.y + k, tok = p.ent_tok[en], slt = p.ent_slot[en];
                        const float w = p.ent_w[en];
                        float* dst = (p.part_tok ? p.part_tok[tok] + (size_t)slt * p.rows_e : p.part + ((size_t)tok * p.top_k + slt) * p.rows_e) + 16 * j + g;
                        dst[0] = w * a; dst[8] = w * b;   // routed :1786: o += w * dot
                    }
                }
            }
        }
        u0 = ue;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // the tables and slots are rewritten by the next phase
    }
}

// Shapes the kernels take: whole 256-column blocks, rows in whole units, and the formats whose weights the lanes load themselves
bool pb_moeh_supported(int type, int d, int ff, int t) {
    return t >= 2 && (type == PB_T_IQ3S_N4 || type == PB_T_Q4_K) && d % 256 == 0 && ff % 256 == 0 && d <= 2048 && ff <= 2048;   // eight tokens of 2048 columns fit beside the weight stages
}

template <int FMT, bool DOWN, int NT>
static int launch_moeh(pb_ctx* ctx, PbExpertParams p, int cols) {
    int el, bs;
    pb_geom(FMT, &el, &bs);
    p.bpr = cols / 256; p.row_bytes = cols / el * bs;
    const PbHGeom h = pb_h_geom<FMT>(cols);
    const size_t fixed = MH_HEAD + (size_t)MH_WARPS * MH_STAGES * h.stage_bytes, tokb = pb_h_tok_bytes<FMT>(cols);
    int ns = (int)(((size_t)ctx->max_smem_optin - 256 - fixed) / tokb);
    p.nslots = ns > 96 ? 96 : ns;
    if (p.nslots < 4 * NT) PB_FAIL(ctx, PB_UNSUPPORTED, "expert kernel: %zu bytes per token", tokb);
    const size_t smem = fixed + (size_t)p.nslots * tokb;
    p.status = ctx->dev_status;
    auto kern = pb_moeh_kernel<FMT, DOWN, NT>;
    PB_TRY(pb_ensure_smem(ctx, kern, smem));
    pb_launch_k(ctx, kern, dim3(ctx->sm_count), dim3(MH_THREADS), smem, p, h);
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    return PB_OK;
}

template <bool DOWN>
static int launch_moeh_g(pb_ctx* ctx, const PbExpertParams& p, int type, int cols) {
    if (type == PB_T_Q4_K) return p.vgroup == PB_VGROUP ? launch_moeh<PB_T_Q4_K, DOWN, 2>(ctx, p, cols) : launch_moeh<PB_T_Q4_K, DOWN, 3>(ctx, p, cols);
    return p.vgroup == PB_VGROUP ? launch_moeh<PB_T_IQ3S_N4, DOWN, 2>(ctx, p, cols) : launch_moeh<PB_T_IQ3S_N4, DOWN, 3>(ctx, p, cols);
}
int pb_launch_moeh_gu(pb_ctx* ctx, const PbExpertParams& p, int type, int cols) { return launch_moeh_g<false>(ctx, p, type, cols); }
int pb_launch_moeh_down(pb_ctx* ctx, const PbExpertParams& p, int type, int cols) { return launch_moeh_g<true>(ctx, p, type, cols); }
