// Grouped expert SwiGLU of a prompt on the fifth-generation tensor cores (tcgen05), re-coded IQ3_S weights: many tokens an expert.
//
// The same sums as the warp-level kernels (pb_moeh.cu), bit for bit: weights as integers times 2^-14 in f16, activations as f16 high and low parts
// after a power of two per token and block, chains of four MMA (64 columns) into a fresh f32 accumulator, the chains added up in rounded f32, then the
// block's factor and the token's power of two.  (tcgen05.mma adds into its accumulator exactly as mma.sync does, by truncation; chains of 4 leave
// 1.4e-7 of the result against 64 bits at 2048 columns, of 16 3.1e-7, of 128 2.5e-6, on both.)
//
// Unit of work: 128 weight rows of one group of up to 24 entries -- 64 rows of gate and the same 64 of up (GU: sixteen and sixteen per warp's 32 lanes, so
// that a shuffle brings the pair together) or 128 output rows (DOWN).  The units, ordered by group, are cut into runs of equal cost, one per CTA.
// A group's activations are prepared once, as the B operand of all its units (up to 48 rows x 2048 columns), and stay in shared memory.
//
// Every role works by the half block (128 columns, two steps): one wait, one arrival per warp.
//   producer warps (3)  one per slot of the ring of raw half blocks: 16-byte asynchronous copies that also rotate a row's four quarters so that the
//                       decoders' reads do not conflict, and blocks further on into L2.  (One warp took 1000 cycles a half block and was the bound; bulk
//                       copies, one per eight rows, 2500.)
//   decoder warps (12)  one thread = one row: three groups of four warps take half blocks in turn, nine instructions per eight weights, into the slot's
//                       two A tiles in tensor memory (tcgen05.st)
//   MMA warp            one thread issues the eight MMA of a half block, its two steps in turn, each into an accumulator of its own: the MMA of a chain
//                       wait for one another, about 107 cycles each however narrow, of two chains 70.  The commit tells the decoders (A tiles free) and
//                       the drain warps (accumulators complete)
//   drain warps (8)     two per 32 lanes, half of the entries each: tcgen05.ld, sums of the chains, and the block's and the unit's ends
// By the step, with the arrivals of all lanes and indexes by division, the MMA warp's own overhead was the bound (1.3 us a half block).
//
// What bounds it: issue slots (64 % busy: per 64 columns and row about 80 of decoding, and 45 of draining for each of its two warps) and the hand-overs
// between the roles, 680 cycles a half block; the warp-level kernel decodes every weight again for each twelve entries and issues the MMA from the
// decoding warps.  1024 tokens, top 10 of 512 experts of 2048 x 512: gate / up 398 us against 514, down 223 against 269.
// Every wait is bounded; one that runs out records a status and the CTA leaves through the common exit, which frees its tensor memory.
#include "pb_tc.cuh"
#include "pb_hmma.cuh"
#include "pb_internal.h"

#include <stddef.h>
#include <stdio.h>

#define MT_DRAIN 8
#define MT_DECODE 12
#define MT_RING 3                   // half blocks under way: raw slots, pairs of A tiles, pairs of accumulators, and groups of decoder warps -- a group meets its
                                    // own slot again, so that no wait is a whole phase early
#define MT_MMA (MT_DRAIN + MT_DECODE + 3)          // behind the three producer warps
#define MT_THREADS ((MT_MMA + 1) * 32)
#define MT_GROUP PB_VGROUP_TC       // entries of a group at most
#define MT_RAW_BYTES (16 * 512 + 16 * 64)   // 16 groups of eight rows: one piece (512 bytes) and the rows' heads (64 bytes) each
#define MT_ACC (64 * MT_RING)       // first accumulator column: behind the A tiles of 32
#define MT_ACCN (2 * MT_GROUP)      // columns of an accumulator
#define MT_TMEM 512                 // 3 * (64 + 96) = 480, rounded to a power of two
static_assert(MT_RING * 4 == MT_DECODE && MT_ACC + 2 * MT_RING * MT_ACCN <= MT_TMEM, "rings");
#define MT_HEAD 6144                // barriers, tables

struct __align__(16) MtHead {
    uint64_t raw_full[MT_RING], raw_empty[MT_RING], a_full[MT_RING], done[MT_RING], acc_empty[MT_RING];
    uint32_t tmem; int bound[2];
    __align__(16) float sc[8 * MT_GROUP];   // [block][entry] inverse powers of two, read four at a time
    float d[8][128];                // block factors of the unit's rows, by block modulo 8: the decoders are at most the rings and their own three half blocks
                                    // ahead of the drain warps
    int tok[MT_GROUP], slt[MT_GROUP]; float w[MT_GROUP];
};
static_assert(sizeof(MtHead) <= MT_HEAD && offsetof(MtHead, sc) % 16 == 0 && MT_GROUP % 4 == 0, "head fits, and its vectors are aligned");

template <int N> struct MtWidth { static constexpr int value = N; };

template <bool DOWN>
__global__ void __launch_bounds__(MT_THREADS, 1) pb_moetc_kernel(const PbExpertParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    MtHead& hd = *reinterpret_cast<MtHead*>(smem);
    uint8_t* bt = smem + MT_HEAD;                                       // [step of 64 columns][np rows of 128 bytes, swizzled]
    const int tid = threadIdx.x, warp = tc_uniform_warp(), lane = tid & 31, quad = warp & 3;
    const int bpr = p.bpr, cols = 256 * bpr, nh = 2 * bpr;              // half blocks of a row
    const uint32_t raw = pb_smem_u32(bt) + (uint32_t)(p.nslots * cols * 4);
    if (tid == 0) {
        for (int i = 0; i < MT_RING; i++) {
            pb_mbar_init(&hd.raw_full[i], 32); pb_mbar_init(&hd.raw_empty[i], 4); pb_mbar_init(&hd.a_full[i], 4); pb_mbar_init(&hd.done[i], 1);
            pb_mbar_init(&hd.acc_empty[i], MT_DRAIN);
        }
        pb_fence_barrier_init();
    }
    if (warp == MT_MMA) tc_alloc(&hd.tmem, MT_TMEM);
    pb_pdl_trigger();
    pb_pdl_wait();          // lists, activations / hidden vectors come from earlier kernels
    const int nv = *p.n_virt, nsh = p.has_shared ? (p.sh_ntok + MT_GROUP - 1) / MT_GROUP : 0;
    const int upg = p.rows_e / (DOWN ? 128 : 64);                       // units per group
    // the CTA's run, as in pb_moeh.cu: the thread whose group holds a boundary finds its unit
    if (tid < 2) hd.bound[tid] = (nv + nsh) * upg;
    const int4 lv = nv > 0 ? p.virt[nv - 1] : make_int4(0, 0, 0, 0);
    const int croute = lv.w + pb_vgroup_cost(lv.z, true), zlast = p.sh_ntok - (nsh - 1) * MT_GROUP;
    const int64_t total = ((int64_t)croute + (nsh > 0 ? (nsh - 1) * pb_vgroup_cost(MT_GROUP, true) + pb_vgroup_cost(zlast, true) : 0)) * upg;
    const int64_t at0 = total * blockIdx.x / gridDim.x, at1 = total * (blockIdx.x + 1) / gridDim.x;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    for (int v = tid; v < nv + nsh; v += MT_THREADS) {
        const int4 e = v < nv ? p.virt[v] : make_int4(0, 0, v == nv + nsh - 1 ? zlast : MT_GROUP, croute + (v - nv) * pb_vgroup_cost(MT_GROUP, true));
        const int c = pb_vgroup_cost(e.z, true);
        const int64_t lo = (int64_t)e.w * upg, hi = lo + (int64_t)c * upg;
        if (at0 >= lo && at0 < hi) hd.bound[0] = v * upg + (int)(at0 - lo) / c;
        if (at1 >= lo && at1 < hi) hd.bound[1] = v * upg + (int)(at1 - lo) / c;
    }
    __syncthreads();
    const int u1 = hd.bound[1];
    const uint32_t tmem = hd.tmem;
    bool ok = true;
    int H = 0;               // half blocks before this group (every role counts alike): slot H % MT_RING
    for (int u0 = hd.bound[0]; u0 < u1;) {
        const int v = u0 / upg, ue = min(u1, (v + 1) * upg), nu = ue - u0;
        int4 e;
        if (v < nv) {
            e = p.virt[v];
            if (e.x < 0 || e.x >= p.n_exp || e.y < 0 || e.z < 1 || e.z > MT_GROUP || e.y + e.z > p.t * p.top_k) { if (tid == 0) atomicExch(p.status, PB_DEV_BAD_INDEX); u0 = ue; continue; }
        } else { const int t0 = (v - nv) * MT_GROUP; e = make_int4(-1, t0, min(MT_GROUP, p.sh_ntok - t0), 0); }
        const int zp = (e.z + 7) & ~7, np = 2 * zp;
        // ---- raw rows of the group's units; the first half blocks are requested before the activations are prepared
        const size_t off = e.x < 0 ? 0 : (size_t)(e.x - p.e_base) * p.rows_e * p.row_bytes;
        const uint8_t *wa = (e.x < 0 ? p.sh_a : p.w_a) + off, *wb = DOWN ? nullptr : (e.x < 0 ? p.sh_b : p.w_b) + off;
        const int u00 = u0 - v * upg;       // first unit inside the group
        const size_t rb8 = (size_t)8 * p.row_bytes;
        // eight rows (group g of the tile's sixteen) of unit j: DOWN rows 128 j + 8 g; GU per warp's 32 lanes two groups of gate, two of up
        auto rows8 = [&](int j, int g) { return DOWN ? wa + (16 * (size_t)j + g) * rb8 : ((g & 2) ? wb : wa) + (8 * (size_t)j + 2 * (g >> 2) + (g & 1)) * rb8; };
        auto issue = [&](int i) {           // half block i of the group's units (a producer warp)
            const int slot = (H + i) % MT_RING, j = u00 + i / nh, h = i % nh;
            if (!tc_warp_wait(&hd.raw_empty[slot], (((H + i) / MT_RING) & 1) ^ 1, p.status)) return false;
            const uint32_t dst = raw + (uint32_t)(slot * MT_RAW_BYTES);
            const size_t col = (size_t)(h >> 1) * 1088;
            const int r = lane >> 2, q = lane & 3;
            uint32_t at = dst + (uint32_t)(r * 64 + ((q + (r >> 1)) & 3) * 16);
            const uint8_t *a = rows8(j, 0) + col + 512 * (h & 1) + 16 * lane, *b = DOWN ? a + 2 * rb8 : rows8(j, 2) + col + 512 * (h & 1) + 16 * lane;
            const size_t step = (DOWN ? 4 : 2) * rb8;
#pragma unroll
            for (int k = 0; k < 4; k++, at += 2048, a += step, b += step) { pb_h_cp16(at, a); pb_h_cp16(at + 512, a + rb8); pb_h_cp16(at + 1024, b); pb_h_cp16(at + 1536, b + rb8); }
#pragma unroll
            for (int k = 0; k < 2; k++) { const int g = 8 * k + (lane >> 2); pb_h_cp16(dst + 8192u + (uint32_t)(g * 64 + (lane & 3) * 16), rows8(j, g) + col + 1024 + 16 * (lane & 3)); }
            tc_cp_async_arrive(&hd.raw_full[slot]);
            // four blocks on, into L2: the ring covers a trip to L2, not one to DRAM.  Lane l: lines of rows (l & 15), the first five or the last four
            const int bn = (i >> 1) + 4;
            if (!(i & 1) && bn < nu * bpr) {
                const uint8_t* f = rows8(u00 + bn / bpr, lane & 15) + (size_t)(bn % bpr) * 1088 + (lane < 16 ? 0 : 640);
#pragma unroll
                for (int k = 0; k < 5; k++) if (k < 4 || lane < 16) asm volatile("prefetch.global.L2 [%0];" ::"l"(f + 128 * k));
            }
            return true;
        };
        const int nhb = nu * nh;
        // producer warp k takes the half blocks that go through slot k (H counts whole half blocks, so the first one is k's only if it is its turn)
        int next = warp >= MT_DRAIN + MT_DECODE && warp < MT_MMA ? (warp - MT_DRAIN - MT_DECODE - H % MT_RING + MT_RING) % MT_RING : nhb;
        if (next < nhb && ok) { ok = issue(next); next += MT_RING; }
        // ---- the group's entries and activations: a block of an entry per warp
        if (tid < e.z) {
            int tok = e.x < 0 ? p.sh_tok0 + e.y + tid : p.ent_tok[e.y + tid];
            if (tok < 0 || tok >= p.t) { atomicExch(p.status, PB_DEV_BAD_INDEX); tok = 0; }
            hd.tok[tid] = tok; hd.slt[tid] = e.x < 0 ? 0 : p.ent_slot[e.y + tid]; hd.w[tid] = e.x < 0 ? 1.f : p.ent_w[e.y + tid];
        }
        __syncthreads();
        const int c0 = pb_h_c0<PB_T_IQ3S_N4>(lane), c1 = pb_h_c1<PB_T_IQ3S_N4>(lane), pq = lane & 3, pu = lane >> 2;
#pragma unroll 2
        for (int i = warp; i < e.z * bpr; i += MT_THREADS / 32) {
            const int k = i / bpr, blk = i - k * bpr;
            const float* src; float sc = 1.0f; bool norm = false;
            if (DOWN) src = (e.x < 0 ? p.h_sh + (size_t)(p.sh_tok0 + e.y + k) * cols : p.h + (size_t)(e.y + k) * cols) + 256 * blk;
            else {
                const int tok = hd.tok[k];
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
            uint32_t hi[4], lo[4];
            const float ip = pb_h_split<PB_T_IQ3S_N4>(x, hi, lo);
            if (lane == 0) hd.sc[blk * MT_GROUP + k] = ip;
            // word u of quarter q: step u / 2 of the block, MMA 2 (u & 1) and the next; quarter q holds its k = 4 q .. 4 q + 3
            uint8_t* t = bt + (size_t)(4 * blk + (pu >> 1)) * ((size_t)np * 128);
#pragma unroll
            for (int half = 0; half < 2; half++) {      // high parts in row k, low parts in row zp + k
                const int n = half ? zp + k : k;
                uint8_t* row = t + n * 128 + 8 * (pq & 1);
                const uint32_t* s = half ? lo : hi;
                const int ch = 4 * (pu & 1) + (pq >> 1);
                *reinterpret_cast<uint2*>(row + ((ch ^ (n & 7)) << 4)) = make_uint2(s[0], s[1]);
                *reinterpret_cast<uint2*>(row + (((ch + 2) ^ (n & 7)) << 4)) = make_uint2(s[2], s[3]);
            }
        }
        pb_fence_proxy_async();     // the tensor core reads the tiles through the async proxy
        __syncthreads();
        if (warp >= MT_DRAIN + MT_DECODE && warp < MT_MMA) {
            // ------------------------------------------------------------ producers
            for (; next < nhb && ok; next += MT_RING) ok = issue(next);
        } else if (warp == MT_MMA) {
            // ------------------------------------------------------------ MMA issue
            const uint32_t idesc = tc_idesc(128, np);
            const uint64_t bdesc = tc_desc(pb_smem_u32(bt));
            const uint64_t tile = (uint64_t)(np * 8);                                   // a step's B tile (addresses enter a descriptor in units of 16 bytes)
            const bool elected = tc_elect();
            int slot = H % MT_RING, ph = (H / MT_RING) & 1, h = 0;                      // h: half block of the row
            uint64_t b = bdesc;
            for (int i = 0; i < nhb; i++) {
                // (acc_empty of the first round of slots: the phase before the first counts as complete)
                ok = tc_warp_wait(&hd.acc_empty[slot], ph ^ 1, p.status) && tc_warp_wait(&hd.a_full[slot], ph, p.status);
                if (!ok) break;
                tc_fence_after();
                if (elected) {
                    const uint32_t d = tmem + MT_ACC + (uint32_t)slot * (2 * MT_ACCN), a = tmem + (uint32_t)slot * 64;
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        tc_mma_f16_ts(d, a + 8 * kk, b + 2 * kk, idesc, kk ? 1u : 0u);
                        tc_mma_f16_ts(d + MT_ACCN, a + 32 + 8 * kk, b + tile + 2 * kk, idesc, kk ? 1u : 0u);
                    }
                    tc_commit(&hd.done[slot]);
                }
                __syncwarp();
                b += 2 * tile;
                if (++h == nh) { h = 0; b = bdesc; }
                if (++slot == MT_RING) { slot = 0; ph ^= 1; }
            }
        } else if (warp >= MT_DRAIN) {
            // ------------------------------------------------------------ decoders
            const int grp = (warp - MT_DRAIN) >> 2, row = 32 * quad + lane, g = row >> 3, r = row & 7;
            for (int i = grp; i < nhb && ok; i += MT_RING) {   // (H and the half blocks of a row are even)
                const int slot = (H + i) % MT_RING;
                ok = tc_warp_wait(&hd.raw_full[slot], ((H + i) / MT_RING) & 1, p.status);
                if (!ok) break;
                const uint32_t src = raw + (uint32_t)(slot * MT_RAW_BYTES);
                const uint2 head = pb_ldsa64(src + 8192u + (uint32_t)(g * 64 + r * 8));
                uint4 w[4];
#pragma unroll
                for (int q = 0; q < 4; q++) w[q] = pb_ldsa128(src + (uint32_t)(g * 512 + r * 64 + ((q + (r >> 1)) & 3) * 16));
                __half2 mlo[4], mhi[4], mof[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const __half2 s = pb_h2_int((head.y >> (8 * q + 4 * (i & 1))) & 0xF);
                    mlo[q] = __hfma2(s, pb_as_h2(0x6C006C00u), pb_as_h2(0x68006800u));
                    mhi[q] = __hfma2(s, pb_as_h2(0x5C005C00u), pb_as_h2(0x58005800u));
                    mof[q] = __hfma2(s, pb_as_h2(0x97809780u), pb_as_h2(0x93809380u));
                }
                if ((i & 1) == 0) hd.d[((H + i) >> 1) & 7][row] = pb_h2f((uint16_t)(head.x & 0xFFFF)) * PB_H_UNIT;
                tc_warp_arrive(&hd.raw_empty[slot], lane);
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    uint32_t cells[32];
#pragma unroll
                    for (int q = 0; q < 4; q++)
#pragma unroll
                        for (int uu = 0; uu < 2; uu++) {
                            const uint32_t x = s ? (uu ? w[q].w : w[q].z) : (uu ? w[q].y : w[q].x), x8 = x >> 8;
                            cells[16 * uu + 2 * q] = pb_as_u32(__hfma2(pb_as_h2(x & 0x000F000Fu), mlo[q], mof[q]));
                            cells[16 * uu + 2 * q + 1] = pb_as_u32(__hfma2(pb_as_h2(x & 0x00F000F0u), mhi[q], mof[q]));
                            cells[16 * uu + 8 + 2 * q] = pb_as_u32(__hfma2(pb_as_h2(x8 & 0x000F000Fu), mlo[q], mof[q]));
                            cells[16 * uu + 8 + 2 * q + 1] = pb_as_u32(__hfma2(pb_as_h2(x8 & 0x00F000F0u), mhi[q], mof[q]));
                        }
                    if (s == 0) {   // the slot's tiles are free (its first use: the phase before the first counts as complete)
                        ok = tc_warp_wait(&hd.done[slot], (((H + i) / MT_RING) & 1) ^ 1, p.status);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    tc_st32_nowait(tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(64 * slot + 32 * s), cells);
                }
                if (!ok) break;
                tc_wait_st();
                tc_fence_before();
                tc_warp_arrive(&hd.a_full[slot], lane);
            }
        } else {
            // ------------------------------------------------------------ drain
            auto drain = [&](auto width) {
                constexpr int W = decltype(width)::value, NE = 4 * W, ZP = 8 * W;   // entries of this warp, of the group (padded)
                const int half = warp >> 2, e0 = NE * half;
                const uint32_t at = tmem + ((uint32_t)(32 * quad) << 16) + MT_ACC + e0;   // (its columns of accumulator 0)
                float tot[NE];
                int slot = H % MT_RING, ph = (H / MT_RING) & 1;
#pragma unroll
                for (int j = 0; j < NE; j++) tot[j] = 0.f;
                for (int i = 0; i < nu && ok; i++) {
                    for (int blk = 0; blk < bpr && ok; blk++) {
                        float acc[2 * NE];
#pragma unroll
                        for (int hb = 0; hb < 2; hb++) {
                            ok = ok && tc_warp_wait(&hd.done[slot], ph, p.status);
                            tc_fence_after();
                            float c[2][2 * NE];
#pragma unroll
                            for (int s = 0; s < 2; s++)
#pragma unroll
                                for (int j = 0; j < NE; j += 4) {
                                    tc_ld4(at + (uint32_t)((2 * slot + s) * MT_ACCN + j), c[s] + j);
                                    tc_ld4(at + (uint32_t)((2 * slot + s) * MT_ACCN + ZP + j), c[s] + NE + j);
                                }
                            tc_wait_ld();
#pragma unroll
                            for (int j = 0; j < 2 * NE; j++) asm volatile("" : "+f"(c[0][j]), "+f"(c[1][j]));   // (used only behind the wait)
                            tc_fence_before();
                            tc_warp_arrive(&hd.acc_empty[slot], lane);
                            if (++slot == MT_RING) { slot = 0; ph ^= 1; }
#pragma unroll
                            for (int s = 0; s < 2; s++)
#pragma unroll
                                for (int j = 0; j < 2 * NE; j += 2) {
                                    const float2 x = hb == 0 && s == 0 ? make_float2(c[0][j], c[0][j + 1]) : pb_f2_get(pb_add2(pb_f2(acc[j], acc[j + 1]), pb_f2(c[s][j], c[s][j + 1])));
                                    acc[j] = x.x; acc[j + 1] = x.y;
                                }
                        }
                        const float d = hd.d[((H + i * nh) / 2 + blk) & 7][32 * quad + lane];
#pragma unroll
                        for (int j = 0; j < NE; j += 4) {
                            const float4 s4 = *reinterpret_cast<const float4*>(&hd.sc[blk * MT_GROUP + e0 + j]);
                            const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                            for (int q = 0; q < 4; q++) tot[j + q] = __fadd_rn(tot[j + q], __fmul_rn(__fadd_rn(__fmul_rn(d, acc[j + q]), __fmul_rn(d, acc[NE + j + q])), sv[q]));
                        }
                    }
                    const int j0 = u0 - v * upg + i;
                    if (!DOWN) {
                        // hidden = silu(gate . x) * (up . x)   (routed :1781-1783, ffn :1680); the lower lanes finish the even entries, the upper the odd ones
                        float* dst = (e.x < 0 ? p.h_sh + (size_t)(p.sh_tok0 + e.y) * p.rows_e : p.h + (size_t)e.y * p.rows_e) + 64 * j0 + 16 * quad + (lane & 15);
#pragma unroll
                        for (int j = 0; j < NE; j += 2) {
                            const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? tot[j + 1] : tot[j], 16);
                            const float gate = lane < 16 ? tot[j] : other, up = lane < 16 ? other : tot[j + 1];
                            const int k = e0 + j + (lane >> 4);
                            if (k < e.z) dst[(size_t)k * p.rows_e] = pb_silu(gate) * up;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < NE; j++)
                            if (e0 + j < e.z) {
                                const int row = 128 * j0 + 32 * quad + lane, k = e0 + j;
                                if (e.x < 0) p.part_sh[(size_t)(p.sh_tok0 + e.y + k) * p.rows_e + row] = tot[j];
                                else p.part[((size_t)hd.tok[k] * p.top_k + hd.slt[k]) * p.rows_e + row] = hd.w[k] * tot[j];   // routed :1786: o += w * dot
                            }
                    }
#pragma unroll
                    for (int j = 0; j < NE; j++) tot[j] = 0.f;
                }
            };
            if (np == 16) drain(MtWidth<1>()); else if (np == 32) drain(MtWidth<2>()); else drain(MtWidth<3>());
        }
        ok = __syncthreads_and(ok) != 0;     // the tables and tiles are rewritten for the next group
        if (!ok) break;
        H += nhb;
        u0 = ue;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == MT_MMA) { tc_fence_after(); tc_dealloc(tmem, MT_TMEM); }
}

// Shapes: the re-coded IQ3_S form, rows in whole units, activations of a group beside the raw ring, a partial-row buffer of this GPU
bool pb_moetc_supported(int type, int d, int ff) { return type == PB_T_IQ3S_N4 && d % 256 == 0 && ff % 256 == 0 && d <= 2048 && ff <= 2048; }

template <bool DOWN>
static int launch_moetc(pb_ctx* ctx, PbExpertParams p, int cols) {
    p.bpr = cols / 256; p.row_bytes = cols / 256 * 136;
    p.nslots = MT_GROUP;
    const size_t smem = MT_HEAD + (size_t)MT_GROUP * cols * 4 + (size_t)MT_RING * MT_RAW_BYTES;
    if (smem > (size_t)ctx->max_smem_optin || p.part_tok) PB_FAIL(ctx, PB_UNSUPPORTED, "expert kernel of prompts: %zu bytes of shared memory", smem);
    p.status = ctx->dev_status;
    auto kern = pb_moetc_kernel<DOWN>;
    PB_TRY(pb_ensure_smem(ctx, kern, smem));
    pb_launch_k(ctx, kern, dim3(ctx->sm_count), dim3(MT_THREADS), smem, p);
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    return PB_OK;
}
int pb_launch_moetc_gu(pb_ctx* ctx, const PbExpertParams& p, int cols) { return launch_moetc<false>(ctx, p, cols); }
int pb_launch_moetc_down(pb_ctx* ctx, const PbExpertParams& p, int cols) { return launch_moetc<true>(ctx, p, cols); }
