// Dequant-GEMM for 16 and more activation columns on the fifth-generation tensor cores (tcgen05), IQ3_S weights.
//
//   y[b][yoff_s + r] (+)= sum_c W_s[r][c] * act(x)[b][c]        b = 0 .. t-1,  t >= 16
//
// This is the path of prefill chunks, wide verify windows and batched decode: the reference switches to its tensor-core
// GEMM at 16 tokens as well (gmm, src/model/qwen4exp_gguf.rs:3264-3266; k_gemm_tc, src/model/qn_cube.rs:153, host side
// gemm_pfx :6559-6587).  One CTA owns a tile of 128 weight rows x up to 256 tokens and walks the contraction in steps of
// 64 columns through a ring of 3 or 6 stages (a weight tile in tensor memory + the activation tiles in shared memory):
//
//   producer warp       brings the activations of each step -- f16 high and low parts (x = hi + lo, 22 significant
//                       bits), prepared once per GEMM by pb_xt_prep_kernel in exactly the operand layout -- with 1-D
//                       bulk copies.
//   decoder warps (8)   stream the re-coded IQ3_S rows of the tile (4-bit codes, PB_T_IQ3S_N4: 136 bytes per row and 256
//                       columns) into a double buffer of raw bytes with 16-byte cp.async (all 256 threads share the
//                       copies), then one thread = one row x 64 columns per step: f16 weights stored with tcgen05.st
//                       into the thread's own lane of a weight tile in tensor memory (the A operand is read from
//                       there, behind the accumulator).  (2c - 15) * (1 + 2s) is
//                       exact in f16; the block scale d is folded in with one rounding (relative 2^-11), after a
//                       per-tile power-of-two shift that keeps d * 465 inside the f16 range and is undone at the end.
//   MMA warp            one elected thread issues tcgen05.mma (kind::f16, M = 128, N = tokens, K = 16) for the high and
//                       the low part into one f32 accumulator in tensor memory (128 lanes x N columns) and frees the
//                       stage with tcgen05.commit -> mbarrier.
//   epilogue            the decoder warps read the accumulator with tcgen05.ld (lane = row), undo the scales and store.
//
// Every wait is bounded; a wait that runs out records a status (the host call returns PB_ERR_DEVICE) and the CTA leaves
// through the common exit, which frees its tensor memory.  A matrix of few tiles is cut along its columns over a cluster of up to eight CTAs, whose
// sums meet through distributed shared memory; nothing is multicast, operands come only from this GPU.
#include "pb_tc.cuh"
#include "pb_internal.h"

#include <cuda_fp16.h>
#include <stdio.h>

#define TC_ROWS 128                 // weight rows per tile = MMA M
#define TC_NARROW 128               // tokens per CTA, narrow form: the MMA's N is twice the (padded) token count, high and low parts side by side
#define TC_WIDE 256                 // wide form: the two parts are two MMAs into the same columns, and one decode of a weight tile serves twice the tokens
#define TC_KSTEP 64                 // contraction columns per step
#define TC_STAGES 6                 // ring depth: a stage = a decoded weight tile in tensor memory (32 columns behind the accumulator's
                                    // 256) + the activation tiles of the same step in shared memory (wide: 3 stages)
#define TC_ACC_COLS 256             // accumulator columns
#define TC_A_COLS (TC_KSTEP / 2)    // a weight tile is 128 lanes x 32 columns: two f16 per 32-bit cell
#define TC_TMEM_COLS 512            // 256 + 6 x 32 = 448, rounded to the power of two: the whole tensor memory of the SM (one CTA per SM)
#define TC_RAW_STAGES 2             // raw double buffer: one block (256 columns = 4 steps) each (deeper rings measured the same)
#define TC_RAW_BYTES (TC_ROWS * 136)
#define TC_DECODERS 8
#define TC_THREADS ((TC_DECODERS + 2) * 32)
#define TC_B_BYTES (2 * TC_NARROW * TC_KSTEP * 2)                 // high and low activation tiles of a stage: 32 KB, in the wide form twice that
#define TC_XT_HEAD 4096             // bytes of per-token prescale inverses in front of the activation tiles

// ---------------------------------------------------------------- activations -> operand tiles

// byte offset of element (token n of its block, column c) inside the block's tiles; np = padded tokens of the block
__device__ __forceinline__ size_t pb_xt_off(int np, int n, int c, int lo) {
    const int ks = c >> 6, kk = c & 63;
    return (size_t)ks * (2 * (size_t)np * 128) + (lo ? (size_t)np * 128 : 0) + (size_t)n * 128 + (size_t)(((kk >> 3) ^ (n & 7)) * 16) + (size_t)(kk & 7) * 2;
}
__device__ __forceinline__ void pb_xt_store(uint8_t* blk, int np, int n, int c, float4 v) {
    const __half2 h01 = __floats2half2_rn(v.x, v.y), h23 = __floats2half2_rn(v.z, v.w);
    const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
    const __half2 l01 = __floats2half2_rn(v.x - f01.x, v.y - f01.y), l23 = __floats2half2_rn(v.z - f23.x, v.w - f23.y);
    *reinterpret_cast<uint2*>(blk + pb_xt_off(np, n, c, 0)) = make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
    *reinterpret_cast<uint2*>(blk + pb_xt_off(np, n, c, 1)) = make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
}
__host__ __device__ __forceinline__ int pb_xt_np(int t, int tb, int nb) { const int n = t - tb * nb < nb ? t - tb * nb : nb; return (n + 15) & ~15; }   // nb: tokens of a block

// One CTA per token slot (the slots past t of the last block are written as zeros).  The activation function is the
// one of the other GEMV kernels: PLAIN (with an exact power-of-two prescale into [0.5, 1) so that f16 neither overflows
// nor loses small columns), NORM (RMS norm times weight), GNORM (per-head RMS norm times weight times sigmoid(z)).
// xbuf: TC_XT_HEAD bytes of prescale inverses [t], then per block of nb tokens, per step of 64 columns, the high
// tile and the low tile, each np x 64 f16 as swizzled 128-byte rows.
__global__ void __launch_bounds__(256) pb_xt_prep_kernel(const PbGemvQParams p, int nb, uint8_t* __restrict__ xbuf) {
    constexpr int CT = 256;
    const int slot = (int)blockIdx.x;
    const int tb = slot / nb, n = slot - tb * nb;
    const int np = pb_xt_np(p.t, tb, nb);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cols = p.bpr * 256;
    __shared__ float red0[8];
    pb_pdl_wait();
    pb_pdl_trigger();
    if (n >= np) return;
    const int tok = tb * nb + n;
    const bool live = tok < p.t;
    const float* x = p.x + (size_t)tok * p.ldx;
    const float* z = p.z ? p.z + (size_t)tok * p.ldz : nullptr;
    uint8_t* blk = xbuf + TC_XT_HEAD + (size_t)tb * ((size_t)cols / 64) * (2 * (size_t)nb * 128);
    float* xinv = reinterpret_cast<float*>(xbuf);
    if (tid == 0 && live) xinv[tok] = 1.0f;
    if (p.mode == PB_ACT_GNORM) {
        const int nheads = cols / p.head_dim;   // head_dim == 128 (checked on the host)
        for (int h = warp; h < nheads; h += 8) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live) {
                v = *reinterpret_cast<const float4*>(x + h * p.head_dim + 4 * lane);
                const float ss = pb_warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
                const float s = 1.0f / sqrtf(ss / (float)p.head_dim + p.eps);
                const float4 w = *reinterpret_cast<const float4*>(p.norm_w + 4 * lane);
                const float4 zz = *reinterpret_cast<const float4*>(z + h * p.head_dim + 4 * lane);
                v.x = v.x * (s * w.x) * pb_sigm(zz.x); v.y = v.y * (s * w.y) * pb_sigm(zz.y); v.z = v.z * (s * w.z) * pb_sigm(zz.z); v.w = v.w * (s * w.w) * pb_sigm(zz.w);
            }
            pb_xt_store(blk, np, n, h * p.head_dim + 4 * lane, v);
        }
        return;
    }
    float r = 0.f;
    if (live) for (int c = tid; c < cols; c += CT) { const float v = x[c]; r = p.mode == PB_ACT_NORM ? r + v * v : fmaxf(r, fabsf(v)); }
    r = p.mode == PB_ACT_NORM ? pb_warp_sum(r) : pb_warp_max(r);
    if (lane == 0) red0[warp] = r;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) tot = p.mode == PB_ACT_NORM ? tot + red0[i] : fmaxf(tot, red0[i]);
    float s = 1.0f;
    if (p.mode == PB_ACT_NORM) s = 1.0f / sqrtf(tot / (float)cols + p.eps);
    else if (tot > 0.f && tot <= 3.0e38f) {
        int e; (void)frexpf(tot, &e);
        s = ldexpf(1.0f, -e);
        if (tid == 0 && live) xinv[tok] = ldexpf(1.0f, e);
    }
    for (int c = tid * 4; c < cols; c += CT * 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) {
            v = *reinterpret_cast<const float4*>(x + c);
            if (p.mode == PB_ACT_NORM) { const float4 w = *reinterpret_cast<const float4*>(p.norm_w + c); v.x = v.x * s * w.x; v.y = v.y * s * w.y; v.z = v.z * s * w.z; v.w = v.w * s * w.w; }
            else { v.x *= s; v.y *= s; v.z *= s; v.w *= s; }
        }
        pb_xt_store(blk, np, n, c, v);
    }
}

// ---------------------------------------------------------------- weights -> operand tile

// raw bytes of one quarter (64 weights) of a re-coded block: {d (f16) | pad, four sub-scale bytes}, 32 bytes of codes
struct TcRaw { uint2 head; uint2 c[4]; };
// from the raw ring: `b` = shared-memory address of the block of this row's group of eight (pb_repack.cu), row = row in the group
__device__ __forceinline__ void tc_load_raw(TcRaw& r, uint32_t b, int row, int qt, bool live) {
    if (!live) { r.head = make_uint2(0u, 0u); r.c[0] = r.c[1] = r.c[2] = r.c[3] = make_uint2(0x77777777u, 0x77777777u); return; }
    // volatile with a memory clobber: these loads must stay behind the wait for the block's copies
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.head.x), "=r"(r.head.y) : "r"(b + 1024 + 8 * row) : "memory");
#pragma unroll
    for (int i = 0; i < 2; i++) asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.c[2 * i].x), "=r"(r.c[2 * i].y), "=r"(r.c[2 * i + 1].x), "=r"(r.c[2 * i + 1].y) : "r"(b + 512 * i + (4 * row + qt) * 16) : "memory");
}
// decode the 64 columns of step ks of this thread's row and store them as its lane of the weight tile at taddr
// (tensor memory: lane = row, cell j = columns 2j, 2j + 1 of the step)
__device__ __forceinline__ void tc_decode_store(const TcRaw& r, int ks, uint32_t taddr, float shift) {
    const int qt = ks & 3;
    const float d = pb_h2f((uint16_t)(r.head.x & 0xFFFF)) * shift;
    const uint32_t sc = (r.head.y >> (8 * qt)) & 0xFF;
    const float f0 = (float)(1 + 2 * (int)(sc & 0xF)), f1 = (float)(1 + 2 * (int)(sc >> 4));
    const __half2 a0 = __float2half2_rn(2.0f * f0), b0 = __float2half2_rn(-15.0f * f0);
    const __half2 a1 = __float2half2_rn(2.0f * f1), b1 = __float2half2_rn(-15.0f * f1);
    const __half2 k1024 = __float2half2_rn(1024.0f), d2 = __float2half2_rn(d);
    uint32_t cells[32];
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int u = 2 * i + j;                      // word u = weights 8u .. 8u+7 of the quarter = core matrix u along K
            const uint32_t w = j ? r.c[i].y : r.c[i].x;
            const uint32_t lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
            const uint32_t c4[4] = {pb_prmt(lo, 0x64006400u, 0x7150u), pb_prmt(lo, 0x64006400u, 0x7352u), pb_prmt(hi, 0x64006400u, 0x7150u), pb_prmt(hi, 0x64006400u, 0x7352u)};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                // (1024 + c) - 1024 = c, c * 2m - 15m = (2c - 15) m: exact in f16; the product with d rounds once
                const __half2 v = __hmul2(__hfma2(__hsub2(*reinterpret_cast<const __half2*>(&c4[e]), k1024), u < 4 ? a0 : a1, u < 4 ? b0 : b1), d2);
                cells[4 * u + e] = *reinterpret_cast<const uint32_t*>(&v);
            }
        }
    }
    tc_st32(taddr, cells);
}

struct TcParams {
    PbGemvQSeg seg[4];      // chunk0 = first tile of the segment
    int nseg, ntiles;
    int row_bytes, cols, t;
    const uint8_t* xt;      // prepared activations (pb_xt_prep_kernel)
    float* y; int64_t ldy;
    int accumulate;
    int ks;                 // CTAs of a cluster: each takes cols / ks columns of its tile, their sums meet through distributed shared memory
    int* status;
};

template <bool WIDE>
__global__ void __launch_bounds__(TC_THREADS, 1) pb_gemmtc_iq3s_kernel(const TcParams p) {
    constexpr int NB = WIDE ? TC_WIDE : TC_NARROW, NST = WIDE ? TC_STAGES / 2 : TC_STAGES;   // tokens of a CTA, stages of the ring
    constexpr size_t STB = WIDE ? 2 * TC_B_BYTES : TC_B_BYTES;                               // and their bytes
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);             // [TC_STAGES] the arrivals of four decoder warps + the producer's, and the bulk-copy bytes
    uint64_t* empty = full + TC_STAGES;                             // [TC_STAGES] tcgen05.commit: the MMAs that read the stage are done
    uint64_t* raw_full = empty + TC_STAGES;                         // [TC_RAW_STAGES] 256 decoder threads (cp.async)
    uint64_t* raw_empty = raw_full + TC_RAW_STAGES;                 // [TC_RAW_STAGES] 8 decoder warps
    uint64_t* acc_full = raw_empty + TC_RAW_STAGES;                 // accumulator complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 384);
    float* red = reinterpret_cast<float*>(smem + 416);              // [8] per-warp maxima of d
    uint8_t* b_ring = smem + 1024;                                  // [TC_STAGES][high tile | low tile], swizzled 128-byte rows
    uint8_t* raw = b_ring + TC_STAGES * TC_B_BYTES;               // [TC_RAW_STAGES][128 rows][136 bytes]
    float* part = reinterpret_cast<float*>(b_ring);                 // [tokens][TC_ROWS] sums of this CTA's share of the contraction, once the MMAs are done
    static_assert((TC_STAGES * 2 + TC_RAW_STAGES * 2 + 1) * 8 <= 384 && TC_ACC_COLS + TC_STAGES * TC_A_COLS <= TC_TMEM_COLS, "barriers fit in front of the TMEM slot");
    const int tid = threadIdx.x, warp = tc_uniform_warp(), lane = tid & 31;

    const int ks = p.ks, rank = (int)blockIdx.x % ks, tile = (int)blockIdx.x / ks, tb = (int)blockIdx.y;   // (clusters are consecutive CTAs)
    int s = 0;
    while (s + 1 < p.nseg && tile >= p.seg[s + 1].chunk0) s++;
    const int r0 = (tile - p.seg[s].chunk0) * TC_ROWS;
    const int nr = min(TC_ROWS, p.seg[s].rows - r0);
    const int np = pb_xt_np(p.t, tb, NB);             // padded tokens of this block = MMA N
    const int nt = min(NB, p.t - tb * NB);  // live tokens
    const int nkt = p.cols / TC_KSTEP, nk = nkt / ks, kb0 = rank * (nk / 4);   // steps of a row, of this CTA, and its first block
    const uint32_t bbytes = 2u * (uint32_t)np * 128u;

    if (tid == 0) {
        for (int i = 0; i < TC_STAGES; i++) { pb_mbar_init(&full[i], 4 + 1); pb_mbar_init(&empty[i], 1); }
        for (int i = 0; i < TC_RAW_STAGES; i++) { pb_mbar_init(&raw_full[i], TC_DECODERS * 32); pb_mbar_init(&raw_empty[i], TC_DECODERS); }
        pb_mbar_init(acc_full, 1);
        pb_fence_barrier_init();
    }
    if (warp == TC_DECODERS + 1) tc_alloc(tmem_slot, TC_TMEM_COLS);
    pb_pdl_trigger();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // (pb_pdl_wait below, per role: the activation tiles, and y when accumulating, come from earlier launches; the weights do not)

    if (warp == TC_DECODERS) {
        // ------------------------------------------------------------ producer: activation tiles, a ring ahead
        pb_pdl_wait();
        if (lane == 0) {
            const uint8_t* src = p.xt + TC_XT_HEAD + (size_t)tb * (size_t)nkt * (2 * (size_t)NB * 128) + (size_t)rank * nk * bbytes;
            int k = 0;
            for (; k < nk; k++) {
                const int st = k % NST;
                if (k >= NST && !pb_mbar_wait(&empty[st], ((k / NST) - 1) & 1, p.status, PB_DEV_TC_TIMEOUT)) break;
                pb_mbar_expect_tx(&full[st], bbytes);
                pb_bulk_g2s(b_ring + (size_t)st * STB, src + (size_t)k * bbytes, bbytes, &full[st]);
            }
            // error path: the copies in flight get a bounded chance to land before the CTA may exit
            // (a stage's barrier also counts the decoders' arrivals: on the error path it may never complete; the wait is bounded)
            if (k < nk) for (int j = max(0, k - NST); j < k; j++) pb_mbar_wait(&full[j % NST], (j / NST) & 1, nullptr, 0);
        }
    } else if (warp == TC_DECODERS + 1) {
        // ------------------------------------------------------------ MMA issue
        // narrow form: the high and the low tile are stacked along N: one instruction of N = 2 np columns per 16 columns of K
        // reads the weight tile once, and the epilogue adds the two halves of the accumulator
        pb_pdl_wait();
        const uint32_t idesc = tc_idesc(TC_ROWS, WIDE ? np : 2 * np);
        const uint64_t bdesc = tc_desc(pb_smem_u32(b_ring));
        const bool elected = tc_elect();
        bool ok = true;
        for (int k = 0; k < nk && ok; k++) {
            const int st = k % NST;
            ok = tc_warp_wait(&full[st], (k / NST) & 1, p.status);
            if (!ok) break;
            tc_fence_after();
            if (elected) {
                const uint32_t a_t = tmem + TC_ACC_COLS + (uint32_t)st * TC_A_COLS;
                const uint64_t b = bdesc + (uint64_t)((uint32_t)st * (uint32_t)(STB >> 4));       // (addresses enter a descriptor in units of 16 bytes)
#pragma unroll
                for (int kk = 0; kk < TC_KSTEP / 16; kk++) {
                    tc_mma_f16_ts(tmem, a_t + kk * 8, b + 2 * kk, idesc, kk ? 1u : (k ? 1u : 0u));
                    if (WIDE) tc_mma_f16_ts(tmem, a_t + kk * 8, b + (uint64_t)((uint32_t)np * 8u) + 2 * kk, idesc, 1u);
                }
                tc_commit(&empty[st]);
            }
            __syncwarp();
        }
        if (ok && elected) tc_commit(acc_full);
        __syncwarp();
    } else {
        // ------------------------------------------------------------ decoders, then epilogue
        const int grp = warp >> 2;                 // two groups of four warps take alternate steps
        const int row = (warp & 3) * 32 + lane;    // row of the tile
        const bool live = row < nr;
        const uint8_t* wbase = p.seg[s].w + (size_t)r0 * p.row_bytes + (size_t)kb0 * 1088;   // (within a group of eight rows a block is 1088 bytes)
        // raw bytes: block kb of the tile's rows -> raw[kb % TC_RAW_STAGES]; thread tid copies 16-byte words tid, tid + 256, ..
        const int nkb = nk / 4, nwords = (nr + 7) / 8 * 68;
        auto issue_raw = [&](int kb) {
            const uint32_t dst = pb_smem_u32(raw + (size_t)(kb % TC_RAW_STAGES) * TC_RAW_BYTES);
            for (int i = tid; i < nwords; i += TC_DECODERS * 32) {
                const int gr = i / 68, w = i - gr * 68;
                tc_cp_async16(dst + (uint32_t)(gr * 1088 + w * 16), wbase + (size_t)gr * 8 * p.row_bytes + (size_t)kb * 1088 + w * 16);
            }
            tc_cp_async_arrive(&raw_full[kb % TC_RAW_STAGES]);
        };
        for (int i = 0; i < TC_RAW_STAGES && i < nkb; i++) issue_raw(i);
        // per-tile power-of-two shift: the largest |d| of the tile's rows times 465 lands in [2^14, 2^15)
        float dm = 0.f;
        // (the two groups take alternate blocks; eight loads at a time: one after the other they were a trip to HBM each)
        if (live) for (int b0 = grp; b0 < nkb; b0 += 16) {
            float dv[8];
#pragma unroll
            for (int i = 0; i < 8; i++) dv[i] = b0 + 2 * i < nkb ? fabsf(pb_h2f(__ldg(reinterpret_cast<const uint16_t*>(wbase + (size_t)(row & ~7) * p.row_bytes + (size_t)(b0 + 2 * i) * 1088 + 1024 + 8 * (row & 7))))) : 0.f;
#pragma unroll
            for (int i = 0; i < 8; i++) dm = fmaxf(dm, dv[i]);
        }
        dm = pb_warp_max(dm);
        if (lane == 0) red[warp] = dm;
        pb_pdl_wait();
        pb_named_barrier(1, TC_DECODERS * 32);
        dm = fmaxf(fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])), fmaxf(fmaxf(red[4], red[5]), fmaxf(red[6], red[7])));
        int sh = 0;
        if (dm > 0.f && dm < 3.0e38f) { int e; (void)frexpf(dm * 465.0f, &e); sh = 15 - e; }   // dm * 465 * 2^sh in [2^14, 2^15)
        const float shift = ldexpf(1.0f, sh), unshift = ldexpf(1.0f, -sh);

        bool ok = true;
        for (int k = grp; k < nk; k += 2) {
            const int st = k % NST, kb = k >> 2, rs = kb % TC_RAW_STAGES;
            // this group's steps of a block are quarters grp and grp + 2: wait for the bytes at the first; after the second,
            // release the buffer and -- once all 256 threads have released it -- refill it
            if ((k & 3) == grp && !tc_warp_wait(&raw_full[rs], (kb / TC_RAW_STAGES) & 1, p.status)) { ok = false; break; }
            TcRaw cur;
            tc_load_raw(cur, pb_smem_u32(raw + (size_t)rs * TC_RAW_BYTES) + (uint32_t)(row >> 3) * 1088u, row & 7, k & 3, live);
            if ((k & 3) == grp + 2) {
                tc_warp_arrive(&raw_empty[rs], lane);
                if (kb + TC_RAW_STAGES < nkb) {
                    if (!tc_warp_wait(&raw_empty[rs], (kb / TC_RAW_STAGES) & 1, p.status)) { ok = false; break; }
                    issue_raw(kb + TC_RAW_STAGES);
                }
            }
            if (k >= NST && !tc_warp_wait(&empty[st], ((k / NST) - 1) & 1, p.status)) { ok = false; break; }
            tc_decode_store(cur, k, tmem + ((uint32_t)((warp & 3) * 32) << 16) + TC_ACC_COLS + (uint32_t)st * TC_A_COLS, shift);
            tc_fence_before();                    // the stores are complete (wait::st); order them before the MMA warp's instructions
            tc_warp_arrive(&full[st], lane);
        }
        // ---- epilogue: warp w reads lanes 32 (w % 4) .. + 31 (its rows); warps 0-3 take the first half of the tokens, 4-7 the rest; columns
        //      [0, np) hold the sums, or (narrow) the high parts' with the low parts' in [np, 2 np)
        if (ok && tc_warp_wait(acc_full, 0, p.status)) {
            tc_fence_after();
            const int half = ((np + 1) / 2 + 31) / 32 * 32;
            for (int c0 = grp * half; c0 < (grp + 1) * half && c0 < np; c0 += 32) {
                // the prescales and (accumulating) the old values of the 32 tokens share one trip to L2
                float* dst = p.y + (size_t)(tb * NB + c0) * p.ldy + p.seg[s].yoff + r0 + row;
                const float xi = c0 + lane < nt ? reinterpret_cast<const float*>(p.xt)[tb * NB + c0 + lane] : 0.f;
                float old[32];
#pragma unroll
                for (int j = 0; j < 32; j++) old[j] = p.accumulate && ks == 1 && live && c0 + j < nt ? dst[(size_t)j * p.ldy] : 0.f;
                uint32_t v[32], vl[32];
                tc_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
                if (!WIDE) tc_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(np + c0), vl);
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const float sum = WIDE ? __uint_as_float(v[j]) : __uint_as_float(v[j]) + __uint_as_float(vl[j]);
                    const float o = sum * (unshift * __shfl_sync(0xffffffffu, xi, j));
                    if (!live || c0 + j >= nt) continue;
                    if (ks > 1) part[(c0 + j) * TC_ROWS + row] = o;
                    else dst[(size_t)j * p.ldy] = old[j] + o;
                }
            }
        }
    }
    __syncwarp();
    if (ks > 1) {
        // the CTAs of the cluster add their sums in the order of the contraction, each a share of the tokens
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const uint32_t src = pb_smem_u32(part);
        const int i1 = nt * (rank + 1) / ks * TC_ROWS;
        for (int ib = nt * rank / ks * TC_ROWS + tid; ib < i1; ib += 4 * TC_THREADS) {   // four outputs at a time
            float v[4][8], old[4];
            float* dst[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = ib + u * TC_THREADS, b = i / TC_ROWS, row = i - b * TC_ROWS;
                dst[u] = i < i1 && row < nr ? p.y + (size_t)(tb * NB + b) * p.ldy + p.seg[s].yoff + r0 + row : nullptr;
                old[u] = dst[u] && p.accumulate ? *dst[u] : 0.f;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    v[u][c] = 0.f;
                    if (c < ks && dst[u]) {
                        uint32_t a;
                        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(src + 4u * (uint32_t)i), "r"(c));
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[u][c]) : "r"(a) : "memory");
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (dst[u]) { float o = v[u][0]; 
#pragma unroll
                    for (int c = 1; c < 8; c++) o += v[u][c]; *dst[u] = old[u] + o; }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // no CTA leaves while its sums are read
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // (error paths) no copy of this thread is still in flight when the CTA exits
    tc_fence_before();
    __syncthreads();
    if (warp == TC_DECODERS + 1) { tc_fence_after(); tc_dealloc(tmem, TC_TMEM_COLS); }
}

bool pb_gemmtc_supported(int type, int cols, int t) { return type == PB_T_IQ3_S && t >= 16 && cols % 256 == 0 && cols >= 256; }

// Fewest tokens the dispatchers send here.  The kernel works from 16 tokens on; there the warp-level kernel is as short or shorter (us, this kernel / that
// one: 4096 x 2048 12.4 / 12.4, 12351 x 2048 20.5 / 16.7, 151936 x 2048 153 / 82).  From 17 tokens on that one is longer on the layers' matrices, in one launch
// (4096 x 2048, 17 tokens 13.3 / 14.4, 31 14.4 / 17.6) and in two (12351 x 2048, 20.6 / 24.7 and 20.6 / 31.8), and from 32 on the lm-head (31 tokens
// 158 / 158, 33 162 / 195); but its weights are exact, and here they are rounded to f16 (2e-4 of the result against 1e-7): up to 31 tokens, the longest call
// that the warp-level kernel takes in two launches at most, results keep their exact weights.  PYRE_B200_TC_MIN overrides (tests run the kernel at 16).
int pb_gemmtc_min_tokens() {
    const char* e = getenv("PYRE_B200_TC_MIN");
    const int v = e ? atoi(e) : 32;
    return v < 16 ? 16 : v;
}

int pb_gemmtc_max_tokens(int cols) {
    const size_t n = (PB_XH_BYTES - TC_XT_HEAD) / ((size_t)cols * 4) / TC_WIDE * TC_WIDE;
    return (int)(n < TC_XT_HEAD / 4 ? n : TC_XT_HEAD / 4);
}

int pb_launch_gemmtc(pb_ctx* ctx, const PbGemvQArgs& a) {
    if (!pb_gemmtc_supported(a.type, a.cols, a.t)) PB_FAIL(ctx, PB_UNSUPPORTED, "tensor-core gemm: type %d cols %d t %d", a.type, a.cols, a.t);
    if (a.mode == PB_ACT_PREQ) PB_FAIL(ctx, PB_UNSUPPORTED, "tensor-core gemm: pre-split activations are not accepted");
    if (a.mode == PB_ACT_GNORM && a.head_dim != 128) PB_FAIL(ctx, PB_UNSUPPORTED, "tensor-core gemm: gated norm over heads of %d (128 is built)", a.head_dim);
    if (((uintptr_t)a.x & 15) || (a.ldx & 3)) PB_FAIL(ctx, PB_ERR_ARG, "tensor-core gemm: activations must be 16-byte aligned");
    if (a.nseg < 1 || a.nseg > 4) PB_FAIL(ctx, PB_ERR_ARG, "tensor-core gemm: %d segments", a.nseg);
    for (int sg = 0; sg < a.nseg; sg++) if (!a.seg[sg].wr) PB_FAIL(ctx, PB_UNSUPPORTED, "tensor-core gemm: segment %d has no re-coded copy", sg);
    int ntiles = 0;
    for (int sg = 0; sg < a.nseg; sg++) ntiles += (int)((a.seg[sg].rows + TC_ROWS - 1) / TC_ROWS);
    if (ntiles == 0) return PB_OK;
    const size_t smem = 1024 + (size_t)TC_STAGES * TC_B_BYTES + (size_t)TC_RAW_STAGES * TC_RAW_BYTES;
    // Tokens per CTA and CTAs per tile, by the rounds the SMs need: a CTA walks its columns serially, a wide one takes half as long again per block
    // and twice as long around it (256 tokens of 12352 x 2048: two rounds of narrow ones 47 us, one of wide ones 39); a matrix with
    // fewer tiles than SMs is cut along its columns, and the parts' sums meet at the end (256 tokens of 2048 x 4096: 64 us uncut, 26 in four).
    const int ft = a.form_t > 0 && a.t % a.form_t == 0 && a.form_t % TC_WIDE == 0 ? a.form_t : a.t;
    int nb = TC_NARROW, cut = 1, best = 0;
    for (int w = TC_NARROW; w <= (ft > TC_NARROW ? TC_WIDE : TC_NARROW); w *= 2)
        for (int ks = 1; ks <= 8 && a.cols / 256 % ks == 0 && (ks == 1 || a.cols / 256 / ks >= 2); ks *= 2) {
            const void* k = w == TC_WIDE ? reinterpret_cast<const void*>(pb_gemmtc_iq3s_kernel<true>) : reinterpret_cast<const void*>(pb_gemmtc_iq3s_kernel<false>);
            PB_TRY(pb_ensure_smem_fn(ctx, k, smem));
            const int room = pb_max_clusters(ctx, k, TC_THREADS, smem, ks), rounds = (ntiles * ((ft + w - 1) / w) + room - 1) / room;
            const int cost = rounds * ((w == TC_WIDE ? 12 : 6) + (ks > 1 ? 4 : 0) + a.cols / 256 / ks * (w == TC_WIDE ? 3 : 2));
            if (best == 0 || cost < best) { best = cost; nb = w; cut = ks; }
        }
    const int nblk = (a.t + nb - 1) / nb;
    const size_t need = TC_XT_HEAD + (size_t)nblk * nb * a.cols * 4;
    if ((size_t)a.t * 4 > TC_XT_HEAD || need > PB_XH_BYTES) PB_FAIL(ctx, PB_UNSUPPORTED, "tensor-core gemm: %d tokens of %d columns exceed the %zu-byte operand buffer", a.t, a.cols, (size_t)PB_XH_BYTES);
    {
        PbGemvQParams q;
        memset(&q, 0, sizeof q);
        q.bpr = a.cols / 256; q.x = a.x; q.ldx = a.ldx; q.t = a.t; q.mode = a.mode; q.norm_w = a.norm_w; q.z = a.z; q.ldz = a.ldz; q.head_dim = a.head_dim; q.eps = a.eps;
        pb_launch_k(ctx, pb_xt_prep_kernel, dim3((nblk - 1) * nb + pb_xt_np(a.t, nblk - 1, nb)), dim3(256), (size_t)0, q, nb, ctx->xh_buf);
        ctx->kernels_launched++;
        PB_CUDA(ctx, cudaGetLastError());
    }
    TcParams p;
    memset(&p, 0, sizeof p);
    p.nseg = a.nseg; p.row_bytes = a.cols / 256 * 136; p.cols = a.cols; p.t = a.t; p.xt = ctx->xh_buf; p.y = a.y; p.ldy = a.ldy; p.accumulate = a.accumulate; p.status = ctx->dev_status;
    for (int sg = 0, n = 0; sg < a.nseg; sg++) {
        p.seg[sg].w = a.seg[sg].wr; p.seg[sg].rows = (int)a.seg[sg].rows; p.seg[sg].yoff = (int)a.seg[sg].yoff; p.seg[sg].chunk0 = n;
        n += (int)((a.seg[sg].rows + TC_ROWS - 1) / TC_ROWS);
    }
    p.ntiles = ntiles; p.ks = cut;
    if (nb == TC_WIDE) pb_launch_kc(ctx, pb_gemmtc_iq3s_kernel<true>, dim3(ntiles * cut, nblk), dim3(TC_THREADS), smem, cut, p);
    else pb_launch_kc(ctx, pb_gemmtc_iq3s_kernel<false>, dim3(ntiles * cut, nblk), dim3(TC_THREADS), smem, cut, p);
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    return PB_OK;
}
