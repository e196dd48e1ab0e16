// Gated DeltaNet decode step: depthwise causal conv1d + SiLU, q/k L2 norm, decay / beta gates,
// delta-rule state update and readout, fused in one kernel.
//
// Restates linear_core of the reference (src/model/qwen4exp_gguf.rs:1624-1673; GPU twins
// k_conv / k_delta, src/model/qn_cube.rs:2753-2839).  The gated RMSNorm that follows the
// readout (:1667) needs the whole 128-wide head, so it lives in the prologue of the output
// projection (PB_ACT_GNORM in pb_gemvq.cu).
//
// Work split: one CTA per (sequence, V head, slice of 32 state columns).  The f32 state
// S[h][i][j] (dk x dv per head, 64 KB) is read once and written once; a warp owns 16 rows i,
// a lane one column j, so every row access is a coalesced 128-byte line and the two
// reductions over i (S^T k and S^T q) are 16 FMAs per lane plus a sum across the 8 warps in
// shared memory.  The conv history is a 4-slot ring ([slot][channel], slot = position mod
// conv_k), so no CTA ever writes a slot another CTA reads in the same step.
#include "pb_deltanet.cuh"

#include <stdio.h>

struct PbDeltaCtaPolicy {
    __device__ static __forceinline__ void sync() { __syncthreads(); }
    __device__ __forceinline__ void wait_inputs() {}   // the kernel waited for its predecessor before anything was read
};

// grid (nv * dv / (DN_COLS * NS), batch).  NS = column slices of 32 one CTA walks in turn (1: most CTAs, shortest
// latency; dv / 32: the conv, norm and gate phases run once per head instead of once per slice, which pays when
// there are thousands of CTAs)
template <int RPW, int NS>
__global__ void __launch_bounds__(DN_THREADS) pb_deltanet_kernel(const PbDeltaParams p) {
    const int splits = p.dv / (DN_COLS * NS);
    const int h = blockIdx.x / splits, j0 = (blockIdx.x % splits) * DN_COLS * NS;
    const int b = blockIdx.y, tid = threadIdx.x;
    const bool st_first = tid == 0 && blockIdx.x == 0 && blockIdx.y == 0, st_last = tid == 0 && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1;
    pb_stamp(p.stamps, 0, st_first); pb_stamp(p.stamps, 6, st_last);
    pb_pdl_wait();
    pb_pdl_trigger();
    extern __shared__ float sm[];
    __shared__ float nrm[2];
    PbDeltaCtaPolicy pol;
    // (requesting the state early pays only with few sequences: with thousands of CTAs the SM already overlaps them,
    // and holding the slice through the first phases costs more than it hides)
    pb_deltanet_unit<RPW, NS>(p, p.pos[b], h, j0, b, tid, gridDim.y <= 4, sm, nrm, pol, p.stamps, st_first);
    pb_stamp(p.stamps, 5, st_first); pb_stamp(p.stamps, 7, st_last);
}

// ---- T consecutive tokens of ONE sequence (a prefill chunk, a verify window), in two kernels ----
//
// Only the state recurrence is sequential in the tokens.  Everything that feeds it -- conv + SiLU, L2 norms, gates -- is made for all
// tokens at once by pb_deltanet_inputs_kernel; pb_deltanet_run_kernel then walks the tokens with its slice of S in registers.
// What bounds the walk is the latency of one token: two dot products over dk, their reduction, the update.  A column of S is held by four
// lanes (dk / 4 rows each, so the reduction is two shuffles), both dots run over the state as the previous token left it
// (S'^T q = g (S^T q) + delta (k.q), with k.q made beforehand), the multiply-adds are packed pairs, and no barrier is taken per token:
// the inputs of PB_DR_TB tokens at a time are brought into shared memory behind the computation.  256 tokens of 32 heads of 128 x 128:
// 535 us as one kernel with six barriers per token, now 20 us for the inputs and 86 for the walk.
// The reference loops the tokens inside k_delta_m (src/model/qn_cube.rs:2839-2913).
#define PB_DR_TB 8       // tokens per block of inputs

// scratch rows of the run: normalized q | k per K head, conv'd v, {decay, beta} per V head, k.q per K head; for runs in blocks of eight
// tokens per block and K head the products k_t.k_s and q_t.k_s (s <= t, the rest zero)
struct PbDeltaRun { float* qk; float* v; float2* gb; float* kq; float* gram; };

// TB tokens per CTA: 8 for a chunk (the taps of neighbouring tokens are loaded once), 1 for a window, whose few tokens then spread over the GPU.
// grid (token blocks, nk + nv), dk (q / k heads) or dv (v heads) threads at most 256 -- one channel (or one of q and one of k) per thread
template <int TB>
__global__ void __launch_bounds__(256) pb_deltanet_inputs_kernel(const PbDeltaParams p, int T, const PbDeltaRun r) {
    constexpr int K = 4;                                    // conv taps (checked by the launcher)
    const int nk = p.nk, nv = p.nv, dk = p.dk, dv = p.dv, ch = 2 * nk * dk + nv * dv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int t0 = blockIdx.x * TB, t1 = min(T, t0 + TB);
    const bool isv = (int)blockIdx.y >= nk;
    const int head = isv ? (int)blockIdx.y - nk : (int)blockIdx.y;
    __shared__ float red[2][3][8];
    constexpr int LD = 130;                                 // rows of a block's k and q, 4 banks apart
    __shared__ __align__(16) double kqs[TB == 8 ? 2 : 1][TB == 8 ? 8 * LD : 1];
    const int n = isv ? dv : dk;
    const bool live = tid < n;
    const int c0 = isv ? 2 * nk * dk + head * dv + tid : head * dk + tid, c1 = nk * dk + head * dk + tid;   // q and k channel, or the v channel
    float w0[K], w1[K];
    if (live) {
#pragma unroll
        for (int k = 0; k < K; k++) { w0[k] = p.conv_w[(size_t)c0 * K + k]; w1[k] = isv ? 0.f : p.conv_w[(size_t)c1 * K + k]; }
    }
    pb_pdl_wait();
    pb_pdl_trigger();
    const int64_t pos0 = p.pos[0];
    // inputs of tokens t0 - 3 .. t1 - 1: rows of proj, before token 0 the ring slots of their positions
    float x0[TB + K - 1], x1[TB + K - 1];
#pragma unroll
    for (int i = 0; i < TB + K - 1; i++) {
        const int j = t0 + i - (K - 1);
        x0[i] = x1[i] = 0.f;
        if (live && j < t1) {
            const float* src = j >= 0 ? p.proj + (size_t)j * p.ldp : p.conv + (size_t)((pos0 + j + K) % K) * ch;
            x0[i] = src[c0];
            if (!isv) x1[i] = src[c1];
        }
    }
#pragma unroll
    for (int i = 0; i < TB; i++) {
        const int j = t0 + i;
        if (j >= t1) break;
        // o = w[K-1] * cur + sum_{k < K-1} w[k] * hist[k], then SiLU   (:1645)
        float a = 0.f, b = 0.f;
        if (live) {
            a = w0[K - 1] * x0[i + K - 1];
#pragma unroll
            for (int k = 0; k < K - 1; k++) a = fmaf(w0[k], x0[i + k], a);
            a = pb_silu(a);
            if (!isv) {
                b = w1[K - 1] * x1[i + K - 1];
#pragma unroll
                for (int k = 0; k < K - 1; k++) b = fmaf(w1[k], x1[i + k], b);
                b = pb_silu(b);
            }
        }
        if (isv) {
            if (live) r.v[(size_t)j * nv * dv + head * dv + tid] = a;
            if (tid == 0) {   // gates (:1660)
                const float* pr = p.proj + (size_t)j * p.ldp + ch + nv * dv;
                r.gb[(size_t)j * nv + head] = make_float2(expf(pb_softplus(pr[nv + head] + p.dt[head]) * p.a[head]), pb_sigm(pr[head]));
            }
        } else {
            // x * (1/sqrt(sum x^2 + 1e-6)), q also times 1/sqrt(dk)  (:1650-1651); and k.q of the normalized vectors
            const float sq = pb_warp_sum(a * a), sk = pb_warp_sum(b * b), sd = pb_warp_sum(a * b);
            float (&rd)[3][8] = red[i & 1];
            if (lane == 0) { rd[0][warp] = sq; rd[1][warp] = sk; rd[2][warp] = sd; }
            __syncthreads();
            float tq = 0.f, tk = 0.f, td = 0.f;
            for (int w = 0; w < nw; w++) { tq += rd[0][w]; tk += rd[1][w]; td += rd[2][w]; }
            const float fq = 1.0f / sqrtf(tq + 1e-6f) * (1.0f / sqrtf((float)dk)), fk = 1.0f / sqrtf(tk + 1e-6f);
            float* dst = r.qk + ((size_t)j * nk + head) * 2 * dk;
            if (live) { dst[tid] = a * fq; dst[dk + tid] = b * fk; }
            if (TB == 8 && r.gram) { kqs[0][i * LD + tid] = b * fk; kqs[1][i * LD + tid] = a * fq; }   // (dk = 128: every thread has a channel)
            if (tid == 0) r.kq[(size_t)j * nk + head] = td * fq * fk;
        }
    }
    if (TB == 8 && r.gram && !isv) {
        __syncthreads();
        const int which = tid >> 6, t = (tid >> 3) & 7, s = tid & 7;   // 128 threads: k_t.k_s and q_t.k_s
        // in 64 bits, rounded once: a product enters up to seven corrections and outputs, and its rounding with it (1024 tokens of 16 K heads: 66 us with
        // sums in f32, 70 so)
        double d = 0.0;
        if (s <= t && t0 + t < t1) {
            double u[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
            for (int c = 0; c < 128; c += 4) {
                const double2 x0 = *reinterpret_cast<const double2*>(&kqs[which][t * LD + c]), x1 = *reinterpret_cast<const double2*>(&kqs[which][t * LD + c + 2]);
                const double2 y0 = *reinterpret_cast<const double2*>(&kqs[0][s * LD + c]), y1 = *reinterpret_cast<const double2*>(&kqs[0][s * LD + c + 2]);
                u[0] = fma(x0.x, y0.x, u[0]); u[1] = fma(x0.y, y0.y, u[1]); u[2] = fma(x1.x, y1.x, u[2]); u[3] = fma(x1.y, y1.y, u[3]);
            }
            d = (u[0] + u[1]) + (u[2] + u[3]);
        }
        r.gram[((size_t)blockIdx.x * nk + head) * 128 + tid] = (float)d;
    }
}


// grid nv * dv / DN_COLS, 128 threads: lane = 4 * column + part; part r holds rows 16 m + 4 r + {0..3} of its column
template <int DK, bool CK>
__global__ void __launch_bounds__(128) pb_deltanet_run_kernel(const PbDeltaParams p, int T, const PbDeltaRun r, const PbDeltaCk ck) {
    constexpr int K = 4, NM = DK / 16, ROW = 2 * DK + DN_COLS + 4;   // floats of one token's inputs: q | k | v | decay, beta, k.q
    const int nk = p.nk, nv = p.nv, dv = p.dv;
    const int splits = dv / DN_COLS, h = blockIdx.x / splits, j0 = (blockIdx.x % splits) * DN_COLS, kh = h % nk;
    const int tid = threadIdx.x, lane = tid & 31, part = lane & 3, col = (tid >> 5) * 8 + (lane >> 2);
    const int ch = 2 * nk * DK + nv * dv;
    __shared__ __align__(16) float in[2][PB_DR_TB][ROW];
    pb_pdl_wait();
    pb_pdl_trigger();
    auto fetch = [&](int t0, int buf) {
        const int n = min(PB_DR_TB, T - t0);
        constexpr int PQ = 2 * DK / 4, PV = DN_COLS / 4;
        for (int i = tid; i < n * (PQ + PV); i += 128) {
            const int t = i / (PQ + PV), c = i - t * (PQ + PV);
            const float* src = c < PQ ? r.qk + ((size_t)(t0 + t) * nk + kh) * 2 * DK + 4 * c : r.v + (size_t)(t0 + t) * nv * dv + h * dv + j0 + 4 * (c - PQ);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(pb_smem_u32(&in[buf][t][4 * c])), "l"(src) : "memory");
        }
        if (tid < 3 * n) {
            const int t = tid / 3, c = tid - 3 * t;
            const float* src = c < 2 ? reinterpret_cast<const float*>(r.gb + (size_t)(t0 + t) * nv + h) + c : r.kq + (size_t)(t0 + t) * nk + kh;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(pb_smem_u32(&in[buf][t][2 * DK + DN_COLS + c])), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    float* S = p.ssm + ((size_t)h * DK) * dv + j0 + col;
    unsigned long long s[2 * NM];
#pragma unroll
    for (int m = 0; m < NM; m++) {
        const float* c = S + (size_t)(16 * m + 4 * part) * dv;
        s[2 * m] = pb_f2(c[0], c[dv]); s[2 * m + 1] = pb_f2(c[2 * (size_t)dv], c[3 * (size_t)dv]);
    }
    auto store = [&](float* base) {
#pragma unroll
        for (int m = 0; m < NM; m++) {
            float* c = base + (size_t)(16 * m + 4 * part) * dv;
            const float2 a = pb_f2_get(s[2 * m]), b = pb_f2_get(s[2 * m + 1]);
            c[0] = a.x; c[dv] = a.y; c[2 * (size_t)dv] = b.x; c[3 * (size_t)dv] = b.y;
        }
    };
    int buf = 0;
    for (int t0 = 0; t0 < T; t0 += PB_DR_TB, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                    // this block's inputs have landed; the other buffer is free
        if (t0 + PB_DR_TB < T) fetch(t0 + PB_DR_TB, buf ^ 1);
        const int n = min(PB_DR_TB, T - t0);
        // k and q of a token are read from shared memory while the token before it is computed
        unsigned long long k2[2 * NM], q2[2 * NM];
        auto load = [&](int t, unsigned long long (&kk)[2 * NM], unsigned long long (&qq)[2 * NM]) {
            const float* x = in[buf][t] + 4 * part;
#pragma unroll
            for (int m = 0; m < NM; m++) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + 16 * m), b = *reinterpret_cast<const ulonglong2*>(x + DK + 16 * m);
                qq[2 * m] = a.x; qq[2 * m + 1] = a.y; kk[2 * m] = b.x; kk[2 * m + 1] = b.y;
            }
        };
        load(0, k2, q2);
#pragma unroll 2
        for (int t = 0; t < n; t++) {
            const float* x = in[buf][t];
            const float g = x[2 * DK + DN_COLS], bt = x[2 * DK + DN_COLS + 1], kq = x[2 * DK + DN_COLS + 2], v = x[2 * DK + col];
            unsigned long long a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0}, kn[2 * NM], qn[2 * NM];   // zeros: pairs of f32 0
#pragma unroll
            for (int i = 0; i < 2 * NM; i++) { a[i & 3] = pb_fma2(s[i], k2[i], a[i & 3]); b[i & 3] = pb_fma2(s[i], q2[i], b[i & 3]); }
            load(t + 1 < n ? t + 1 : t, kn, qn);
            const float2 ax = pb_f2_get(pb_add2(pb_add2(a[0], a[1]), pb_add2(a[2], a[3]))), bx = pb_f2_get(pb_add2(pb_add2(b[0], b[1]), pb_add2(b[2], b[3])));
            float mem = ax.x + ax.y, oq = bx.x + bx.y;
            mem += __shfl_xor_sync(0xffffffffu, mem, 1); oq += __shfl_xor_sync(0xffffffffu, oq, 1);
            mem += __shfl_xor_sync(0xffffffffu, mem, 2); oq += __shfl_xor_sync(0xffffffffu, oq, 2);
            const unsigned long long g2 = pb_f2(g, g);
#pragma unroll
            for (int i = 0; i < 2 * NM; i++) s[i] = pb_mul2(s[i], g2);
            const float delta = (v - g * mem) * bt;         // mem_j = sum_i (g S[i][j]) k_i   (:1663)
            const unsigned long long d2 = pb_f2(delta, delta);
#pragma unroll
            for (int i = 0; i < 2 * NM; i++) s[i] = pb_fma2(k2[i], d2, s[i]);
            const int j = t0 + t;
            if (part == 0) p.out[(size_t)j * p.ldo + h * dv + j0 + col] = fmaf(delta, kq, g * oq);   // readout before the gated norm
            if (CK && j < 8 && j + 1 < T && ck.ssm[j]) store(ck.ssm[j] + ((size_t)h * DK) * dv + j0 + col);   // rollback checkpoint after token j
#pragma unroll
            for (int i = 0; i < 2 * NM; i++) { k2[i] = kn[i]; q2[i] = qn[i]; }
        }
    }
    store(S);
    // the conv ring keeps the last K inputs, a checkpoint the K - 1 inputs the next token's conv reads, at their ring slots.  Channels:
    // this slice's v columns; q and k of a K head by the first slice of the first V head that reads it
    const int64_t pos0 = p.pos[0];
    const int nel = DN_COLS + (h == kh && j0 == 0 ? 2 * DK : 0);
    for (int i = tid; i < nel; i += 128) {
        const int c = i < DN_COLS ? 2 * nk * DK + h * dv + j0 + i : (i - DN_COLS < DK ? kh * DK + i - DN_COLS : nk * DK + kh * DK + i - DN_COLS - DK);
        float before[K - 1];                                // inputs at positions pos0 - 3 .. pos0 - 1
#pragma unroll
        for (int k = 0; k < K - 1; k++) before[k] = p.conv[(size_t)((pos0 + 1 + k) % K) * ch + c];
        for (int j = 0; CK && j < 8 && j + 1 < T; j++)
            if (ck.conv[j])
#pragma unroll
                for (int k = 0; k < K - 1; k++) {
                    const int jj = j - (K - 2) + k;
                    ck.conv[j][(size_t)((pos0 + jj + K) % K) * ch + c] = jj >= 0 ? p.proj[(size_t)jj * p.ldp + c] : before[jj + K - 1];
                }
        for (int j = max(0, T - K); j < T; j++) p.conv[(size_t)((pos0 + j) % K) * ch + c] = p.proj[(size_t)j * p.ldp + c];
    }
}

// The same walk in blocks of eight tokens.  Inside a block only the eight corrections of a column depend on each other:
//   g_t S_{t-1}^T k_t = G_t (S_0^T k_t) + sum_{s<t} (G_t / G_s) (k_s.k_t) delta_s,     G_t = g_0 .. g_t
// so the sixteen products S_0^T k_t and S_0^T q_t of a block are formed from the state as the block found it, without waiting for one another,
// then a triangular system of eight unknowns per column is solved by substitution, and the state takes its eight rank-one updates at once.  A
// warp holds eight columns, its lanes eight groups of sixteen rows x four pairs of columns; k of the block stays in registers from the products to the
// update.  What bounds it: the instructions of one warp per scheduler and the reads of k and q from shared memory (the token-by-token walk: the
// latency of one token).  1024 tokens of 32 heads of 128 x 128: 344 us token by token, 246 in blocks.
// A token's values never enter an earlier token's: the sums run over s < t only.
#define DB_C 8               // tokens of a block
__global__ void __launch_bounds__(128, 1) pb_deltanet_block_kernel(const PbDeltaParams p, int T, const PbDeltaRun r) {
    constexpr int DK = 128, C = DB_C, NT = 128;
    const int nk = p.nk, nv = p.nv, dv = p.dv;
    const int splits = dv / DN_COLS, h = blockIdx.x / splits, j0 = (blockIdx.x % splits) * DN_COLS, kh = h % nk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rg = lane >> 2, cp = lane & 3;
    struct __align__(16) In { float qk[C][2 * DK]; float v[C][DN_COLS]; float gram[2 * C * C]; float2 gb[C]; };
    __shared__ In in[2];
    __shared__ __align__(16) float mat[2][C][C], dec[2][C];            // decayed products (k.k, q.k); G_t and G_7 / G_s
    __shared__ __align__(16) float ab[4][2][8][C], del[4][C][8];       // per warp: S^T k and S^T q of its columns, corrections
    pb_pdl_wait();
    pb_pdl_trigger();
    auto fetch = [&](int t0, int buf) {
        const int n = min(C, T - t0);
        constexpr int PQ = 2 * DK / 4, PV = DN_COLS / 4;
        In& d = in[buf];
        for (int i = tid; i < C * (PQ + PV); i += NT) {
            const int t = i / (PQ + PV), c = i - t * (PQ + PV);
            float* dst = c < PQ ? &d.qk[t][4 * c] : &d.v[t][4 * (c - PQ)];
            if (t < n) {
                const float* src = c < PQ ? r.qk + ((size_t)(t0 + t) * nk + kh) * 2 * DK + 4 * c : r.v + (size_t)(t0 + t) * nv * dv + h * dv + j0 + 4 * (c - PQ);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(pb_smem_u32(dst)), "l"(src) : "memory");
            } else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (tid >= NT - 2 * C * C / 4) { const int i = tid - (NT - 2 * C * C / 4); asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(pb_smem_u32(&d.gram[4 * i])), "l"(r.gram + ((size_t)(t0 / C) * nk + kh) * (2 * C * C) + 4 * i) : "memory"); }
        else if (tid >= NT - 2 * C * C / 4 - C) {
            const int t = tid - (NT - 2 * C * C / 4 - C);
            if (t < n) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(pb_smem_u32(&d.gb[t])), "l"(r.gb + (size_t)(t0 + t) * nv + h) : "memory");
            else d.gb[t] = make_float2(1.f, 0.f);       // past the run: no decay, no correction
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    // the lane's rows 32 j + 4 rg + {0..3}, j = 0..3, of its two columns, as pairs of rows
    float* S = p.ssm + ((size_t)h * DK) * dv + j0 + 8 * warp + 2 * cp;
    unsigned long long s[2][8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = 32 * (i >> 1) + 4 * rg + 2 * (i & 1);
        const float2 a = *reinterpret_cast<const float2*>(S + (size_t)row * dv), b = *reinterpret_cast<const float2*>(S + (size_t)(row + 1) * dv);
        s[0][i] = pb_f2(a.x, b.x); s[1][i] = pb_f2(a.y, b.y);
    }
    int buf = 0;
    for (int t0 = 0; t0 < T; t0 += C, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                    // this block's inputs have landed; the other buffer and the tables are free
        if (t0 + C < T) fetch(t0 + C, buf ^ 1);
        const In& d = in[buf];
        const int n = min(C, T - t0);
        {   // thread (t, which, s): the product decayed from s to t; then G_t and G_7 / G_s
            const int t = tid >> 4, which = (tid >> 3) & 1, q = tid & 7;
            float f = 1.f;
#pragma unroll
            for (int i = 1; i < C; i++) if (i > q && i <= t) f *= d.gb[i].x;
            mat[which][t][q] = f * d.gram[which * C * C + t * C + q];   // (the entries that are read: s < t, or s <= t for q.k)
            if (tid < 2 * C) {
                float e = 1.f;
#pragma unroll
                for (int i = 0; i < C; i++) if (which == 0 ? i <= q : i > q) e *= d.gb[i].x;
                dec[which][q] = e;
            }
        }
        // S_0^T k_t and S_0^T q_t of the lane's rows, all of the block before anything is summed over the lanes
        ulonglong2 k[C][4];
        float v[2][C][2];
#pragma unroll
        for (int t = 0; t < C; t++) {
            ulonglong2 q[4];
#pragma unroll
            for (int j = 0; j < 4; j++) { q[j] = *reinterpret_cast<const ulonglong2*>(&d.qk[t][32 * j + 4 * rg]); k[t][j] = *reinterpret_cast<const ulonglong2*>(&d.qk[t][DK + 32 * j + 4 * rg]); }
#pragma unroll
            for (int c = 0; c < 2; c++) {
                unsigned long long a[2], b[2];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    a[0] = j ? pb_fma2(s[c][2 * j], k[t][j].x, a[0]) : pb_mul2(s[c][0], k[t][0].x); a[1] = j ? pb_fma2(s[c][2 * j + 1], k[t][j].y, a[1]) : pb_mul2(s[c][1], k[t][0].y);
                    b[0] = j ? pb_fma2(s[c][2 * j], q[j].x, b[0]) : pb_mul2(s[c][0], q[0].x); b[1] = j ? pb_fma2(s[c][2 * j + 1], q[j].y, b[1]) : pb_mul2(s[c][1], q[0].y);
                }
                const float2 x = pb_f2_get(pb_add2(a[0], a[1])), y = pb_f2_get(pb_add2(b[0], b[1]));
                v[0][t][c] = x.x + x.y; v[1][t][c] = y.x + y.y;
            }
        }
        {   // sums over the eight row groups (lane bits 2 .. 4): bit 4 keeps k or q, bit 3 half of the tokens, bit 2 a quarter
            const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
            for (int c = 0; c < 2; c++) {
                float w[C], u[C / 2], z[C / 4];
#pragma unroll
                for (int t = 0; t < C; t++) w[t] = (b4 ? v[1][t][c] : v[0][t][c]) + __shfl_xor_sync(0xffffffffu, b4 ? v[0][t][c] : v[1][t][c], 16);
#pragma unroll
                for (int t = 0; t < C / 2; t++) u[t] = (b3 ? w[t + 4] : w[t]) + __shfl_xor_sync(0xffffffffu, b3 ? w[t] : w[t + 4], 8);
#pragma unroll
                for (int t = 0; t < C / 4; t++) z[t] = (b2 ? u[t + 2] : u[t]) + __shfl_xor_sync(0xffffffffu, b2 ? u[t] : u[t + 2], 4);
                *reinterpret_cast<float2*>(&ab[warp][lane >> 4][2 * cp + c][(b3 ? 4 : 0) + (b2 ? 2 : 0)]) = make_float2(z[0], z[1]);
            }
        }
        __syncthreads();                                    // the tables are complete (and the warp's sums)
        // corrections of column `col` of the warp, all of them by each of the column's four lanes: delta_t = (v_t - g_t mem_t) beta_t (:1663).  What the
        // earlier corrections add to a token's memory is summed by itself: taken out of v_t one by one they would each round at
        // v_t's magnitude (16 tokens with decays near 1, readout and state against 64 bits: 9.9e-8 and 10.4e-8 of the result that way, 8.6e-8 and 8.8e-8 so,
        // token by token 9.5e-8 and 8.9e-8)
        const int col = lane & 7, rr = lane >> 3;
        float de[C], m[C][C], av[C], gv[C], sum[C];
        {
            const float4 x = *reinterpret_cast<const float4*>(&ab[warp][0][col][0]), y = *reinterpret_cast<const float4*>(&ab[warp][0][col][4]);
            const float4 g = *reinterpret_cast<const float4*>(&dec[0][0]), e = *reinterpret_cast<const float4*>(&dec[0][4]);
            const float xy[C] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w}, ge[C] = {g.x, g.y, g.z, g.w, e.x, e.y, e.z, e.w};
#pragma unroll
            for (int t = 0; t < C; t++) {
                av[t] = xy[t]; gv[t] = ge[t];
                if (t > 0) { const float4 o = *reinterpret_cast<const float4*>(&mat[0][t][0]); m[t][0] = o.x; m[t][1] = o.y; m[t][2] = o.z; m[t][3] = o.w; }
                if (t > 4) { const float4 o = *reinterpret_cast<const float4*>(&mat[0][t][4]); m[t][4] = o.x; m[t][5] = o.y; m[t][6] = o.z; m[t][7] = o.w; }
            }
        }
#pragma unroll
        for (int t = 0; t < C; t++) {
            float mem = t > 1 ? fmaf(gv[t], av[t], sum[t]) : gv[t] * av[t];
            if (t) mem = fmaf(m[t][t - 1], de[t - 1], mem);        // (the token before is what the chain waits for)
            de[t] = t < n ? (d.v[t][8 * warp + col] - mem) * d.gb[t].y : 0.f;
#pragma unroll
            for (int q = t + 2; q < C; q++) sum[q] = t ? fmaf(m[q][t], de[t], sum[q]) : m[q][0] * de[0];
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {   // each of the column's lanes forms two of the outputs: tokens 2 rr and 2 rr + 1
            const int t = 2 * rr + i;
            const float4 x = *reinterpret_cast<const float4*>(&mat[1][t][0]), y = *reinterpret_cast<const float4*>(&mat[1][t][4]);
            const float w[C] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            float o = w[0] * de[0], own = de[0];
#pragma unroll
            for (int q = 1; q < C; q++) { if (q <= t) o = fmaf(w[q], de[q], o); if (q == t) own = de[q]; }
            o = fmaf(dec[0][t], ab[warp][1][col][t], o);     // (the state's part last)
            if (t < n) p.out[(size_t)(t0 + t) * p.ldo + h * dv + j0 + 8 * warp + col] = o;   // readout before the gated norm
            del[warp][t][col] = own * dec[1][t];
        }
        __syncwarp();
        const float g = dec[0][C - 1];
        const unsigned long long g2 = pb_f2(g, g);
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int i = 0; i < 8; i++) s[c][i] = pb_mul2(s[c][i], g2);
#pragma unroll
        for (int t = 0; t < C; t++) {
            const float2 e = *reinterpret_cast<const float2*>(&del[warp][t][2 * cp]);
            const unsigned long long e2[2] = {pb_f2(e.x, e.x), pb_f2(e.y, e.y)};
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int j = 0; j < 4; j++) { s[c][2 * j] = pb_fma2(k[t][j].x, e2[c], s[c][2 * j]); s[c][2 * j + 1] = pb_fma2(k[t][j].y, e2[c], s[c][2 * j + 1]); }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = 32 * (i >> 1) + 4 * rg + 2 * (i & 1);
        const float2 a = pb_f2_get(s[0][i]), b = pb_f2_get(s[1][i]);
        *reinterpret_cast<float2*>(S + (size_t)row * dv) = make_float2(a.x, b.x);
        *reinterpret_cast<float2*>(S + (size_t)(row + 1) * dv) = make_float2(a.y, b.y);
    }
    // the conv ring keeps the last K inputs.  Channels: this slice's v columns; q and k of a K head by the first slice of the first V head that reads it
    constexpr int K = 4;
    const int ch = 2 * nk * DK + nv * dv;
    const int64_t pos0 = p.pos[0];
    const int nel = DN_COLS + (h == kh && j0 == 0 ? 2 * DK : 0);
    for (int i = tid; i < nel; i += NT) {
        const int c = i < DN_COLS ? 2 * nk * DK + h * dv + j0 + i : (i - DN_COLS < DK ? kh * DK + i - DN_COLS : nk * DK + kh * DK + i - DN_COLS - DK);
        for (int j = max(0, T - K); j < T; j++) p.conv[(size_t)((pos0 + j) % K) * ch + c] = p.proj[(size_t)j * p.ldp + c];
    }
}

// T consecutive tokens of sequence 0; false when the shape is outside what the kernels are built for
bool pb_deltanet_seq_supported(const PbDeltaParams& p) { return p.conv_k == 4 && p.dv % DN_COLS == 0 && p.dv <= 256 && (p.dk == 128 || p.dk == 64 || p.dk == 32); }
size_t pb_deltanet_seq_scratch(const PbDeltaParams& p, int T) { return (size_t)T * (2 * p.nk * p.dk + p.nv * p.dv + 2 * p.nv + p.nk) + (size_t)((T + 7) / 8) * p.nk * 128 + 16; }   // floats
int pb_launch_deltanet_seq(pb_ctx* ctx, const PbDeltaParams& p, int T, float* scratch, const PbDeltaCk* ckp) {
    if (!pb_deltanet_seq_supported(p)) PB_FAIL(ctx, PB_UNSUPPORTED, "deltanet run: dk=%d dv=%d conv_k=%d not supported", p.dk, p.dv, p.conv_k);
    PbDeltaCk ck; memset(&ck, 0, sizeof ck);
    if (ckp) ck = *ckp;
    PbDeltaRun r;
    r.qk = scratch; r.v = r.qk + (size_t)T * 2 * p.nk * p.dk; r.gb = reinterpret_cast<float2*>(r.v + (size_t)T * p.nv * p.dv); r.kq = reinterpret_cast<float*>(r.gb + (size_t)T * p.nv);
    // blocks of eight tokens for the one head size they are built for; verify windows need the state after every token.  From 32 tokens on, where the inputs
    // are made eight tokens at a time anyway: below, making them one by one on many CTAs and walking takes 9 to 10 us less per layer (a pass over three layers,
    // blocks / token by token: 16 tokens 387 / 355 us, 24 465 / 438, 31 516 / 489), from there on as long, and from 64 tokens on blocks are shorter
    const bool blocks = !ckp && T >= PB_DELTA_BLOCKS && p.dk == 128 && p.dv <= 128;
    r.gram = blocks ? reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(r.kq + (size_t)T * p.nk) + 15) & ~(uintptr_t)15) : nullptr;
    const int wide = p.dk > p.dv ? p.dk : p.dv;
    if (T >= PB_DELTA_BLOCKS) pb_launch_k(ctx, pb_deltanet_inputs_kernel<8>, dim3((T + 7) / 8, p.nk + p.nv), dim3((wide + 31) & ~31), (size_t)0, p, T, r);
    else pb_launch_k(ctx, pb_deltanet_inputs_kernel<1>, dim3(T, p.nk + p.nv), dim3((wide + 31) & ~31), (size_t)0, p, T, r);
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    const dim3 grid(p.nv * (p.dv / DN_COLS));
    if (blocks) {
        // one CTA per SM, by shared memory that it does not use: started while the inputs' CTAs leave, two often met on one SM and took half as long again
        const size_t apart = (size_t)96 << 10;
        PB_TRY(pb_ensure_smem(ctx, pb_deltanet_block_kernel, apart));
        pb_launch_k(ctx, pb_deltanet_block_kernel, grid, dim3(128), apart, p, T, r);
        ctx->kernels_launched++;
        PB_CUDA(ctx, cudaGetLastError());
        return PB_OK;
    }
#define GO(DK) { if (ckp) pb_launch_k(ctx, pb_deltanet_run_kernel<DK, true>, grid, dim3(128), (size_t)0, p, T, r, ck); else pb_launch_k(ctx, pb_deltanet_run_kernel<DK, false>, grid, dim3(128), (size_t)0, p, T, r, ck); }
    if (p.dk == 128) GO(128) else if (p.dk == 64) GO(64) else GO(32)
#undef GO
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    return PB_OK;
}

int pb_launch_deltanet(pb_ctx* ctx, const PbDeltaParams& p0) {
    PbDeltaParams p = p0;
    p.stamps = pb_stamp_slot(ctx, PB_K_DELTANET);
    if (p.dv % DN_COLS || (p.dk != 128 && p.dk != 64 && p.dk != 32) || p.conv_k < 2 || p.conv_k > 8)
        PB_FAIL(ctx, PB_UNSUPPORTED, "deltanet: dk=%d dv=%d conv_k=%d not supported", p.dk, p.dv, p.conv_k);
    // many sequences: a CTA walks all slices of its head (conv / norm / gates once per head)
    const bool whole = p.batch >= 8 && p.dv == 4 * DN_COLS;
    const dim3 grid(p.nv * (whole ? 1 : p.dv / DN_COLS), p.batch);
    const size_t smem = (size_t)(2 * p.dk + DN_COLS * (whole ? 4 : 1) + 8 * DN_COLS) * 4;
#define GO(R)                                                                                             \
    if (whole) pb_launch_k(ctx, pb_deltanet_kernel<R, 4>, dim3(grid), dim3(DN_THREADS), (size_t)(smem), p); \
    else pb_launch_k(ctx, pb_deltanet_kernel<R, 1>, dim3(grid), dim3(DN_THREADS), (size_t)(smem), p);
    if (p.dk == 128) { GO(16) } else if (p.dk == 64) { GO(8) } else { GO(4) }
#undef GO
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    return PB_OK;
}
