// Tensor-core core for quantized weights that meet a few tokens: warp-level mma.sync m16n8k16, f16 x f16 -> f32.
//
// A warp owns a tile of 16 weight rows over a run of 256-column blocks.  No warp waits for another: the weights of a block come into the
// warp's own ring of shared-memory stages by asynchronous copies issued two blocks ahead, are decoded straight into the A operand, and meet
// the tokens' activations, which the CTA prepared once in shared memory as B operands.
//
//   - Lane (g, q) = (lane >> 2, lane & 3) holds the 64 weights of quarter q of row g of the tile's two halves of eight rows.  The
//     contraction index is permuted so that the four k of an mma that a lane holds are weights of its own quarter; A and B use the same
//     permutation.
//   - Weights enter as f16 integers (code times integer sub-block multiplier, at most 2048: exact), the f16 block scale d is applied in f32 to
//     the sum over the block (PB_H_DIRECT, PB_H_FOLD); formats whose scales do not fold (Q8_0, Q6_K, ..) enter as the f16 high and low
//     parts of the scaled weight, 22 significant bits (PB_H_SPLIT).
//   - Activations are scaled by a power of two per token and block so that the largest lies in [2^9, 2^11), and split into f16 high and low parts
//     (22 significant bits); column 2 j of an n-tile is the high part of token j, column 2 j + 1 its low part.
//   - A token's columns do not depend on the other tokens: the result of a token is the same however tokens are grouped.
#pragma once
#include "pb_stream.cuh"
#include <cuda_fp16.h>

__device__ __forceinline__ void pb_hmma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same with a zero accumulator in
__device__ __forceinline__ void pb_hmma0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ __half2 pb_as_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t pb_as_u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// (w & mask) | bits in one logic operation
__device__ __forceinline__ uint32_t pb_and_or(uint32_t w, uint32_t mask, uint32_t bits) {
    uint32_t d; asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(w), "r"(mask), "r"(bits)); return d;
}
// small non-negative integer (< 1024) in both halves of an f16 pair: the exponent of 1024 makes the mantissa the integer itself
__device__ __forceinline__ __half2 pb_h2_int(uint32_t n) { return __hsub2(pb_as_h2((n * 0x00010001u) | 0x64006400u), pb_as_h2(0x64006400u)); }
// activations in shared memory are rewritten between phases of a kernel: these loads stay where they are written
__device__ __forceinline__ uint4 pb_ldsa128(uint32_t a) { uint4 v; asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t pb_ldsa32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint2 pb_ldsa64(uint32_t a) { uint2 v; asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); return v; }

enum { PB_H_DIRECT = 0,   // 4-bit codes decoded by the nibble
       PB_H_FOLD = 1,     // int8 values, integer multipliers folded into the weights
       PB_H_SPLIT = 2 };  // int8 values, scaled weights as high + low parts
template <int FMT> __host__ __device__ constexpr int pb_h_mode() {
    return FMT == PB_T_IQ3S_N4 || FMT == PB_T_Q4_K ? PB_H_DIRECT : (FMT == PB_T_IQ3_S || FMT == PB_T_IQ2_XS ? PB_H_FOLD : PB_H_SPLIT);
}
// a minimum per 32 weights, which meets the group sums of the activations in one more mma
template <int FMT> __host__ __device__ constexpr bool pb_h_offs() { return FMT == PB_T_Q4_K || FMT == PB_T_Q5_K; }
// order of the k index: words of eight consecutive weights as (0 2)(4 6)(1 3)(5 7), or (Q4_K) of four weights of each of the quarter's two groups
template <int FMT> __host__ __device__ constexpr bool pb_h_twin() { return FMT == PB_T_Q4_K; }

// ---------------------------------------------------------------- weights of one block of a tile -> a stage
// A tile is two halves of eight rows (they may belong to different matrices).
struct PbHTile { const uint8_t *a, *b; int la, lb; };   // first row of each half, last valid row of each (0 .. 7)
struct PbHGeom { int row_bytes, step_bytes, npiece, pitch, stage_bytes; };   // bytes of a row, of a block of 256 columns; 16-byte pieces per row of a stage, its row pitch, its size
template <int FMT> __host__ __device__ constexpr bool pb_h_grouped() { return FMT == PB_T_IQ3S_N4; }   // rows in groups of eight (pb_repack.cu)
template <int FMT>
static inline PbHGeom pb_h_geom(int cols) {
    int el, bs;
    pb_geom(FMT, &el, &bs);
    PbHGeom h;
    h.row_bytes = cols / el * bs; h.step_bytes = 256 / el * bs;
    if (pb_h_grouped<FMT>()) { h.npiece = 68; h.pitch = 136; h.stage_bytes = 2 * 1088; }
    else if (h.step_bytes % 16 == 0 && h.row_bytes % 16 == 0) { h.npiece = h.step_bytes / 16; h.pitch = (h.npiece | 1) * 16; h.stage_bytes = 16 * h.pitch; }
    else { h.npiece = (h.step_bytes + 14 + 15) / 16; h.pitch = (h.npiece | 1) * 16; h.stage_bytes = 16 * h.pitch; }   // an odd number of 16-byte words: the rows start on different banks
    return h;
}
__device__ __forceinline__ void pb_h_cp16(uint32_t dst, const uint8_t* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
// rows start at any even byte: the copy covers the 16-byte pieces around them and keeps their alignment
template <int FMT>
__device__ __forceinline__ void pb_h_stage(uint32_t stage, const PbHTile& t, const PbHGeom& h, int blk, int lane) {
    if constexpr (pb_h_grouped<FMT>()) {
        const uint8_t *a = t.a + blk * 1088 + 16 * lane, *b = t.b + blk * 1088 + 16 * lane;
        stage += 16 * lane;
        pb_h_cp16(stage, a); pb_h_cp16(stage + 512, a + 512); pb_h_cp16(stage + 1088, b); pb_h_cp16(stage + 1600, b + 512);
        if (lane < 8) pb_h_cp16(stage + (lane < 4 ? 1024 : 2112 - 64), lane < 4 ? a + 1024 : b + 960);   // the rows' heads: 64 bytes of each half
    } else {
        for (int i = lane; i < 16 * h.npiece; i += 32) {
            const int r = i / h.npiece, c = i - r * h.npiece;
            const uint8_t* p = (r < 8 ? t.a + (size_t)min(r, t.la) * h.row_bytes : t.b + (size_t)min(r - 8, t.lb) * h.row_bytes) + (size_t)blk * h.step_bytes;
            pb_h_cp16(stage + (uint32_t)(r * h.pitch + 16 * c), p - (reinterpret_cast<uintptr_t>(p) & 15) + 16 * c);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// ---------------------------------------------------------------- nibble formats: the lane's bytes of a block
template <int FMT> struct PbHRaw;
template <> struct PbHRaw<PB_T_IQ3S_N4> {
    uint4 c0, c1; uint2 h;
    __device__ __forceinline__ void load(uint32_t p, int g, int q) {   // p = the half's block
        const uint32_t a = p + (uint32_t)((4 * g + q) * 16);
        c0 = pb_ldsa128(a); c1 = pb_ldsa128(a + 512); h = pb_ldsa64(p + 1024 + 8 * g);
    }
};
template <> struct PbHRaw<PB_T_Q4_K> {
    uint4 c0, c1, h;
    __device__ __forceinline__ void load(uint32_t p, int, int q) {         // p = the row's block
        h = pb_ldsa128(p); c0 = pb_ldsa128(p + 16 + 32 * q); c1 = pb_ldsa128(p + 32 + 32 * q);
    }
};
// decoder over the raw registers: word u -> four f16 pairs.  A nibble left where it lies in its 16-bit half is a subnormal f16, c 2^-24 or
// c 2^-20: one mask and one fused multiply-add give 2^-14 times the integer weight, exactly (every product and sum is a multiple of 2^-14 below
// 2^-4, and every weight that is not zero a normal number); the block's factor takes the 2^14 back.  Nine instructions for eight weights; with the
// nibble in the mantissa of 1024 or 64 and the offset subtracted first it was thirteen (2 tokens x 151936 rows of IQ3_S 47 us, 41 so;
// Q4_K 70 and 66).
#define PB_H_UNIT 16384.0f
template <int FMT> struct PbHDec;
template <> struct PbHDec<PB_T_IQ3S_N4> {
    __half2 lo[2], hi[2], off[2];   // m 2^11, m 2^7 and -15 m 2^-14 of the quarter's two groups, m = 1 + 2 s <= 31
    __device__ __forceinline__ void head(const PbHRaw<PB_T_IQ3S_N4>& r, int q) {
        const uint32_t sc = r.h.y >> (8 * q);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const __half2 s = pb_h2_int((sc >> (4 * i)) & 0xF);
            lo[i] = __hfma2(s, pb_as_h2(0x6C006C00u), pb_as_h2(0x68006800u));     // 4096 s + 2048
            hi[i] = __hfma2(s, pb_as_h2(0x5C005C00u), pb_as_h2(0x58005800u));     // 256 s + 128
            off[i] = __hfma2(s, pb_as_h2(0x97809780u), pb_as_h2(0x93809380u));    // -30 2^-14 s - 15 2^-14
        }
    }
    __device__ static __forceinline__ float d(const PbHRaw<PB_T_IQ3S_N4>& r) { return pb_h2f((uint16_t)(r.h.x & 0xFFFF)); }
    __device__ static __forceinline__ float dmin(const PbHRaw<PB_T_IQ3S_N4>&) { return 0.f; }
    __device__ static __forceinline__ uint32_t offs(const PbHRaw<PB_T_IQ3S_N4>&, int) { return 0u; }
    __device__ __forceinline__ uint32_t centre() const { return 0u; }
    // (2 c - 15) m
    __device__ __forceinline__ void word(const PbHRaw<PB_T_IQ3S_N4>& r, int u, uint32_t (&o)[4]) const {
        const uint4& c = u < 4 ? r.c0 : r.c1;
        const uint32_t w = (u & 3) == 0 ? c.x : ((u & 3) == 1 ? c.y : ((u & 3) == 2 ? c.z : c.w)), w8 = w >> 8;
        o[0] = pb_as_u32(__hfma2(pb_as_h2(w & 0x000F000Fu), lo[u >> 2], off[u >> 2]));
        o[1] = pb_as_u32(__hfma2(pb_as_h2(w & 0x00F000F0u), hi[u >> 2], off[u >> 2]));
        o[2] = pb_as_u32(__hfma2(pb_as_h2(w8 & 0x000F000Fu), lo[u >> 2], off[u >> 2]));
        o[3] = pb_as_u32(__hfma2(pb_as_h2(w8 & 0x00F000F0u), hi[u >> 2], off[u >> 2]));
    }
};
template <> struct PbHDec<PB_T_Q4_K> {
    __half2 lo, hi, off[2];  // 2^10 scale of the first group (low nibbles), 2^6 scale of the second (high nibbles), -8 2^-14 scale of each
    // scale_min_k4 (gguf_q.rs:62-64) of groups 2 q and 2 q + 1: both groups' values in bytes 0 and 1
    __device__ static __forceinline__ uint32_t scales(const uint4& h, int q) {
        return q < 2 ? (h.y >> (16 * q)) & 0x3F3Fu : ((h.w >> (16 * (q - 2))) & 0x0F0Fu) | (((h.y >> (16 * (q - 2))) & 0xC0C0u) >> 2);
    }
    __device__ __forceinline__ void head(const PbHRaw<PB_T_Q4_K>& r, int q) {
        const uint32_t s2 = scales(r.h, q);
        const __half2 s0 = pb_h2_int(s2 & 0xFF), s1 = pb_h2_int((s2 >> 8) & 0xFF), k8 = pb_as_h2(0x90009000u);   // k8 = -8 2^-14
        lo = __hmul2(s0, pb_as_h2(0x64006400u)); hi = __hmul2(s1, pb_as_h2(0x54005400u));
        off[0] = __hmul2(s0, k8); off[1] = __hmul2(s1, k8);
    }
    __device__ static __forceinline__ float d(const PbHRaw<PB_T_Q4_K>& r) { return pb_h2f((uint16_t)(r.h.x & 0xFFFF)); }
    __device__ static __forceinline__ float dmin(const PbHRaw<PB_T_Q4_K>& r) { return pb_h2f((uint16_t)(r.h.x >> 16)); }
    // f16 pair of the two groups' integer minima
    __device__ static __forceinline__ uint32_t offs(const PbHRaw<PB_T_Q4_K>& r, int q) {
        const uint32_t m2 = q < 2 ? (r.h.z >> (16 * q)) & 0x3F3Fu : ((r.h.w >> (16 * (q - 2) + 4)) & 0x0F0Fu) | (((r.h.z >> (16 * (q - 2))) & 0xC0C0u) >> 2);
        return pb_as_u32(__hsub2(pb_as_h2((m2 & 0xFF) | ((m2 & 0xFF00) << 8) | 0x64006400u), pb_as_h2(0x64006400u)));
    }
    // f16 pair of 8 x scale of the two groups
    __device__ __forceinline__ uint32_t centre() const { return pb_as_u32(__hmul2(__halves2half2(__low2half(off[0]), __low2half(off[1])), pb_as_h2(0xF400F400u))); }   // off times -2^14
    // (q - 8) scale: codes around zero, so that activations with a mean do not make large sums that the minima then cancel; the 8 scale comes back
    // with the minima
    __device__ __forceinline__ void word(const PbHRaw<PB_T_Q4_K>& r, int u, uint32_t (&o)[4]) const {
        const uint4& c = u < 4 ? r.c0 : r.c1;
        const uint32_t w = (u & 3) == 0 ? c.x : ((u & 3) == 1 ? c.y : ((u & 3) == 2 ? c.z : c.w)), w8 = w >> 8;
        o[0] = pb_as_u32(__hfma2(pb_as_h2(w & 0x000F000Fu), lo, off[0]));
        o[1] = pb_as_u32(__hfma2(pb_as_h2(w8 & 0x000F000Fu), lo, off[0]));
        o[2] = pb_as_u32(__hfma2(pb_as_h2(w & 0x00F000F0u), hi, off[1]));
        o[3] = pb_as_u32(__hfma2(pb_as_h2(w8 & 0x00F000F0u), hi, off[1]));
    }
};

// ---------------------------------------------------------------- activations in shared memory
// Token slot: per block and word u of 8 weights one 128-byte row [high | low][quarter][8 halves]; then per block the inverse prescale (f32); then,
// for formats with minima, per block and quarter the f16 pair of the two groups' sums and what that rounding lost (8 bytes).
template <int FMT> __host__ __device__ constexpr int pb_h_tok_bytes(int cols) { return cols * 4 + ((cols / 256 * 4 + 15) & ~15) + (pb_h_offs<FMT>() ? cols / 256 * 32 : 0); }
__device__ __forceinline__ uint32_t pb_h_scale_off(int bpr) { return (uint32_t)bpr * 1024u; }
__device__ __forceinline__ uint32_t pb_h_sums_off(int bpr) { return (uint32_t)bpr * 1024u + (uint32_t)((bpr * 4 + 15) & ~15); }

// columns of a block that lane (q = lane & 3, u = lane >> 2) prepares: [c0, c0 + 4) and [c1, c1 + 4)
template <int FMT> __device__ __forceinline__ int pb_h_c0(int lane) { return 64 * (lane & 3) + (pb_h_twin<FMT>() ? 4 : 8) * (lane >> 2); }
template <int FMT> __device__ __forceinline__ int pb_h_c1(int lane) { return pb_h_c0<FMT>(lane) + (pb_h_twin<FMT>() ? 32 : 4); }

// A warp's block of a token, eight activations a lane (columns c0 .., c1 ..), times the power of two that puts the block's largest into [2^9, 2^10): f16
// high and low parts as pairs (0 2)(4 6)(1 3)(5 7), or (0 2)(1 3) of each group.  x is scaled in place; the result is the inverse of the power.
template <int FMT>
__device__ __forceinline__ float pb_h_split(float (&x)[8], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
    float m = fmaxf(fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3]))), fmaxf(fmaxf(fabsf(x[4]), fabsf(x[5])), fmaxf(fabsf(x[6]), fabsf(x[7]))));
    m = pb_warp_max(m);
    float p = 1.0f, ip = 1.0f;
    if (m > 6.1e-36f && m < INFINITY) {   // 2^(9 - exponent) and its inverse, built from the exponent bits: both are normal numbers from 2^-117 on (below, zero)
        const int e = (int)((__float_as_uint(m) >> 23) & 0xFF) - 127;
        p = __uint_as_float((uint32_t)(9 - e + 127) << 23); ip = __uint_as_float((uint32_t)(e - 9 + 127) << 23);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] *= p;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int e0 = pb_h_twin<FMT>() ? (k < 2 ? k : k + 2) : (k < 2 ? 4 * k : 4 * (k - 2) + 1);
        const __half2 h = __floats2half2_rn(x[e0], x[e0 + 2]);
        const float2 r = __half22float2(h);
        hi[k] = pb_as_u32(h); lo[k] = pb_as_u32(__floats2half2_rn(x[e0] - r.x, x[e0 + 2] - r.y));
    }
    return ip;
}
// One warp stores block blk of a token: x = the lane's eight activations.
template <int FMT>
__device__ __forceinline__ void pb_h_put(uint8_t* slot, int bpr, int blk, int lane, const float (&x)[8]) {
    const int q = lane & 3, u = lane >> 2;
    constexpr bool twin = pb_h_twin<FMT>();
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = x[i];
    uint32_t hi[4], lo[4];
    const float ip = pb_h_split<FMT>(v, hi, lo);
    if (lane == 0) *reinterpret_cast<float*>(slot + pb_h_scale_off(bpr) + 4 * blk) = ip;
    uint8_t* row = slot + (size_t)blk * 1024 + u * 128 + q * 16;
    *reinterpret_cast<uint4*>(row) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(row + 64) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    if (pb_h_offs<FMT>()) {
        // sums of the quarter's two groups of 32: over the eight lanes u of the quarter (one group each half of the words unless twin)
        float s0 = (v[0] + v[1]) + (v[2] + v[3]), s1 = (v[4] + v[5]) + (v[6] + v[7]);
        if (!twin) { s0 += s1; s1 = u >= 4 ? s0 : 0.f; s0 = u >= 4 ? 0.f : s0; }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
        if (u == 0) {
            const __half2 h = __floats2half2_rn(s0, s1);
            const float2 r = __half22float2(h);
            *reinterpret_cast<uint2*>(slot + pb_h_sums_off(bpr) + blk * 32 + q * 8) = make_uint2(pb_as_u32(h), pb_as_u32(__floats2half2_rn(s0 - r.x, s1 - r.y)));
        }
    }
}
// The lane's addresses of the activations of tokens 4 nt + ..: b = B rows of token (g >> 1), sums = its group sums, scale = prescales of token q
struct PbHLane { uint32_t b, sums, scale, tok4; };
template <int FMT>
__device__ __forceinline__ PbHLane pb_h_lane(uint32_t slot0, int bpr, int lane) {
    const int g = lane >> 2, q = lane & 3;
    const uint32_t tokb = (uint32_t)pb_h_tok_bytes<FMT>(256 * bpr), s = slot0 + (uint32_t)(g >> 1) * tokb;
    PbHLane l;
    l.b = s + (uint32_t)((g & 1) * 64 + q * 16); l.sums = s + pb_h_sums_off(bpr) + 8u * q; l.scale = slot0 + (uint32_t)q * tokb + pb_h_scale_off(bpr); l.tok4 = 4 * tokb;
    return l;
}

// ---------------------------------------------------------------- one block of one tile
// tot[nt][0] = row g of the first half, tot[nt][1] = row g of the second half, token 4 nt + q.
template <int FMT, int NT>
__device__ __forceinline__ void pb_h_add(const float (&acc)[NT][4], int nt, int blk, float fa, float fb, float oa, float ob, const PbHLane& L, float (&tot)[NT][2]) {
    float va = __fadd_rn(__fmul_rn(fa, acc[nt][0]), __fmul_rn(fa, acc[nt][1])), vb = __fadd_rn(__fmul_rn(fb, acc[nt][2]), __fmul_rn(fb, acc[nt][3]));
    if (pb_h_offs<FMT>()) { va += oa; vb += ob; }
    const float s = __uint_as_float(pb_ldsa32(L.scale + (uint32_t)nt * L.tok4 + 4u * blk));
    tot[nt][0] = __fadd_rn(tot[nt][0], __fmul_rn(va, s)); tot[nt][1] = __fadd_rn(tot[nt][1], __fmul_rn(vb, s));
}
// The tensor core adds into its f32 accumulator by truncation, an error that grows with the chain: chains of four mma, added up in rounded f32, keep
// a sum as precise as the integer dot products of the dp4a kernels (2048 columns, relative to |x| |w|: 2e-9; one chain per block: 7e-9).
__device__ __forceinline__ void pb_h_flush(float (&acc)[4], const float (&c)[4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i] += c[i];
}
template <int FMT, int NT>
__device__ __forceinline__ void pb_h_block_nib(uint32_t stage, const PbHGeom& h, int blk, int lane, const PbHLane& L, float (&tot)[NT][2]) {
    const int g = lane >> 2, q = lane & 3;
    PbHRaw<FMT> ra, rb;
    if constexpr (pb_h_grouped<FMT>()) { ra.load(stage, g, q); rb.load(stage + 1088, g, q); }
    else { ra.load(stage + (uint32_t)(g * h.pitch), g, q); rb.load(stage + (uint32_t)((g + 8) * h.pitch), g, q); }
    PbHDec<FMT> wa, wb;
    wa.head(ra, q); wb.head(rb, q);
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) { acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f; }
    if constexpr (NT <= 2) {
        float c[NT][4];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            uint32_t a[4], b[4];
            wa.word(ra, u, a); wb.word(rb, u, b);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint4 x = pb_ldsa128(L.b + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 1024 + u * 128));
                if (u & 1) pb_hmma(c[nt], a[0], b[0], a[1], b[1], x.x, x.y); else pb_hmma0(c[nt], a[0], b[0], a[1], b[1], x.x, x.y);
                pb_hmma(c[nt], a[2], b[2], a[3], b[3], x.z, x.w);
                if (u & 1) pb_h_flush(acc[nt], c[nt]);
            }
        }
    } else {
        // more n-tiles: both words of a chain are decoded first, so that one chain's accumulator is alive at a time
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
            uint32_t a[2][4], b[2][4];
            wa.word(ra, u, a[0]); wb.word(rb, u, b[0]); wa.word(ra, u + 1, a[1]); wb.word(rb, u + 1, b[1]);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint32_t xa = L.b + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 1024 + u * 128);
                const uint4 x = pb_ldsa128(xa), y = pb_ldsa128(xa + 128);
                float c[4];
                pb_hmma0(c, a[0][0], b[0][0], a[0][1], b[0][1], x.x, x.y);
                pb_hmma(c, a[0][2], b[0][2], a[0][3], b[0][3], x.z, x.w);
                pb_hmma(c, a[1][0], b[1][0], a[1][1], b[1][1], y.x, y.y);
                pb_hmma(c, a[1][2], b[1][2], a[1][3], b[1][3], y.z, y.w);
                pb_h_flush(acc[nt], c);
            }
        }
    }
    const float da = PbHDec<FMT>::d(ra), db = PbHDec<FMT>::d(rb);
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        float oa = 0.f, ob = 0.f;
        if (pb_h_offs<FMT>()) {
            uint2 s = pb_ldsa64(L.sums + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 32));
            if (g & 1) s = make_uint2(0u, 0u);         // low columns: the high columns carry both parts of the sums
            const uint32_t ma = PbHDec<FMT>::offs(ra, q), mb = PbHDec<FMT>::offs(rb, q);
            float mc[4] = {0.f, 0.f, 0.f, 0.f};
            pb_hmma(mc, ma, mb, ma, mb, s.x, s.y);
            float cc[4];
            const uint32_t ca = wa.centre(), cb = wb.centre();
            pb_hmma0(cc, ca, cb, ca, cb, s.x, s.y);
            oa = da * cc[0] - PbHDec<FMT>::dmin(ra) * mc[0]; ob = db * cc[2] - PbHDec<FMT>::dmin(rb) * mc[2];
        }
        pb_h_add<FMT, NT>(acc, nt, blk, da * PB_H_UNIT, db * PB_H_UNIT, oa, ob, L, tot);
    }
}

// ---------------------------------------------------------------- int8 formats (the decoders of the dp4a kernels)
// Integer multipliers of a quarter (per 16 weights) and the f32 factor of the whole block
template <int FMT> __device__ __forceinline__ void pb_h_mults(uint32_t p, int qt, float& d, uint32_t (&m)[4]);
template <> __device__ __forceinline__ void pb_h_mults<PB_T_IQ3_S>(uint32_t p, int qt, float& d, uint32_t (&m)[4]) {
    d = pb_h2f((uint16_t)pb_lds16(p));
    const uint32_t sc = pb_lds8(p + 106 + qt);
    m[0] = m[1] = 1 + 2 * (sc & 0xF); m[2] = m[3] = 1 + 2 * (sc >> 4);
}
template <> __device__ __forceinline__ void pb_h_mults<PB_T_IQ2_XS>(uint32_t p, int qt, float& d, uint32_t (&m)[4]) {
    d = pb_h2f((uint16_t)pb_lds16(p)) * 0.125f;              // d (0.5 + s) / 4 = d / 8 (1 + 2 s)
    const uint32_t sc = pb_lds16(p + 66 + 2 * qt);
#pragma unroll
    for (int h = 0; h < 4; h++) m[h] = 1 + 2 * ((sc >> (4 * h)) & 0xF);
}
// Codebook of this core: as the dp4a kernels have it (pb_fill_qtabs), but for IQ2_XS, whose three magnitudes 8, 25, 43 fit a nibble each: one word of
// eight byte selectors per entry, and the signs come from the index bits by arithmetic (pb_h_word_iq2xs).  With eight bytes per entry and the 16-byte rows of a
// sign table the look-ups took two thirds of the shared-memory wavefronts (16 tokens x 151936 rows: 147 us, 129 so).
template <int FMT> __host__ __device__ constexpr uint32_t pb_h_tab_bytes(int rep) { return pb_h_mode<FMT>() == PB_H_DIRECT ? 0u : (FMT == PB_T_IQ2_XS ? 512u * 4u * (uint32_t)rep : pb_tab_bytes<FMT>(rep)); }
template <int FMT>
__device__ __forceinline__ PbQTabs pb_h_fill_tabs(uint8_t* tab, int rep, int tid, int nthreads, int lane) {
    if constexpr (FMT == PB_T_IQ2_XS) {
        uint32_t* g = reinterpret_cast<uint32_t*>(tab);
        // an entry once for all its copies; the magnitudes' upper nibbles are their numbers (0x08, 0x19, 0x2B).  Formed byte by byte for every copy the
        // table took longer than a small product (4 tokens of 2048 x 512: 10.3 us, 8.3 so; of 2048 x 4096 14.4 and 12.3)
        for (int i = tid; i < 512; i += nthreads) {
            const uint64_t e = PB_IQ2XS_GRID[i];
            uint32_t lo = ((uint32_t)e >> 4) & 0x0F0F0F0Fu, hi = (uint32_t)(e >> 36) & 0x0F0F0F0Fu;
            lo = (lo | lo >> 4) & 0x00FF00FFu; hi = (hi | hi >> 4) & 0x00FF00FFu;
            const uint32_t v = pb_prmt(lo, hi, 0x6420u);
            for (int j = 0; j < rep; j++) g[i * rep + j] = v;
        }
        PbQTabs T = {0u, 0u, 0u};
        T.stride = 4u * (uint32_t)rep; T.grid = pb_smem_u32(tab) + (uint32_t)(lane & (rep - 1)) * 4u;
        return T;
    } else return pb_fill_qtabs<FMT>(tab, rep, tid, nthreads, lane);
}
// Eight weights of an IQ2_XS index (9 bits of grid, 7 of signs, the eighth their parity) as f16 pairs (0 2)(4 6)(1 3)(5 7), times s; k = -1024 s
__device__ __forceinline__ void pb_h_word_iq2xs(const PbQTabs& T, uint32_t q, __half2 s, __half2 k, uint32_t (&o)[4]) {
    const uint32_t sel = pb_lds32(T.grid + (q & 511u) * T.stride);
    const uint32_t s7 = q >> 9, s8 = s7 | ((uint32_t)(__popc(s7) & 1) << 7), z = s8 | (s8 << 14);   // sign bits i and i + 2 sixteen places apart (14 + 2)
    const uint32_t g0 = pb_prmt(0x002B1908u, 0u, sel), g1 = pb_prmt(0x002B1908u, 0u, sel >> 16);      // magnitudes as bytes
    o[0] = pb_as_u32(__hfma2(pb_as_h2(pb_prmt(g0, 0x64646464u, 0x4240u)), s, k)) ^ ((z << 15) & 0x80008000u);
    o[1] = pb_as_u32(__hfma2(pb_as_h2(pb_prmt(g1, 0x64646464u, 0x4240u)), s, k)) ^ ((z << 11) & 0x80008000u);
    o[2] = pb_as_u32(__hfma2(pb_as_h2(pb_prmt(g0, 0x64646464u, 0x4341u)), s, k)) ^ ((z << 14) & 0x80008000u);
    o[3] = pb_as_u32(__hfma2(pb_as_h2(pb_prmt(g1, 0x64646464u, 0x4341u)), s, k)) ^ ((z << 10) & 0x80008000u);
}
// bytes (0, 2) or (1, 3) of a word of four signed bytes, already flipped to unsigned, as the mantissas of 1024 + 128 + v
__device__ __forceinline__ uint32_t pb_h_bytes(uint32_t w, bool odd) { return pb_prmt(w, 0x64646464u, odd ? 0x4341u : 0x4240u); }

template <int FMT, int NT>
__device__ __forceinline__ void pb_h_block_int(uint32_t pa, uint32_t pb, const PbQTabs& T, int blk, int lane, const PbHLane& L, float (&tot)[NT][2]) {
    using D = PbQDec<FMT>;
    const int q = lane & 3;
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) { acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f; }
    PbQuarter wa, wb;
    if constexpr (FMT != PB_T_IQ2_XS) { D::quarter(pa, q, T, wa); D::quarter(pb, q, T, wb); }
    float fa, fb;                                              // f32 factor of the block's sum
    if constexpr (FMT == PB_T_IQ2_XS) {
        uint32_t ma[4], mb[4], qa[4], qb[4];                   // integer multipliers and index words
        pb_h_mults<FMT>(pa, q, fa, ma); pb_h_mults<FMT>(pb, q, fb, mb);
        pb_ld_u32x<4>(pa + 2 + 16 * q, qa); pb_ld_u32x<4>(pb + 2 + 16 * q, qb);
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
            const __half2 sa = pb_h2_int(ma[u >> 1]), sb = pb_h2_int(mb[u >> 1]), k = pb_as_h2(0xE400E400u), ka = __hmul2(sa, k), kb = __hmul2(sb, k);   // -1024
            uint32_t a[2][4], b[2][4];
#pragma unroll
            for (int v = 0; v < 2; v++) {
                pb_h_word_iq2xs(T, (qa[u >> 1] >> (16 * v)) & 0xFFFFu, sa, ka, a[v]);
                pb_h_word_iq2xs(T, (qb[u >> 1] >> (16 * v)) & 0xFFFFu, sb, kb, b[v]);
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint32_t xa = L.b + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 1024 + u * 128);
                const uint4 x = pb_ldsa128(xa), y = pb_ldsa128(xa + 128);
                float c[4];
                pb_hmma0(c, a[0][0], b[0][0], a[0][1], b[0][1], x.x, x.y);
                pb_hmma(c, a[0][2], b[0][2], a[0][3], b[0][3], x.z, x.w);
                pb_hmma(c, a[1][0], b[1][0], a[1][1], b[1][1], y.x, y.y);
                pb_hmma(c, a[1][2], b[1][2], a[1][3], b[1][3], y.z, y.w);
                pb_h_flush(acc[nt], c);
            }
        }
    } else if constexpr (pb_h_mode<FMT>() == PB_H_FOLD) {
        uint32_t ma[4], mb[4];
        pb_h_mults<FMT>(pa, q, fa, ma); pb_h_mults<FMT>(pb, q, fb, mb);
        float c[NT][4];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const __half2 sa = pb_h2_int(ma[u >> 1]), sb = pb_h2_int(mb[u >> 1]), k = pb_as_h2(0xE480E480u);   // -1152
            const __half2 ka = __hmul2(sa, k), kb = __hmul2(sb, k);                                             // exact: at most 9 significant bits
            uint32_t a[4], b[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                a[e] = pb_as_u32(__hfma2(pb_as_h2(pb_h_bytes((uint32_t)wa.w[2 * u + (e & 1)] ^ 0x80808080u, e >= 2)), sa, ka));
                b[e] = pb_as_u32(__hfma2(pb_as_h2(pb_h_bytes((uint32_t)wb.w[2 * u + (e & 1)] ^ 0x80808080u, e >= 2)), sb, kb));
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint4 x = pb_ldsa128(L.b + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 1024 + u * 128));
                if (u & 1) pb_hmma(c[nt], a[0], b[0], a[1], b[1], x.x, x.y); else pb_hmma0(c[nt], a[0], b[0], a[1], b[1], x.x, x.y);
                pb_hmma(c[nt], a[2], b[2], a[3], b[3], x.z, x.w);
                if (u & 1) pb_h_flush(acc[nt], c[nt]);
            }
        }
    } else {
        // power of two that puts the largest scale of the row's block into [1, 2); scales as f16 high + low parts
        auto norm = [&](PbQuarter& w, float& f) {
            float m = fmaxf(fmaxf(fabsf(w.sc[0]), fabsf(w.sc[1])), fmaxf(fabsf(w.sc[2]), fabsf(w.sc[3])));
            if (D::HAS_MIN) m = fmaxf(m, fmaxf(fabsf(w.mn[0]), fabsf(w.mn[1])) * (1.0f / 64.f));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1)); m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            float p = 1.0f; f = 1.0f;
            if (m > 1e-30f && m < 1e30f) { const uint32_t e = (__float_as_uint(m) >> 23) & 0xFF; p = __uint_as_float((254u - e) << 23); f = __uint_as_float(e << 23); }
#pragma unroll
            for (int h = 0; h < 4; h++) w.sc[h] *= p;
            if (D::HAS_MIN) { w.mn[0] *= p; w.mn[1] *= p; }
        };
        norm(wa, fa); norm(wb, fb);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const float sfa = wa.sc[u >> 1], sfb = wb.sc[u >> 1];
            const __half ha = __float2half_rn(sfa), hb = __float2half_rn(sfb);
            const __half2 sah = __half2half2(ha), sbh = __half2half2(hb), sal = __half2half2(__float2half_rn(sfa - __half2float(ha))), sbl = __half2half2(__float2half_rn(sfb - __half2float(hb)));
            const __half2 k = pb_as_h2(0x64806480u);            // 1152
            uint32_t a[4], b[4], al[4], bl[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                // scaled weight = high + low: the remainder of the high product is exact in one fused multiply-add
                const __half2 va = __hsub2(pb_as_h2(pb_h_bytes((uint32_t)wa.w[2 * u + (e & 1)] ^ 0x80808080u, e >= 2)), k);
                const __half2 vb = __hsub2(pb_as_h2(pb_h_bytes((uint32_t)wb.w[2 * u + (e & 1)] ^ 0x80808080u, e >= 2)), k);
                const __half2 pa2 = __hmul2(va, sah), pb2 = __hmul2(vb, sbh);
                a[e] = pb_as_u32(pa2); b[e] = pb_as_u32(pb2);
                al[e] = pb_as_u32(__hfma2(va, sal, __hfma2(va, sah, __hneg2(pa2)))); bl[e] = pb_as_u32(__hfma2(vb, sbl, __hfma2(vb, sbh, __hneg2(pb2))));
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                const uint4 x = pb_ldsa128(L.b + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 1024 + u * 128));
                float c[4];                                      // the low parts first: their sums are small, and so is what truncation takes from them
                pb_hmma0(c, al[0], bl[0], al[1], bl[1], x.x, x.y);
                pb_hmma(c, al[2], bl[2], al[3], bl[3], x.z, x.w);
                pb_hmma(c, a[0], b[0], a[1], b[1], x.x, x.y);
                pb_hmma(c, a[2], b[2], a[3], b[3], x.z, x.w);
                pb_h_flush(acc[nt], c);
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        float oa = 0.f, ob = 0.f;
        if (D::HAS_MIN && pb_h_offs<FMT>()) {
            uint2 s = pb_ldsa64(L.sums + (uint32_t)nt * L.tok4 + (uint32_t)(blk * 32));
            if ((lane >> 2) & 1) s = make_uint2(0u, 0u);
            const __half2 ma = __floats2half2_rn(wa.mn[0], wa.mn[1]), mb = __floats2half2_rn(wb.mn[0], wb.mn[1]);
            const float2 ra = __half22float2(ma), rb = __half22float2(mb);
            const uint32_t la = pb_as_u32(__floats2half2_rn(wa.mn[0] - ra.x, wa.mn[1] - ra.y)), lb = pb_as_u32(__floats2half2_rn(wb.mn[0] - rb.x, wb.mn[1] - rb.y));
            float mc[4] = {0.f, 0.f, 0.f, 0.f};
            pb_hmma(mc, pb_as_u32(ma), pb_as_u32(mb), pb_as_u32(ma), pb_as_u32(mb), s.x, s.y);
            pb_hmma(mc, la, lb, la, lb, s.x, s.y);
            oa = -fa * mc[0]; ob = -fb * mc[2];
        }
        pb_h_add<FMT, NT>(acc, nt, blk, fa, fb, oa, ob, L, tot);
    }
}

// the block in stage `stage` of tile t, whichever the format: block wblk of the weight rows, block blk of the prepared activations
template <int FMT, int NT>
__device__ __forceinline__ void pb_h_block(uint32_t stage, const PbHTile& t, const PbHGeom& h, const PbQTabs& T, int wblk, int blk, int lane, const PbHLane& L, float (&tot)[NT][2]) {
    if constexpr (pb_h_mode<FMT>() == PB_H_DIRECT) pb_h_block_nib<FMT, NT>(stage, h, blk, lane, L, tot);
    else {
        const int g = lane >> 2;
        const uint32_t oa = (uint32_t)(reinterpret_cast<uintptr_t>(t.a) + (uint32_t)min(g, t.la) * (uint32_t)h.row_bytes + (uint32_t)wblk * (uint32_t)h.step_bytes) & 15u;
        const uint32_t ob = (uint32_t)(reinterpret_cast<uintptr_t>(t.b) + (uint32_t)min(g, t.lb) * (uint32_t)h.row_bytes + (uint32_t)wblk * (uint32_t)h.step_bytes) & 15u;
        pb_h_block_int<FMT, NT>(stage + (uint32_t)(g * h.pitch) + oa, stage + (uint32_t)((g + 8) * h.pitch) + ob, T, blk, lane, L, tot);
    }
}
