// Router arithmetic shared by pb_router_kernel (pb_moe.cu) and the fused step kernel (pb_step.cu): both produce the
// same bits, so the expert selection of a token does not depend on which of them ran.
// Restates the router product of ffn (src/model/qwen4exp_gguf.rs:1675-1684) over rms(x) (:209).
#pragma once
#include "pb_common.cuh"

// 1 / sqrt(mean(x^2) + eps) of one row of `cols` values, computed by one warp (every lane gets the result).
// Every multiply-add is spelled out (fmaf): left to the compiler, the fusing of a*a + b*b + .. into multiply-adds may come
// out differently in the two kernels that inline this function, and their results would differ in the last bit.
__device__ __forceinline__ float pb_row_rms_scale(const float* x, int cols, float eps, int lane) {
    float ss = 0.f;
    for (int c = lane * 4; c < cols; c += 128) { const float4 v = *reinterpret_cast<const float4*>(x + c); ss += fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, __fmul_rn(v.w, v.w)))); }
    ss = pb_warp_sum(ss);
    return 1.0f / sqrtf(ss / (float)cols + eps);
}

// One router row of 2048 columns against one token, by one warp: the row times the norm weight is formed in registers,
// the token's scale is applied to the sum (w . (x s n) = s ((w n) . x) up to rounding).  norm_w may be null.
struct PbRouterRow2048 {
    float4 wr[16];
    __device__ __forceinline__ void load(const float* wrow, const float* norm_w, int lane) {
#pragma unroll
        for (int k = 0; k < 16; k++) {
            wr[k] = *reinterpret_cast<const float4*>(wrow + lane * 4 + 128 * k);
            if (norm_w) { const float4 n = *reinterpret_cast<const float4*>(norm_w + lane * 4 + 128 * k); wr[k].x *= n.x; wr[k].y *= n.y; wr[k].z *= n.z; wr[k].w *= n.w; }
        }
    }
    __device__ __forceinline__ float dot(const float* x, float scale, int lane) const {
        const float* xb = x + lane * 4;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float4 v = *reinterpret_cast<const float4*>(xb + 128 * k);
            a0 = fmaf(wr[k].x, v.x, a0); a1 = fmaf(wr[k].y, v.y, a1); a2 = fmaf(wr[k].z, v.z, a2); a3 = fmaf(wr[k].w, v.w, a3);
        }
        return pb_warp_sum((a0 + a1) + (a2 + a3)) * scale;
    }
};

// Four router rows x a quarter of their 2048 columns, held by one warp for several tokens: one fetch of the token's 512 values serves four
// rows (a row per warp is bound by those fetches: 120 us for 256 tokens x 513 rows, this form 73 us).  The quarters of a row meet in shared memory.
struct PbRouterQuad {
    float4 w[4][4];
    __device__ __forceinline__ void load(const float* const (&rows)[4], const float* norm_w, int kq, int lane) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int c = 512 * kq + lane * 4 + 128 * k;
            float4 n = make_float4(1.f, 1.f, 1.f, 1.f);
            if (norm_w) n = *reinterpret_cast<const float4*>(norm_w + c);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (rows[r]) v = *reinterpret_cast<const float4*>(rows[r] + c);
                v.x *= n.x; v.y *= n.y; v.z *= n.z; v.w *= n.w;
                w[r][k] = v;
            }
        }
    }
    // lane l ends up with the sum of row (l >> 3) & 3 over the warp's columns
    __device__ __forceinline__ float dot(const float* x, int kq, int lane) const {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = *reinterpret_cast<const float4*>(x + 512 * kq + lane * 4 + 128 * k);
        float a[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int k = 0; k < 4; k++) { s0 = fmaf(w[r][k].x, v[k].x, s0); s1 = fmaf(w[r][k].y, v[k].y, s1); s0 = fmaf(w[r][k].z, v[k].z, s0); s1 = fmaf(w[r][k].w, v[k].w, s1); }
            a[r] = s0 + s1;
        }
        // rows (0 1 | 2 3) by lane bit 4, then (0 | 1), (2 | 3) by bit 3
        const bool h = lane & 16, l = lane & 8;
        float b0 = (h ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, h ? a[0] : a[2], 16), b1 = (h ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, h ? a[1] : a[3], 16);
        float c = (l ? b1 : b0) + __shfl_xor_sync(0xffffffffu, l ? b0 : b1, 8);
        c += __shfl_xor_sync(0xffffffffu, c, 4); c += __shfl_xor_sync(0xffffffffu, c, 2); c += __shfl_xor_sync(0xffffffffu, c, 1);
        return c;
    }
};

// The same product for one token without keeping the row: (w n) is formed per element on the way (same roundings).
__device__ __forceinline__ float pb_router_row2048_dot1(const float* wrow, const float* norm_w, const float* x, float scale, int lane) {
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll 4
    for (int k = 0; k < 16; k++) {
        float4 w = *reinterpret_cast<const float4*>(wrow + lane * 4 + 128 * k);
        if (norm_w) { const float4 n = *reinterpret_cast<const float4*>(norm_w + lane * 4 + 128 * k); w.x *= n.x; w.y *= n.y; w.z *= n.z; w.w *= n.w; }
        const float4 v = *reinterpret_cast<const float4*>(x + lane * 4 + 128 * k);
        a0 = fmaf(w.x, v.x, a0); a1 = fmaf(w.y, v.y, a1); a2 = fmaf(w.z, v.z, a2); a3 = fmaf(w.w, v.w, a3);
    }
    return pb_warp_sum((a0 + a1) + (a2 + a3)) * scale;
}

// any width (a multiple of 128): one accumulator chain over the normalized activations
__device__ __forceinline__ float pb_router_row_dot(const float* wrow, const float* norm_w, const float* x, float s, int cols, int lane) {
    float acc = 0.f;
#pragma unroll 4
    for (int c = lane * 4; c < cols; c += 128) {
        const float4 w = *reinterpret_cast<const float4*>(wrow + c);
        float4 v = *reinterpret_cast<const float4*>(x + c);
        if (norm_w) {
            const float4 n = *reinterpret_cast<const float4*>(norm_w + c);
            v.x = v.x * s * n.x; v.y = v.y * s * n.y; v.z = v.z * s * n.z; v.w = v.w * s * n.w;
        }
        acc = fmaf(w.x, v.x, acc); acc = fmaf(w.y, v.y, acc); acc = fmaf(w.z, v.z, acc); acc = fmaf(w.w, v.w, acc);
    }
    return pb_warp_sum(acc);
}
