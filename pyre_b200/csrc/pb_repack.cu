// IQ3_S -> PB_T_IQ3S_N4: a lossless re-coding done once when a matrix arrives on the device.
//
// An IQ3_S weight is  d * (1 + 2 s) * sign * g  (dequant, gguf_q.rs:141-151) where g is one byte of a
// codebook entry.  All 2048 codebook bytes are odd numbers 1..15, so sign * g is one of the sixteen values
// -15, -13, .. 15 = 2 c - 15 with a 4-bit code c.  The re-coded block keeps d and the 4-bit sub-scales
// unchanged and stores c for every weight: 136 bytes per 256 weights instead of 110.  The streaming kernels
// then spend two logic operations per eight weights on decoding instead of a codebook walk with sign
// arithmetic, which is what kept the native format at a third of the HBM roofline; the values they
// multiply are bit-identical.
//
// Order of the bytes (PB_T_IQ3S_N4): groups of eight rows, each as long as eight rows of 136 bytes per block, so that any run of
// whole groups is one contiguous range.  Inside a group, block after block (1088 bytes): two pieces of 512 bytes -- piece i holds, for row r
// and quarter q (64 weights) of the block, the 16 bytes of weights 32 i .. 32 i + 31 of the quarter at slot 4 r + q -- then
// eight bytes {d f16, 0, four bytes of 4-bit sub-scales} per row.  A warp that holds 8 rows x 4 quarters (the operand layout of the tensor
// cores) reads a piece as 512 consecutive bytes straight from global memory; a warp that holds the quarters of one row reads it from
// shared memory without bank conflicts (neighbouring blocks are 64 bytes apart modulo 128).  The last group of a matrix is padded with zero blocks.
#include "pb_internal.h"
#include "pb_formats.cuh"

// One thread per output word (8 weights), in the order of the output: a warp writes 128 consecutive bytes.  nrows counts the padding rows,
// rows the real ones.
__global__ void __launch_bounds__(256) pb_repack_iq3s_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t nrows, int64_t rows, int bpr, int* bad) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t gb = i >> 8;                                  // block of a group of eight rows
    const int w8 = (int)(i & 255), piece = w8 >> 7, slot = (w8 >> 2) & 31;
    const int64_t grp = gb / bpr;
    const int b = (int)(gb - grp * bpr), r = slot >> 2, q = slot & 3, k = 4 * piece + (w8 & 3);   // row in the group, quarter, word k of the quarter
    const int64_t row = grp * 8 + r;
    if (row >= nrows) return;
    uint8_t* out = dst + gb * 1088;
    uint32_t* word = reinterpret_cast<uint32_t*>(out) + w8;
    const int m = 8 * q + k;                                    // word of the row's block
    if (row >= rows) { *word = 0u; if (m < 2) reinterpret_cast<uint32_t*>(out + 1024 + 8 * r)[m] = 0u; return; }
    const int64_t blk = row * bpr + b;
    const uint8_t* p = src + blk * 110;
    if (m == 0) {
        uint8_t* h = out + 1024 + 8 * r;
        h[0] = p[0]; h[1] = p[1]; h[2] = 0; h[3] = 0;
        h[4] = p[106]; h[5] = p[107]; h[6] = p[108]; h[7] = p[109];
    }
    // word m = weights 8m .. 8m+7 = codebook entries 2m and 2m+1, sign byte m
    const uint32_t qh = p[66 + (m >> 2)] >> (2 * (m & 3));
    const uint32_t g0 = PB_IQ3S_GRID[p[2 + 2 * m] | ((qh & 1) << 8)];
    const uint32_t g1 = PB_IQ3S_GRID[p[3 + 2 * m] | ((qh & 2) << 7)];
    const uint32_t sg = p[74 + m];
    uint32_t w = 0;
    bool odd = true;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int a = (int)((g0 >> (8 * j)) & 0xFF), c = (int)((g1 >> (8 * j)) & 0xFF);
        odd = odd && (a & 1) && a <= 15 && (c & 1) && c <= 15;
        const int va = (sg >> j) & 1 ? -a : a, vb = (sg >> (4 + j)) & 1 ? -c : c;
        w |= (uint32_t)(((va + 15) >> 1) & 0xF) << (8 * j);
        w |= (uint32_t)(((vb + 15) >> 1) & 0xF) << (8 * j + 4);
    }
    if (!odd) atomicExch(bad, PB_DEV_BAD_INDEX);   // cannot happen with the IQ3_S codebook; checked rather than assumed
    *word = w;
}

int pb_launch_repack_iq3s(pb_ctx* ctx, const uint8_t* src, uint8_t* dst, int64_t rows, int bpr) {
    if (rows <= 0) return PB_OK;
    const int64_t nrows = (rows + 7) & ~(int64_t)7, threads = nrows * bpr * 32;
    pb_repack_iq3s_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, ctx->stream>>>(src, dst, nrows, rows, bpr, ctx->dev_status);
    ctx->kernels_launched++;
    PB_CUDA(ctx, cudaGetLastError());
    return PB_OK;
}
