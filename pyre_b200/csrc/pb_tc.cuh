// tcgen05 (fifth-generation tensor core) wrappers shared by the dequant-GEMM (pb_gemmtc.cu) and the expert kernels of prompts (pb_moetc.cu):
// tensor-memory allocation, loads and stores, MMA issue and commit, operand and instruction descriptors.
#pragma once
#include "pb_stream.cuh"

enum : int { PB_DEV_TC_TIMEOUT = 6 };

// ---------------------------------------------------------------- tcgen05 wrappers (cta_group::1)
__device__ __forceinline__ void tc_alloc(uint32_t* smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pb_smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// One lane of a converged warp.  An MMA takes its operands from uniform registers: in code that the compiler knows to be warp-uniform (the warp's number
// from tc_uniform_warp, one lane elected) one issues every 25 to 40 cycles; behind `lane == 0` with values it takes for a lane's own, every 120 to 190
// (measured on 256 of them, 128 rows x 16 to 128 columns).
__device__ __forceinline__ bool tc_elect() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
// One arrival for the whole warp, behind what all its lanes did.  (An arrival of every lane is 32 operations on one word of shared memory, one after the other:
// with 128 or 256 arrivals a step they were what the pipelines of these kernels waited for.)
__device__ __forceinline__ void tc_warp_arrive(uint64_t* bar, int lane) { __syncwarp(); if (lane == 0) pb_mbar_arrive(bar); }
// A wait of the whole warp: it ends for all lanes alike.  (A lane that left alone, because only its wait ran out, would strand the others at the next
// instruction that takes a converged warp -- tcgen05.ld / st, the arrival above -- and the kernel would never leave.)
__device__ __forceinline__ bool tc_warp_wait(uint64_t* bar, uint32_t phase, int* status) { return __all_sync(0xffffffffu, pb_mbar_wait(bar, phase, status, PB_DEV_TC_TIMEOUT)) != 0; }
__device__ __forceinline__ int tc_uniform_warp() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }
// D (tensor memory) (+)= A (tensor memory: lane = row, two f16 per cell along K) x B (shared memory, by descriptor)
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the mbarrier receives one arrival once every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(pb_smem_u32(bar)) : "memory");
}
// 32 lanes x 32 consecutive columns of 32-bit cells: thread l of the warp gets lane (base lane + l), columns c .. c+31
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory operand descriptor: K-major, 128-byte swizzle.  A row of the tile (one weight row or one token) is 128
// contiguous bytes = the 64 columns of a step; its 16-byte chunk c sits at chunk position c ^ (row & 7); groups of 8
// rows are 1024 bytes apart (the stride offset); the tile starts on a 1024-byte boundary.  A step of 16 columns along K
// is 32 bytes further into the row: the start address moves, the swizzle is applied by the hardware on the address bits.
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor of kind::f16: f32 accumulator, f16 A and B, both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t tc_idesc(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }

__device__ __forceinline__ void tc_cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// the mbarrier (initialised with one count per issuing thread) gets this thread's arrival once its copies so far have landed
__device__ __forceinline__ void tc_cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(pb_smem_u32(bar)) : "memory");
}
// four columns of the warp's lanes, without the wait: the values are there after tc_wait_ld
__device__ __forceinline__ void tc_ld4(uint32_t taddr, float* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 cells of this thread's lane, consecutive columns from taddr on (taddr carries the warp's first lane in bits 16+)
__device__ __forceinline__ void tc_st32_nowait(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
          "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) { tc_st32_nowait(taddr, r); tc_wait_st(); }
