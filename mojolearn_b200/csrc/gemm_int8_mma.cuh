// Integer products on the fifth-generation tensor cores: what the int8i32.v1 and int15i64.v1 kernels share.
//
// C[i][j] = ftz(f32(sum_p qa[i][p] * qb[j][p]) * 2^(ea[i] + eb[j])) is the one profile of the path where a tensor-core MMA is
// contract-legal: the sum of products of int8 codes is an exact int32 (k <= 131072 keeps it inside 31 bits), so the order in
// which the hardware adds cannot move a bit (gemm/IDENTICAL_LOWBIT_CONTRACT.md:66-109 of the reference; its sm_80 form is
// gemm/checks/gemm_int8_mma.mojo:263-281, :545-620). The float32 products cannot use it: they round once per step.
//
// Both operands are K-major (rows of codes), which is the layout tcgen05.mma.kind::i8 takes without a transpose. The kernels
// are gemm_int8_pair_kernel and gemm_int8_tma_kernel, and in gemm_int15.cuh the fifteen-bit ones.
#pragma once
#include "decode.cuh" // mbarrier helpers, g_decode_status
#include "lowbit.cuh"

namespace b200i {

constexpr int I8_TILE_M = 128; // rows of A per CTA = lanes of the accumulator
constexpr int I8_KB = 128;     // bytes of k per stage
constexpr int I8_THREADS = 128;

// K-major, no swizzle: start address, leading (k) and stride (row group) byte offsets in 16-byte units, descriptor version 1.
__device__ __forceinline__ unsigned long long i8_smem_desc(unsigned smem_addr) {
    return (unsigned long long)((smem_addr & 0x3FFFFu) >> 4) | ((unsigned long long)(128u >> 4) << 16) |
           ((unsigned long long)(1024u >> 4) << 32) | (1ull << 46);
}
// D = S32, A = B = signed 8-bit, both K-major, N = tn, M = 128.
__host__ __device__ constexpr unsigned i8_idesc(int tn) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(tn >> 3) << 17) | ((unsigned)(I8_TILE_M >> 4) << 24);
}

__device__ __forceinline__ void i8_mma(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void i8_commit(unsigned long long *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void i8_cp16(void *dst, const void *src, unsigned src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes) : "memory");
}

// Copies 128 bytes of k (from byte k0) of ROWS rows starting at row0 into one operand buffer, in the canonical no-swizzle
// K-major form: 8 rows x 16 bytes = one 128-byte core matrix; core matrices of one row group lie side by side along k
// (leading byte offset 128), row groups follow each other (stride byte offset 1024). Zero filled past the edges. A warp instruction
// covers 8 rows x 64 bytes: whole 32-byte sectors of global memory, and four conflict-free 128-byte core matrices.
template <int ROWS>
__device__ __forceinline__ void i8_load_operand(unsigned char *buf, const signed char *src, int row0, int rows_total, int k, int k0, int tid) {
#pragma unroll
    for (int it = 0; it < ROWS * (I8_KB / 16) / I8_THREADS; it++) {
        const int idx = it * I8_THREADS + tid;
        const int lane = idx & 31, w = idx >> 5;
        const int r = (w >> 1) * 8 + (lane & 7);           // ROWS / 8 row groups x 8 rows
        const int chunk = (w & 1) * 4 + (lane >> 3);       // 16-byte chunk of the 128 bytes: 0..7
        const int row = row0 + r, kb = k0 + chunk * 16;
        const bool in = row < rows_total && kb < k;        // k is a multiple of 16: a chunk is inside or outside as a whole
        const signed char *from = in ? src + (size_t)row * k + kb : src;
        i8_cp16(buf + ((r >> 3) * (I8_KB / 16) + chunk) * 128 + (r & 7) * 16, from, in ? 16u : 0u);
    }
}

// k a multiple of 16 and 16-byte aligned operands: every 16-byte copy is then aligned and inside one row.
inline bool gemm_int8_mma_fits(const void *qa, const void *qb, long long k) {
    return k % 16 == 0 && ((reinterpret_cast<uintptr_t>(qa) | reinterpret_cast<uintptr_t>(qb)) & 15) == 0;
}

} // namespace b200i
