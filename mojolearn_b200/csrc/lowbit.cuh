// Low-bit conversion kernels (contract clauses L-1 .. L-6 of the reference's
// gemm/IDENTICAL_LOWBIT_CONTRACT.md) and the int8i32.v1 product.
//
// Reference kernels these replace: bf16_widen_kernel / bf16_narrow_kernel
// (gemm/checks/gemm_lowbit.mojo:166-187), quantize_rows_int8_kernel /
// dequantize_rows_int8_kernel (:435-477), identical_gemm_int8_flat_kernel
// (:480-511). All of them are HBM-bound byte work: 128-bit coalesced loads,
// one pass, grid sized from the element count.
#pragma once
#include "seams.cuh"

namespace b200i {

__global__ void to_bf16_kernel(unsigned short *__restrict__ dst, const float *__restrict__ src, long long count) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool vec = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) && ((reinterpret_cast<uintptr_t>(dst) & 7) == 0);
    const long long quads = vec ? count / 4 : 0;
    for (long long q = i0; q < quads; q += stride) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(src) + q);
        uint2 w;
        w.x = (unsigned)f32_to_bf16_bits_rne(v.x) | ((unsigned)f32_to_bf16_bits_rne(v.y) << 16);
        w.y = (unsigned)f32_to_bf16_bits_rne(v.z) | ((unsigned)f32_to_bf16_bits_rne(v.w) << 16);
        reinterpret_cast<uint2 *>(dst)[q] = w;
    }
    for (long long i = quads * 4 + i0; i < count; i += stride) dst[i] = f32_to_bf16_bits_rne(src[i]);
}

__global__ void from_bf16_kernel(float *__restrict__ dst, const unsigned short *__restrict__ src, long long count) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool vec = ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) && ((reinterpret_cast<uintptr_t>(src) & 7) == 0);
    const long long quads = vec ? count / 4 : 0;
    for (long long q = i0; q < quads; q += stride) {
        const uint2 w = __ldg(reinterpret_cast<const uint2 *>(src) + q);
        float4 v;
        v.x = __uint_as_float(w.x << 16);
        v.y = __uint_as_float(w.x & 0xFFFF0000u);
        v.z = __uint_as_float(w.y << 16);
        v.w = __uint_as_float(w.y & 0xFFFF0000u);
        reinterpret_cast<float4 *>(dst)[q] = v;
    }
    for (long long i = quads * 4 + i0; i < count; i += stride) dst[i] = bf16_bits_to_f32(src[i]);
}

// One warp per row: the row's absmax after the flush (a maximum is exact and
// order-free, so a shuffle butterfly is as good as any walk), the power-of-two
// exponent, then every value scaled, rounded half-even and clamped.
__global__ void quantize_int8_kernel(signed char *__restrict__ q, int *__restrict__ e, const float *__restrict__ x,
                                     long long rows, long long cols) {
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long r = warp; r < rows; r += nwarps) {
        const float *row = x + r * cols;
        float best = 0.f;
        for (long long c = lane; c < cols; c += 32) {
            float v = fabsf(ftz_bits(row[c]));
            if (v > best) best = v; // a NaN never compares greater and is skipped, as in the scalar walk
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) best = fmaxf(best, __shfl_xor_sync(0xFFFFFFFFu, best, off));
        const int ex = int8_row_exponent(best);
        if (lane == 0) e[r] = ex;
        for (long long c = lane; c < cols; c += 32) q[r * cols + c] = quantize_int8_value(row[c], ex);
    }
}

// One value's code in three instructions: the product by the row's power of two (input and result flushed: a result that
// the flush could touch rounds to code 0 either way), a conversion that rounds half to even, saturates and takes a NaN to
// 0, and the lower clamp: quantize_int8_value's answer for every input.
__device__ __forceinline__ unsigned quantize_int8_byte(float x, float scale) {
    float s;
    int q;
    asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(s) : "f"(x), "f"(scale));
    asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(s));
    return (unsigned)max(q, -127) & 0xFFu;
}
__device__ __forceinline__ unsigned quantize_int8_quad(float4 v, float scale) {
    return quantize_int8_byte(v.x, scale) | quantize_int8_byte(v.y, scale) << 8 | quantize_int8_byte(v.z, scale) << 16 | quantize_int8_byte(v.w, scale) << 24;
}
// fmaxf passes over a NaN, as the scalar walk does; a subnormal maximum is flushed by int8_row_exponent
__device__ __forceinline__ float absmax4(float4 v, float best) {
    return fmaxf(fmaxf(fmaxf(best, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
}

// The same for rows that are whole float4s: WARPS warps share a row and keep it in registers between the maximum and the
// rounding, so it is read once, 16 bytes a lane, and its codes leave 4 bytes a lane. Bound: HBM, 5 bytes per element
// ([4096, 4096]: 84 MB). One row per 1024 * WARPS columns at most; a block of 256 threads holds 8 / WARPS rows.
constexpr int QUANT_VEC = 8; // float4s a lane holds
template <int WARPS>
__global__ void __launch_bounds__(256) quantize_int8_rows_kernel(signed char *__restrict__ q, int *__restrict__ e, const float *__restrict__ x,
                                                                 long long rows, int cols) {
    __shared__ float part[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long r = (long long)blockIdx.x * (8 / WARPS) + warp / WARPS;
    const int first = (warp % WARPS) * 32 + lane, quads = cols >> 2;
    const bool live = r < rows;
    const float4 *row = reinterpret_cast<const float4 *>(x + (live ? r : 0) * cols);
    float4 v[QUANT_VEC];
    float best = 0.f;
#pragma unroll
    for (int i = 0; i < QUANT_VEC; i++) {
        const int c = first + i * 32 * WARPS;
        v[i] = (live && c < quads) ? __ldg(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < QUANT_VEC; i++) best = absmax4(v[i], best);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = fmaxf(best, __shfl_xor_sync(0xFFFFFFFFu, best, off));
    if (WARPS > 1) {
        if (lane == 0) part[warp] = best;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < WARPS; w++) best = fmaxf(best, part[warp / WARPS * WARPS + w]);
    }
    if (!live) return;
    const int ex = int8_row_exponent(best);
    if (first == 0) e[r] = ex;
    const float scale = pow2_f32(-ex);
    unsigned *out = reinterpret_cast<unsigned *>(q + r * cols);
#pragma unroll
    for (int i = 0; i < QUANT_VEC; i++) {
        const int c = first + i * 32 * WARPS;
        if (c < quads) out[c] = quantize_int8_quad(v[i], scale);
    }
}

// Rows too wide for that: a block of 512 threads per row, which is read twice (the second time from L2).
__global__ void __launch_bounds__(512) quantize_int8_wide_kernel(signed char *__restrict__ q, int *__restrict__ e, const float *__restrict__ x, long long quads) {
    __shared__ float part[16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float4 *row = reinterpret_cast<const float4 *>(x) + (long long)blockIdx.x * quads;
    unsigned *out = reinterpret_cast<unsigned *>(q) + (long long)blockIdx.x * quads;
    float best = 0.f;
#pragma unroll 4
    for (long long c = threadIdx.x; c < quads; c += 512) best = absmax4(__ldg(row + c), best);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = fmaxf(best, __shfl_xor_sync(0xFFFFFFFFu, best, off));
    if (lane == 0) part[warp] = best;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 16; w++) best = fmaxf(best, part[w]);
    const int ex = int8_row_exponent(best);
    if (threadIdx.x == 0) e[blockIdx.x] = ex;
    const float scale = pow2_f32(-ex);
#pragma unroll 4
    for (long long c = threadIdx.x; c < quads; c += 512) out[c] = quantize_int8_quad(__ldg(row + c), scale);
}

// The row kernels where rows are whole aligned float4s; the walk over scalars elsewhere.
inline void launch_quantize_int8(signed char *q, int *e, const float *x, long long rows, long long cols, int sms, cudaStream_t st) {
    const bool quads = cols % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0;
    const long long span = 32 * 4 * QUANT_VEC; // columns one warp holds
    if (quads && rows <= 0x7FFFFFFFll) {
        if (cols <= span) quantize_int8_rows_kernel<1><<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(q, e, x, rows, (int)cols);
        else if (cols <= 2 * span) quantize_int8_rows_kernel<2><<<(unsigned)((rows + 3) / 4), 256, 0, st>>>(q, e, x, rows, (int)cols);
        else if (cols <= 4 * span) quantize_int8_rows_kernel<4><<<(unsigned)((rows + 1) / 2), 256, 0, st>>>(q, e, x, rows, (int)cols);
        else if (cols <= 8 * span) quantize_int8_rows_kernel<8><<<(unsigned)rows, 256, 0, st>>>(q, e, x, rows, (int)cols);
        else quantize_int8_wide_kernel<<<(unsigned)rows, 512, 0, st>>>(q, e, x, cols / 4);
        return;
    }
    long long blocks = (rows * 32 + 255) / 256, cap = (long long)sms * 16;
    if (blocks > cap) blocks = cap;
    quantize_int8_kernel<<<(unsigned)(blocks < 1 ? 1 : blocks), 256, 0, st>>>(q, e, x, rows, cols);
}

__global__ void dequantize_int8_kernel(float *__restrict__ y, const signed char *__restrict__ q,
                                       const int *__restrict__ e, long long rows, long long cols) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long total = rows * cols;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const long long r = i / cols;
        y[i] = dequant_int8_pow2((int)q[i], pow2_f32(__ldg(e + r)));
    }
}

// int32 accumulator to float32 by the pinned spelling: a 20-bit high part and
// a 12-bit low part, both exact, one exact scaling, ONE rounding addition.
__device__ __forceinline__ float i32_to_f32_pinned(int v) {
    const bool neg = v < 0;
    const unsigned mag = neg ? (unsigned)(-(long long)v) : (unsigned)v;
    const float hi = (float)(int)(mag >> 12), lo = (float)(int)(mag & 0xFFFu);
    const float r = __fadd_rn(__fmul_rn(hi, 4096.0f), lo);
    return neg ? -r : r;
}

// int8i32.v1 at OP_NT, one thread per cell: order cannot move a bit of an
// exact integer sum, so the walk uses 4-wide dot products where aligned.
__global__ void gemm_int8_flat_kernel(float *__restrict__ c, const signed char *__restrict__ qa,
                                      const int *__restrict__ ea, const signed char *__restrict__ qb,
                                      const int *__restrict__ eb, int m, int n, int k) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)m * n) return;
    const int i = (int)(idx / n), j = (int)(idx % n);
    const signed char *ra = qa + (size_t)i * k, *rb = qb + (size_t)j * k;
    int acc = 0;
    int p = 0;
    if ((k & 3) == 0 && ((reinterpret_cast<uintptr_t>(qa) | reinterpret_cast<uintptr_t>(qb)) & 3) == 0)
        for (; p + 3 < k; p += 4)
            acc = __dp4a(*reinterpret_cast<const int *>(ra + p), *reinterpret_cast<const int *>(rb + p), acc);
    for (; p < k; p++) acc += (int)ra[p] * (int)rb[p];
    const long long esum = (long long)ea[i] + (long long)eb[j];
    const int eclamped = esum > 1000 ? 1000 : (esum < -1000 ? -1000 : (int)esum);
    c[idx] = nan_canon(ftz_bits(__fmul_rn(i32_to_f32_pinned(acc), pow2_f32(eclamped))));
}

// Peak-rate probe for the roofline denominator: 16 independent accumulator
// chains per thread of bare fused multiply-adds, scalar (packed == 0) or as
// fma.rn.f32x2 pairs (packed == 1). 2 * 16 * iters flops per thread (scalar),
// twice that packed. The sum is stored so the chains cannot be removed.
__global__ void ffma_probe_kernel(float *out, int iters, int packed, float seed) {
    float x = seed + (float)threadIdx.x * 1e-9f, y = 0.999f;
    if (packed) {
        unsigned long long acc[16];
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] = pack2(x + i, x - i);
        const unsigned long long m2 = pack2(y, y), a2 = pack2(1e-3f, 2e-3f);
        for (int it = 0; it < iters; it++) {
#pragma unroll
            for (int i = 0; i < 16; i++) acc[i] = fma2_bare(acc[i], m2, a2);
        }
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) { float lo, hi; unpack2(acc[i], lo, hi); s += lo + hi; }
        if (s == 123.456f) out[0] = s;
    } else {
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; i++) acc[i] = x + i;
        for (int it = 0; it < iters; it++) {
#pragma unroll
            for (int i = 0; i < 16; i++) acc[i] = __fmaf_rn(acc[i], y, 1e-3f);
        }
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) s += acc[i];
        if (s == 123.456f) out[0] = s;
    }
}

} // namespace b200i
