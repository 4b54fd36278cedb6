// A^T B of tall operands: few output cells, very many rows contracted (Gram matrices, normal equations, covariance).
//
// The tile plans cut k into at most MAX_GROUPS leaf groups, so a 32 x 32 product over a million rows ran as 64 CTAs that
// each walked 16 leaves of 977 serial steps: 1.19 ms against 0.04 ms for the 256 MB it reads. Here every leaf of every
// 32 x 32 tile is a task of its own:
//
//   - gemm_tall_kernel: ONE WARP per (leaf, tile), a CTA of 32 threads. In OP_TN both operands are stored row by row of
//     k, so a leaf is a contiguous slab of each; the warp streams it through its own ring of 16-step windows with
//     cp.async (16 bytes per lane where the rows allow it, else 4), with no barrier wider than the warp. A thread owns
//     8 x 4 cells as pairs along m, so the left operand's pairs come out of shared memory ready and only the four words
//     of the right operand are doubled: 3 LDS.128 + 16 fma.rn.f32x2 per step. Each lane takes the admission keys of the
//     words it copied itself; the vote that publishes the window is also the warp's barrier.
//   - fold_deep_kernel: up to 1024 nodes per cell, cut into aligned blocks of 2^SUB nodes that are folded by different
//     warps and whose roots form the same adjacent-pair tree SUB levels up.
//
// Bound: HBM and the fma pipe together (32 x 32: 8 flops per byte, both floors near 0.03 to 0.04 ms at a million rows).
// Measured, a million rows: 32 x 32 1187 -> 69 us, fold included. Up to 128 x 128 every shape tried from 2048 rows on is at
// least as fast as the best tile split (128 x 128 over 131072 rows: 203 against 214 us; over 2048: both launch-bound), so
// the rule asks only for sixteen leaves.
#pragma once
#include "gemm_tile.cuh"

namespace b200i {

constexpr int TALL_TILE = 32;
constexpr int TALL_STAGES = 5;
constexpr int TALL_STAGE_FLOATS = KS * 2 * TALL_TILE; // a window's 16 rows: 32 words of A, 32 words of B
constexpr int TALL_MAX_EXTENT = 128;

struct TallArgs {
    const float *a, *b; // [k][m], [k][n]
    float *nodes;       // [leaves][m][n]
    int m, n, k, leaf, tiles_m, tiles_n;
};

__device__ __forceinline__ void tall_copy16(float *dst, const float *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tall_copy4(float *dst, const float *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// VEC: both operands' rows are whole 16-byte words (m % 4 == 0, n % 4 == 0, 16-byte aligned storage).
template <bool VEC>
__global__ void __launch_bounds__(32) gemm_tall_kernel(const TallArgs g) {
    __shared__ __align__(16) float ring[TALL_STAGES][TALL_STAGE_FLOATS];
    const int lane = threadIdx.x;
    const int tm = blockIdx.x / g.tiles_n, tn = blockIdx.x % g.tiles_n, t = blockIdx.y;
    const int i0 = tm * TALL_TILE, j0 = tn * TALL_TILE;
    const int kb = t * g.leaf, leaf_len = min(g.leaf, g.k - kb);
    const int windows = (leaf_len + KS - 1) / KS;

    // A lane copies the same column of one operand in every window: words [q, q + 3] of rows 2u + lane / 16 (VEC), or word
    // `lane` of every row of both. Its source pointer moves one window at a time.
    const int q = (lane & 15) * 4;
    const bool left = q < TALL_TILE;
    const int col = left ? i0 + q : j0 + q - TALL_TILE, ld = left ? g.m : g.n;
    const bool in = VEC ? col < ld : false;
    const float *src = in ? (left ? g.a : g.b) + (size_t)(kb + (lane >> 4)) * ld + col : g.a;
    const size_t two_rows = in ? (size_t)2 * ld : 0, window_words = in ? (size_t)KS * ld : 0;
    const bool in_a = i0 + lane < g.m, in_b = j0 + lane < g.n;
    auto issue = [&](int w) {
        if (w < windows) {
            float *st = ring[w % TALL_STAGES];
            const int len = min(KS, leaf_len - w * KS);
            if (VEC) {
                float *dst = st + (lane >> 4) * (2 * TALL_TILE) + q;
                const int bytes = in ? 16 : 0; // 0: zero filled
                if (len == KS) {
#pragma unroll
                    for (int u = 0; u < 8; u++) tall_copy16(dst + u * (4 * TALL_TILE), src + u * two_rows, bytes);
                } else {
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const bool row = 2 * u + (lane >> 4) < len;
                        tall_copy16(dst + u * (4 * TALL_TILE), row ? src + u * two_rows : g.a, row ? bytes : 0);
                    }
                }
                src += window_words;
            } else {
                const float *pa = g.a + (size_t)(kb + w * KS) * g.m + i0 + lane, *pb = g.b + (size_t)(kb + w * KS) * g.n + j0 + lane;
#pragma unroll 4
                for (int r = 0; r < KS; r++) {
                    const bool row = r < len;
                    tall_copy4(st + r * (2 * TALL_TILE) + lane, row && in_a ? pa : g.a, row && in_a ? 4 : 0);
                    tall_copy4(st + r * (2 * TALL_TILE) + TALL_TILE + lane, row && in_b ? pb : g.a, row && in_b ? 4 : 0);
                    pa += g.m;
                    pb += g.n;
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int w = 0; w < TALL_STAGES - 1; w++) issue(w);

    const int tx = lane & 7, ty = lane >> 3; // columns tx*4 .. +3; rows ty*4 .. +3 and 16 + ty*4 .. +3
    unsigned long long acc[4][4];            // [pair of rows][column]
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0ull;

    bool clean = true;
    for (int w = 0; w < windows; w++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(TALL_STAGES - 2) : "memory");
        const float *st = ring[w % TALL_STAGES];
        unsigned key = 0xFFFFFFFFu; // of the words this lane copied: they are visible to it without a barrier
        if (VEC) {
#pragma unroll
            for (int u = 0; u < 8; u++) key = key4(*reinterpret_cast<const float4 *>(st + (2 * u + (lane >> 4)) * (2 * TALL_TILE) + q), key);
        } else {
#pragma unroll 8
            for (int u = 0; u < 32; u++) key = min(key, admit_key(st[u * TALL_TILE + lane]));
        }
        // publishes the window to the warp, and tells that every lane has left the window before it
        const bool admitted = __all_sync(0xFFFFFFFFu, key >= ADMIT_MIN);
        __syncwarp();
        issue(w + TALL_STAGES - 1);
        const int len = min(KS, leaf_len - w * KS);
        clean = clean && admitted;
        if (clean && len == KS) {
#pragma unroll
            for (int kk = 0; kk < KS; kk++) {
                const float *row = st + kk * (2 * TALL_TILE);
                const ulonglong2 alo = *reinterpret_cast<const ulonglong2 *>(row + ty * 4), ahi = *reinterpret_cast<const ulonglong2 *>(row + 16 + ty * 4);
                const float4 bv = *reinterpret_cast<const float4 *>(row + TALL_TILE + tx * 4);
                const unsigned long long av[4] = {alo.x, alo.y, ahi.x, ahi.y};
                const unsigned long long b2[4] = {pack2(bv.x, bv.x), pack2(bv.y, bv.y), pack2(bv.z, bv.z), pack2(bv.w, bv.w)};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = fma2_bare(av[i], b2[j], acc[i][j]);
            }
        } else {
#pragma unroll 1
            for (int kk = 0; kk < len; kk++) { // the defining step: operands flushed, one rounding, flush
                const float *row = st + kk * (2 * TALL_TILE);
                unsigned long long av[4], b2[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float *p = row + (i >> 1) * 16 + ty * 4 + (i & 1) * 2;
                    av[i] = pack2(ftz_bits(p[0]), ftz_bits(p[1]));
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float v = ftz_bits(row[TALL_TILE + tx * 4 + j]);
                    b2[j] = pack2(v, v);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = ftz2_hw(fma2_bare(av[i], b2[j], acc[i][j]));
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    float *out = g.nodes + (size_t)t * (size_t)g.m * (size_t)g.n;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; j++) unpack2(ftz2_hw(acc[i][j]), lo[j], hi[j]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int row = i0 + (i >> 1) * 16 + ty * 4 + (i & 1) * 2 + h, col = j0 + tx * 4;
            const float *v = h ? hi : lo;
            if (row >= g.m) continue;
            float *dst = out + (size_t)row * g.n + col;
            if (VEC) { // n % 4 == 0: the quad is inside the row or past it
                if (col < g.n) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (col + e < g.n) dst[e] = v[e];
            }
        }
    }
}

// One lane per cell, one warp per aligned block of 2^SUB nodes (the last one possibly ragged); warp 0 folds the block
// roots. grid.x = ceil(cells / 32), block = 32 * ceil(nodes / 2^SUB) <= 1024 threads.
template <int SUB>
__global__ void __launch_bounds__(1024) fold_deep_kernel(const float *__restrict__ ws, float *__restrict__ c, long long cells, int nodes, Epilogue epi,
                                                         int n) {
    __shared__ float roots[32][32];
    const int lane = threadIdx.x & 31, sub = threadIdx.x >> 5, subs = blockDim.x >> 5;
    const long long idx = (long long)blockIdx.x * 32 + lane;
    const bool live = idx < cells;
    const int g0 = sub << SUB, count = min(1 << SUB, nodes - g0);
    if (live) {
        float stack[SUB][1], v[1] = {0.f}, x[1 << SUB];
#pragma unroll
        for (int j = 0; j < (1 << SUB); j++) // all in flight
            if (j < count) x[j] = __ldcg(ws + (size_t)(g0 + j) * (size_t)cells + idx);
#pragma unroll
        for (int j = 0; j < (1 << SUB); j++)
            if (j < count) {
                v[0] = x[j];
                fold_push<1, SUB>(stack, v, j, count - 1);
            }
        roots[sub][lane] = v[0];
    }
    __syncthreads();
    if (sub != 0 || !live) return;
    float stack[5][1], v[1] = {0.f};
    for (int s = 0; s < subs; s++) {
        v[0] = roots[s][lane];
        fold_push<1, 5>(stack, v, s, subs - 1);
    }
    fold_finish<1>(v, c, idx, epi, n);
}

inline void launch_fold_deep(const float *ws, float *c, long long cells, int nodes, cudaStream_t st, Epilogue epi, int n) {
    const unsigned grid = (unsigned)((cells + 31) / 32);
    if (nodes <= 256) fold_deep_kernel<3><<<grid, 32 * ((nodes + 7) / 8), 0, st>>>(ws, c, cells, nodes, epi, n);
    else fold_deep_kernel<5><<<grid, 32 * ((nodes + 31) / 32), 0, st>>>(ws, c, cells, nodes, epi, n);
}

inline size_t tall_workspace_bytes(long long m, long long n, long long k) { return (size_t)leaf_count(k) * (size_t)m * (size_t)n * 4; }

inline void launch_tall(const GemmArgs &g, cudaStream_t st) {
    TallArgs t{g.a, static_cast<const float *>(g.b), g.ws, g.m, g.n, g.k, g.leaf, (g.m + TALL_TILE - 1) / TALL_TILE, (g.n + TALL_TILE - 1) / TALL_TILE};
    const dim3 grid((unsigned)(t.tiles_m * t.tiles_n), (unsigned)g.leaves); // the tiles of a leaf run side by side and share its rows in L2
    const bool vec = g.m % 4 == 0 && g.n % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(g.a) | reinterpret_cast<uintptr_t>(g.b) | reinterpret_cast<uintptr_t>(g.ws)) & 15u) == 0;
    if (vec) gemm_tall_kernel<true><<<grid, 32, 0, st>>>(t);
    else gemm_tall_kernel<false><<<grid, 32, 0, st>>>(t);
    launch_fold_deep(g.ws, g.c, (long long)g.m * g.n, g.leaves, st, g.epi, g.n);
}

} // namespace b200i
