// The large identical-mode product on packed operands: a warp-specialised,
// bulk-copy fed version of the 128 x 128 tile plan.
//
// Numerical plan: the contract's (see gemm_tile.cuh). Execution plan for B200:
//
//   1. pack_operands_kernel rewrites each operand once per product into tile-major
//      panels P[tile][k][128]: 128 rows (or columns) of the operand side by side
//      for every k, already materialised to float32 (bf16 widened, int8
//      dequantised) and flushed, rows past the edge zero. It also writes one
//      admission flag per (tile, 16-step window): 1 when every word of the window
//      passes the admission test of seams.cuh. The pass moves (m + n) * k words,
//      against m * n * k fused multiply-adds in the product.
//   2. gemm_packed_kernel: a CTA owns a 128 x 128 output tile. In panel layout the operands of a stage (32 k-steps, two
//      admission windows) are ONE contiguous 16 KB block each, so one lane streams them into a ring of shared-memory stages
//      with two cp.async.bulk copies per stage (completion on an mbarrier), refilling the slot of the stage before the one
//      its warp has just finished; the eight warps take turns at that. Nothing is staged through registers, no CTA-wide
//      barrier sits in the k loop, and the admission test is a flag read a stage ahead. A consumer thread owns 8 x 8 cells
//      as packed pairs (fma.rn.f32x2), exactly the inner loop of the tile kernel, and folds its leaves on a stack whose two
//      lower levels are its own columns of tensor memory.
//
// Bound: the fma pipe. The inner loop alone, operands resident, runs at 66.9 TFLOP/s (73.3 for bare packed fmas); the kernel
// at 59.1 on 4096^3 (56.3 with six one-window stages issued by thread 0, the whole stack in local memory and tiles in row
// order), 59.3 on 4096 x 2048 x 8192 (57.4), 59.1 on 8192^2 x 1024 (58.9). A thread tile of 8 x 16 with 128 threads has the
// faster inner loop (68.2) and the slower kernel (52.6 on 4096^3): two warps per scheduler do not hide a stage's start.
//
// Every wait on an mbarrier is bounded; one that runs out sets the status word
// read by b200i_decode_status (4 = producer, 5 = consumer) and the kernel runs on
// to its end without the data.
#pragma once
#include "decode.cuh"
#include "gemm_tile.cuh"

namespace b200i {

constexpr int PK_TILE = 128;                        // rows of A / columns of B per panel and per CTA
constexpr int PK_SK = 2 * KS;                       // k-steps per ring stage: two admission windows
constexpr int PK_STAGES = 3;
constexpr int PK_BAND = 16;
constexpr int PK_STAGE_FLOATS = 2 * PK_SK * PK_TILE; // A then B
constexpr int PK_TM = 8, PK_TN = 8, PK_CELLS = PK_TM * PK_TN;
constexpr int PK_CONSUMERS = PK_TILE * PK_TILE / PK_CELLS / 32; // warps
constexpr int PK_TMEM_LEVELS = 2;                   // levels of the fold stack that live in tensor memory
constexpr unsigned PK_TMEM_COLS = PK_TMEM_LEVELS * PK_CELLS * (PK_CONSUMERS / 4); // 256 of 512 columns: two CTAs per SM
constexpr int PK_THREADS = 32 * PK_CONSUMERS;
constexpr int PK_SMEM_BYTES = PK_STAGES * PK_STAGE_FLOATS * 4 + 2 * PK_STAGES * 8 + 16; // ring, barriers, tensor-memory address

__host__ __device__ inline int pk_windows_per_leaf(int leaf) { return (leaf + KS - 1) / KS; }
inline size_t pk_panel_floats(long long extent, long long k) { return (size_t)((extent + PK_TILE - 1) / PK_TILE) * PK_TILE * (size_t)k; }
inline size_t pk_flag_bytes(long long extent, long long k) {
    const size_t n = (size_t)((extent + PK_TILE - 1) / PK_TILE) * (size_t)leaf_count(k) * (size_t)pk_windows_per_leaf((int)leaf_size(k));
    return (n + 255) / 256 * 256;
}
// scratch of the packed plan for one product, group nodes excluded
inline size_t pk_workspace_bytes(long long m, long long n, long long k) {
    return (pk_panel_floats(m, k) + pk_panel_floats(n, k)) * 4 + pk_flag_bytes(m, k) + pk_flag_bytes(n, k);
}

struct PackArgs {
    float *panel;
    unsigned char *flags;
    const void *x;
    const void *scale;
    int extent, k, leaf, leaves, wpl;
    int kcontig; // 1: x is [extent][k]; 0: x is [k][extent]
    int vec;     // four consecutive elements may be read at once (every quad of a row starts on a 4-element boundary)
};

__device__ __forceinline__ float pk_element(const void *x, const void *scale, int wkind, size_t off, int row) {
    if (wkind == W_F32) return ftz_bits(__ldg(static_cast<const float *>(x) + off));
    if (wkind == W_BF16) return ftz_bits(bf16_bits_to_f32(__ldg(static_cast<const unsigned short *>(x) + off)));
    const float f = (wkind == W_INT8_EXP) ? pow2_f32(__ldg(static_cast<const int *>(scale) + row)) : __ldg(static_cast<const float *>(scale) + row);
    return dequant_int8_pow2((int)__ldg(static_cast<const signed char *>(x) + off), f);
}

// Both operands of a product in one launch: grid.x walks the (leaf, pair of windows) blocks, grid.y the tiles of A, then
// those of B. A block of 256 threads moves 128 rows x 32 k-steps. k-contiguous operands are read 128 bytes of a row at a
// time (eight lanes, four rows per warp instruction, four such reads in flight) and turned through shared memory, whose
// 4-word groups are permuted by the lane's k group so that both the turned stores and the 16-byte reads are free of
// conflicts; operands stored row by row of k are copied straight through registers. Every panel row leaves as 512
// contiguous bytes. Bound: HBM, 8 bytes per float32 word. One block per leaf of 128 steps (the split before) left
// 64 blocks on a 1000 x 1000 operand and a CTA barrier between its loads: 39 us there, 13 us at [128, 4096].
constexpr int PACK_K = 2 * KS;

// four consecutive elements starting at `off` as float32 words, exact
template <int WK>
__device__ __forceinline__ float4 pk_quad(const void *x, const void *scale, size_t off, int row) {
    float4 v;
    if (WK == W_F32) {
        v = __ldg(reinterpret_cast<const float4 *>(static_cast<const float *>(x) + off));
    } else if (WK == W_BF16) {
        const uint2 w = __ldg(reinterpret_cast<const uint2 *>(static_cast<const unsigned short *>(x) + off));
        v = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xFFFF0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xFFFF0000u));
    } else {
        const unsigned w = __ldg(reinterpret_cast<const unsigned *>(static_cast<const signed char *>(x) + off));
        const float f = (WK == W_INT8_EXP) ? pow2_f32(__ldg(static_cast<const int *>(scale) + row)) : __ldg(static_cast<const float *>(scale) + row);
        v = make_float4(dequant_int8_pow2((int)(signed char)(w & 0xFFu), f), dequant_int8_pow2((int)(signed char)((w >> 8) & 0xFFu), f),
                        dequant_int8_pow2((int)(signed char)((w >> 16) & 0xFFu), f), dequant_int8_pow2((int)(signed char)(w >> 24), f));
    }
    return make_float4(ftz_bits(v.x), ftz_bits(v.y), ftz_bits(v.z), ftz_bits(v.w));
}

template <int WK>
__device__ __forceinline__ void pack_block(const PackArgs &a, int tile, float (*turn)[PK_TILE], int (*ok)[2]) {
    const int cpl = (a.wpl + 1) / 2; // blocks per leaf
    const int t = blockIdx.x / cpl, w0 = (blockIdx.x % cpl) * 2;
    const int kb = t * a.leaf, leaf_len = min(a.leaf, a.k - kb), k0 = kb + w0 * KS;
    const int len = min(PACK_K, leaf_len - w0 * KS); // k-steps of this block; <= 0 past the end of a short last leaf
    if (len <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, row0 = tile * PK_TILE;
    float *panel = a.panel + (size_t)tile * (size_t)a.k * PK_TILE + (size_t)k0 * PK_TILE;
    unsigned key[2] = {0xFFFFFFFFu, 0xFFFFFFFFu}; // of the words this thread moved, by window
    if (a.kcontig) {
        const int kq = lane & 7; // k-steps kq * 4 .. + 3
        float4 v[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int r = p * 32 + warp * 4 + (lane >> 3), row = row0 + r;
            v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < a.extent && kq * 4 < len) {
                const size_t off = (size_t)row * a.k + k0 + kq * 4;
                if (a.vec && kq * 4 + 3 < len) {
                    v[p] = pk_quad<WK>(a.x, a.scale, off, row);
                } else {
                    v[p].x = pk_element(a.x, a.scale, WK, off, row);
                    if (kq * 4 + 1 < len) v[p].y = pk_element(a.x, a.scale, WK, off + 1, row);
                    if (kq * 4 + 2 < len) v[p].z = pk_element(a.x, a.scale, WK, off + 2, row);
                    if (kq * 4 + 3 < len) v[p].w = pk_element(a.x, a.scale, WK, off + 3, row);
                }
            }
        }
        unsigned mine = 0xFFFFFFFFu;
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int r = (p * 32 + warp * 4 + (lane >> 3)) ^ (kq * 4);
            mine = key4(v[p], mine);
            turn[kq * 4 + 0][r] = v[p].x;
            turn[kq * 4 + 1][r] = v[p].y;
            turn[kq * 4 + 2][r] = v[p].z;
            turn[kq * 4 + 3][r] = v[p].w;
        }
        key[0] = kq < 4 ? mine : 0xFFFFFFFFu;
        key[1] = kq < 4 ? 0xFFFFFFFFu : mine;
        __syncthreads();
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int kk = p * 8 + warp;
            if (kk < len)
                *reinterpret_cast<float4 *>(panel + (size_t)kk * PK_TILE + lane * 4) = *reinterpret_cast<const float4 *>(&turn[kk][(lane * 4) ^ ((kk >> 2) * 4)]);
        }
    } else {
        float4 v[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int kk = p * 8 + warp, row = row0 + lane * 4;
            v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (kk < len && row < a.extent) {
                const size_t off = (size_t)(k0 + kk) * a.extent + row;
                if (a.vec && row + 3 < a.extent) {
                    v[p] = pk_quad<WK>(a.x, a.scale, off, row);
                } else {
                    v[p].x = pk_element(a.x, a.scale, WK, off, row);
                    if (row + 1 < a.extent) v[p].y = pk_element(a.x, a.scale, WK, off + 1, row + 1);
                    if (row + 2 < a.extent) v[p].z = pk_element(a.x, a.scale, WK, off + 2, row + 2);
                    if (row + 3 < a.extent) v[p].w = pk_element(a.x, a.scale, WK, off + 3, row + 3);
                }
            }
        }
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const int kk = p * 8 + warp;
            key[p >> 1] = key4(v[p], key[p >> 1]);
            if (kk < len) *reinterpret_cast<float4 *>(panel + (size_t)kk * PK_TILE + lane * 4) = v[p];
        }
    }
#pragma unroll
    for (int w = 0; w < 2; w++) {
        const bool all = __all_sync(0xFFFFFFFFu, key[w] >= ADMIT_MIN);
        if (lane == 0) ok[warp][w] = all ? 1 : 0;
    }
    __syncthreads();
    if (tid < 2 && tid * KS < len) {
        int all = 1;
#pragma unroll
        for (int w = 0; w < 8; w++) all &= ok[w][tid];
        a.flags[((size_t)tile * a.leaves + t) * a.wpl + w0 + tid] = (unsigned char)all;
    }
}

// Six blocks on an SM for float32 (40 registers); eight for the low-bit kinds (32), whose quads are 8 or 4 bytes, so that a block
// has fewer bytes in flight: packing and fold of a 128 x 11008 x 4096 product 76.4 us with bf16 weights and 73.4 with scaled
// int8 ones at six blocks, 70.3 and 66.6 at eight.
template <int WK>
__global__ void __launch_bounds__(256, WK == W_F32 ? 6 : 8) pack_operands_kernel(const PackArgs a, const PackArgs b, int tiles_a, int first_tile) {
    __shared__ __align__(16) float turn[PACK_K][PK_TILE];
    __shared__ int ok[8][2];
    const int tile = (int)blockIdx.y + first_tile;
    if (tile < tiles_a) pack_block<W_F32>(a, tile, turn, ok);
    else pack_block<WK>(b, tile - tiles_a, turn, ok);
}

// shared memory of the form that reads B's rows itself: A ring, two raw stages of B, two turned ones
constexpr int PK_HALF_FLOATS = PK_SK * PK_TILE; // one operand's stage
constexpr int PK_RAW_STAGES = 2;
constexpr int PK_RAW_SMEM_BYTES = (PK_STAGES + PK_RAW_STAGES + 2) * PK_HALF_FLOATS * 4 + 2 * PK_STAGES * 8 + 16;

struct PackedGemmArgs {
    const float *pa, *pb;               // panels
    const unsigned char *fa, *fb;       // window flags
    float *c, *ws;
    int m, n, k, leaf, leaves, wpl;
    int group_leaves, groups, tiles_n, vec_c;
    const float *braw = nullptr; // RAWB: B itself, [n][k] float32, 16-byte rows
};

// 32 of the calling lane's tensor-memory words as 16 pairs, and back. A warp reaches the 32 lanes of its quarter.
__device__ __forceinline__ void pk_tmem_store(unsigned addr, const unsigned long long *v) {
    unsigned w[32];
#pragma unroll
    for (int i = 0; i < 16; i++) asm("mov.b64 {%0, %1}, %2;" : "=r"(w[2 * i]), "=r"(w[2 * i + 1]) : "l"(v[i]));
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
        "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
        "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]),
        "r"(w[13]), "r"(w[14]), "r"(w[15]), "r"(w[16]), "r"(w[17]), "r"(w[18]), "r"(w[19]), "r"(w[20]), "r"(w[21]), "r"(w[22]), "r"(w[23]), "r"(w[24]),
        "r"(w[25]), "r"(w[26]), "r"(w[27]), "r"(w[28]), "r"(w[29]), "r"(w[30]), "r"(w[31])
        : "memory");
}
__device__ __forceinline__ void pk_tmem_load(unsigned addr, unsigned long long *v) {
    unsigned w[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]), "=r"(w[8]), "=r"(w[9]), "=r"(w[10]), "=r"(w[11]),
          "=r"(w[12]), "=r"(w[13]), "=r"(w[14]), "=r"(w[15]), "=r"(w[16]), "=r"(w[17]), "=r"(w[18]), "=r"(w[19]), "=r"(w[20]), "=r"(w[21]), "=r"(w[22]),
          "=r"(w[23]), "=r"(w[24]), "=r"(w[25]), "=r"(w[26]), "=r"(w[27]), "=r"(w[28]), "=r"(w[29]), "=r"(w[30]), "=r"(w[31])
        : "r"(addr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) asm("mov.b64 %0, {%1, %2};" : "=l"(v[i]) : "r"(w[2 * i]), "r"(w[2 * i + 1]));
}
// fold_add of two pairs of flushed words (see add_flushed)
__device__ __forceinline__ unsigned long long add2_flushed(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// RAWB: a product of one row of tiles uses each panel of B once, so packing B would write and read it again for nothing
// (128 x 11008 x 4096: 72 of 307 us). The CTA then fetches the rows itself by cp.async, and each thread turns the pieces
// that it copied, under the barrier that publishes a stage and its verdict: 260 us, the kernel's 222 having become 246.
template <bool RAWB>
__global__ void __launch_bounds__(PK_THREADS, 2) gemm_packed_kernel(const PackedGemmArgs g) {
    constexpr int STAGE_FLOATS = RAWB ? PK_HALF_FLOATS : PK_STAGE_FLOATS; // of the bulk-copied ring
    constexpr int TM = PK_TM, TN = PK_TN, PAIRS = PK_CELLS / 2, LOCAL_LEVELS = FOLD_LEVELS - PK_TMEM_LEVELS;
    extern __shared__ __align__(128) float pk_smem[];
    float *raw = pk_smem + PK_STAGES * STAGE_FLOATS, *turned = raw + PK_RAW_STAGES * PK_HALF_FLOATS; // RAWB only
    unsigned long long *full = reinterpret_cast<unsigned long long *>(RAWB ? turned + 2 * PK_HALF_FLOATS : raw);
    unsigned long long *empty = full + PK_STAGES;
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(empty + PK_STAGES);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Tiles go in bands of PK_BAND tile rows, down a band's column before the next column: the 296 CTAs of a wave then read
    // sixteen panels of A and about nineteen of B, where a walk along the rows read two and 296
    const int tiles_m = (g.m + PK_TILE - 1) / PK_TILE, band = (int)blockIdx.x / (PK_BAND * g.tiles_n), in_band = (int)blockIdx.x - band * PK_BAND * g.tiles_n;
    const int band_rows = min(PK_BAND, tiles_m - band * PK_BAND);
    const int tile_m = band * PK_BAND + in_band % band_rows, tile_n = in_band / band_rows;
    const int t_first = blockIdx.y * g.group_leaves;
    const int t_end = min(t_first + g.group_leaves, g.leaves);

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < PK_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], PK_CONSUMERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(PK_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot, tmem_mine = tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)((warp >> 2) * PK_TMEM_LEVELS * PK_CELLS);

    // ---- the copy stream, PK_STAGES - 1 stages ahead of the compute. Every warp keeps its place in it; a stage is issued by
    // one lane of the warp whose turn it is, so that no warp runs behind the others for it ----
    const float *pa = g.pa + (size_t)tile_m * (size_t)g.k * PK_TILE;
    const float *pb = g.pb + (size_t)tile_n * (size_t)g.k * PK_TILE;
    int pt = t_first, pkoff = 0, pslot = 0; // next stage to copy
    auto issue_next = [&](bool mine) {
        if (pt >= t_end) return;
        const int kb = pt * g.leaf, leaf_len = min(g.leaf, g.k - kb);
        if (mine) {
            float *dst = pk_smem + pslot * STAGE_FLOATS;
            const unsigned bytes = (unsigned)min(PK_SK, leaf_len - pkoff) * PK_TILE * 4u;
            mbar_expect_tx(&full[pslot], RAWB ? bytes : 2u * bytes);
            bulk_copy_g2s(dst, pa + (size_t)(kb + pkoff) * PK_TILE, bytes, &full[pslot]);
            if (!RAWB) bulk_copy_g2s(dst + PK_HALF_FLOATS, pb + (size_t)(kb + pkoff) * PK_TILE, bytes, &full[pslot]);
        }
        if (++pslot == PK_STAGES) pslot = 0;
        pkoff += PK_SK;
        if (pkoff >= leaf_len) { pkoff = 0; pt++; }
    };
    for (int i = 0; i < PK_STAGES - 1; i++) issue_next(tid == 0);

    constexpr int TXN = PK_TILE / TN, CSTEP = 4 * TXN; // rows ty*4 .. +3 and 64 + ty*4 .. +3; columns r*CSTEP + tx*4 .. +3
    const int tx = tid % TXN, ty = tid / TXN;
    const int wpl = g.wpl;
    const unsigned char *fa = g.fa + (size_t)tile_m * g.leaves * wpl;
    const unsigned char *fb = g.fb + (size_t)tile_n * g.leaves * wpl;

    unsigned long long acc[PAIRS]; // [row][pair of columns]
#pragma unroll
    for (int i = 0; i < PAIRS; i++) acc[i] = 0ull;
    unsigned long long local_stack[LOCAL_LEVELS][PAIRS];

    auto step = [&](const float *as, const float *bs, int kk, bool flush) { // panel words are already flushed, B's own rows not
        const int sw = RAWB ? ((kk >> 2) & 7) * 4 : 0;
        float av[TM];
        unsigned long long b2[TN / 2];
#pragma unroll
        for (int r = 0; r < TM / 4; r++) {
            const float4 v = *reinterpret_cast<const float4 *>(as + kk * PK_TILE + r * 64 + ty * 4);
            av[4 * r + 0] = v.x; av[4 * r + 1] = v.y; av[4 * r + 2] = v.z; av[4 * r + 3] = v.w;
        }
#pragma unroll
        for (int r = 0; r < TN / 4; r++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(bs + kk * PK_TILE + ((r * CSTEP + tx * 4) ^ sw));
            b2[2 * r] = v.x;
            b2[2 * r + 1] = v.y;
        }
        if (RAWB && flush) {
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
                float lo, hi;
                unpack2(b2[j], lo, hi);
                b2[j] = pack2(ftz_bits(lo), ftz_bits(hi));
            }
        }
#pragma unroll
        for (int i = 0; i < TM; i++) {
            const unsigned long long a2 = pack2(av[i], av[i]);
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
                const unsigned long long d = fma2_bare(a2, b2[j], acc[i * (TN / 2) + j]);
                acc[i * (TN / 2) + j] = flush ? ftz2_hw(d) : d;
            }
        }
    };
    // The accumulators as the node of one finished leaf, merged with the stack levels below the counter's lowest clear
    // bit: levels 0 and 1 (three of every four pushes and merges) in tensor memory, the rest in local memory.
    auto merge = [&](int lvl) {
        if (lvl < PK_TMEM_LEVELS) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < PAIRS; c += 16) {
                unsigned long long t[16];
                pk_tmem_load(tmem_mine + (unsigned)(lvl * PK_CELLS + 2 * c), t);
#pragma unroll
                for (int i = 0; i < 16; i++) acc[c + i] = add2_flushed(t[i], acc[c + i]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < PAIRS; c++) acc[c] = add2_flushed(local_stack[lvl - PK_TMEM_LEVELS][c], acc[c]);
        }
    };
    auto push_leaf = [&](int local_leaf) {
        __syncwarp(); // the tensor-memory instructions are the whole warp's
#pragma unroll
        for (int c = 0; c < PAIRS; c++) acc[c] = ftz2_hw(acc[c]);
        int lvl = 0;
#pragma unroll 1
        for (int bits = local_leaf; bits & 1; bits >>= 1, lvl++) merge(lvl);
        if (lvl < PK_TMEM_LEVELS) {
#pragma unroll
            for (int c = 0; c < PAIRS; c += 16) pk_tmem_store(tmem_mine + (unsigned)(lvl * PK_CELLS + 2 * c), &acc[c]);
        } else {
#pragma unroll
            for (int c = 0; c < PAIRS; c++) local_stack[lvl - PK_TMEM_LEVELS][c] = acc[c];
        }
#pragma unroll
        for (int c = 0; c < PAIRS; c++) acc[c] = 0ull;
    };

    int stage = 0, turn = 0;
    unsigned phase = 0, prev_phase = 0;
    bool alive = true;
    // RAWB: stage s of B is k-steps [32 s, 32 s + 32) of the CTA's range (leaves are whole stages but for the last one). This
    // thread's pieces: k-steps (tid % 8) * 4 .. + 3 of rows u * 32 + tid / 8.
    const int rq = tid & 7, kbase = t_first * g.leaf, klen = min(g.k, t_end * g.leaf) - kbase;
    auto raw_issue = [&](int s) { // one commit always
        if (s * PK_SK < klen) {
            float *dst = raw + (s % PK_RAW_STAGES) * PK_HALF_FLOATS;
            const int kk = s * PK_SK + rq * 4;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int r = u * 32 + (tid >> 3), row = tile_n * PK_TILE + r;
                const bool in = row < g.n && kk < klen; // k is a multiple of 4
                const float *src = in ? g.braw + (size_t)row * g.k + kbase + kk : g.braw;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + (u * 256 + tid) * 4)), "l"(src), "r"(in ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto raw_turn = [&](int s) { // stage s, landed; returns whether this thread's words are admitted
        const float *src = raw + (s % PK_RAW_STAGES) * PK_HALF_FLOATS;
        float *dst = turned + (s & 1) * PK_HALF_FLOATS;
        unsigned key = 0xFFFFFFFFu;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float4 v = *reinterpret_cast<const float4 *>(src + (u * 256 + tid) * 4);
            const int c = (u * 32 + (tid >> 3)) ^ (rq * 4);
            key = key4(v, key);
            dst[(rq * 4 + 0) * PK_TILE + c] = v.x;
            dst[(rq * 4 + 1) * PK_TILE + c] = v.y;
            dst[(rq * 4 + 2) * PK_TILE + c] = v.z;
            dst[(rq * 4 + 3) * PK_TILE + c] = v.w;
        }
        return key >= ADMIT_MIN;
    };
    bool b_mine = true;
    if (RAWB) {
        raw_issue(0);
        raw_issue(1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        b_mine = raw_turn(0);
    }
    // admission flags of a stage's windows, read a stage ahead; the windows of the leaves follow one another
    fa += (size_t)t_first * wpl;
    fb += (size_t)t_first * wpl;
    auto flags = [&](bool second) {
        const unsigned lo = RAWB ? __ldg(fa) : __ldg(fa) & __ldg(fb), hi = !second ? 0u : (unsigned)(RAWB ? __ldg(fa + 1) : __ldg(fa + 1) & __ldg(fb + 1));
        return lo | hi << 1;
    };
    unsigned admitted = flags(min(g.leaf, g.k - t_first * g.leaf) > KS);
    for (int t = t_first; t < t_end; t++) {
        const int kb = t * g.leaf, leaf_len = min(g.leaf, g.k - kb);
        bool leaf_clean = true;
        for (int koff = 0; koff < leaf_len; koff += PK_SK) {
            const int len = min(PK_SK, leaf_len - koff);
            fa += len > KS ? 2 : 1;
            fb += len > KS ? 2 : 1;
            unsigned ahead = 0u;
            const int rest = koff + PK_SK < leaf_len ? leaf_len - koff - PK_SK : (t + 1 < t_end ? min(g.leaf, g.k - kb - g.leaf) : 0);
            if (rest > 0) ahead = flags(rest > KS);
            if (alive && !mbar_wait(&full[stage], phase)) {
                if (lane == 0) atomicExch(&g_decode_status, 5);
                alive = false;
            }
            const float *as = pk_smem + stage * STAGE_FLOATS, *bs = RAWB ? turned + (turn & 1) * PK_HALF_FLOATS : as + PK_HALF_FLOATS;
            if (RAWB) {
                // publishes the turned stage and its verdict; every thread has read its pieces of the raw one and has left
                // the stage before
                if (!__syncthreads_and(b_mine)) admitted = 0u;
                raw_issue(turn + PK_RAW_STAGES);
            }
            if (admitted == 3u && leaf_clean && len == PK_SK) {
#pragma unroll
                for (int kk = 0; kk < PK_SK; kk++) step(as, bs, kk, false);
            } else {
                for (int w = 0; w * KS < len; w++) {
                    if ((admitted >> w) & 1u && leaf_clean && len >= (w + 1) * KS) {
#pragma unroll 2
                        for (int kk = w * KS; kk < (w + 1) * KS; kk++) step(as, bs, kk, false);
                    } else {
                        leaf_clean = false;
#pragma unroll 1
                        for (int kk = w * KS; kk < min(len, (w + 1) * KS); kk++) step(as, bs, kk, true);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[stage]);
            // the slot of the stage before this one takes the stage PK_STAGES - 1 ahead once every warp has left it; they
            // have had a whole stage to do so
            const bool mine = turn % PK_CONSUMERS == warp && lane == 0;
            if (mine && turn >= 1 && pt < t_end && alive && !mbar_wait(&empty[pslot], prev_phase)) {
                atomicExch(&g_decode_status, 4);
                alive = false;
            }
            issue_next(mine);
            turn++;
            if (RAWB) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                if (turn * PK_SK < klen) b_mine = raw_turn(turn);
            }
            admitted = ahead;
            prev_phase = phase; // of the slot that is refilled next: this one
            if (++stage == PK_STAGES) { stage = 0; phase ^= 1u; }
        }
        if (t + 1 < t_end) push_leaf(t - t_first); // the group's last leaf stays in registers for the drain
    }

    __syncwarp();
    const int count = t_end - t_first;
    float *out = g.groups > 1 ? g.ws + (size_t)blockIdx.y * (size_t)g.m * (size_t)g.n : g.c;
#pragma unroll
    for (int c = 0; c < PAIRS; c++) acc[c] = ftz2_hw(acc[c]);
    if (count > 1) {
        const int last = count - 1;
#pragma unroll 1
        for (int lvl = 0; (last >> lvl) != 0; lvl++)
            if ((last >> lvl) & 1) merge(lvl);
    }
    const int bm0 = tile_m * PK_TILE, bn0 = tile_n * PK_TILE;
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int row = bm0 + (i / 4) * 64 + ty * 4 + (i % 4);
        if (row < g.m) {
#pragma unroll
            for (int jr = 0; jr < TN / 4; jr++) {
                float vals[4];
                unpack2(acc[i * (TN / 2) + 2 * jr], vals[0], vals[1]);
                unpack2(acc[i * (TN / 2) + 2 * jr + 1], vals[2], vals[3]);
#pragma unroll
                for (int e = 0; e < 4; e++) vals[e] = nan_canon(vals[e]);
                const int col = bn0 + jr * CSTEP + tx * 4;
                float *dst = out + (size_t)row * (size_t)g.n + col;
                if (g.vec_c && col + 3 < g.n) *reinterpret_cast<float4 *>(dst) = make_float4(vals[0], vals[1], vals[2], vals[3]);
                else
                    for (int e = 0; e < 4; e++)
                        if (col + e < g.n) dst[e] = vals[e];
            }
        }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); // the last push's words, where none was read again
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PK_TMEM_COLS) : "memory");
}

} // namespace b200i
