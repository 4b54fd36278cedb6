// C[m, n] = A[m, k] . W[n, k]^T for 5 to 16 rows over a large float32 or bf16 weight: warps that stream the weight on their own.
//
// The rows, band and skinny kernels bring a weight by 16-byte pieces that a CTA's or a warp's threads ask for one window ahead,
// and walk it between barriers or on short per-warp rings; on float32 weights of tens of millions of words they stay at half of
// the HBM rate ([11008, 4096] at eight rows 57 us for 28 of bytes). Here:
//
//   - one CTA of sixteen warps per SM, the warps independent after one barrier. The work is cut into items (leaf group, unit of
//     64 columns), numbered leaf group by leaf group, and every CTA takes an equal run of them, so it meets at most two leaf
//     groups, whose activations are staged once, [k][MT] with the row quads permuted by k so that the turning stores are free of
//     bank conflicts;
//   - a warp owns an item and brings its weights itself: one tensor-map copy (cp.async.bulk.tensor.2d, 64 bytes of 64 rows,
//     64-byte swizzle) per stage of its own ring, completion on its own mbarriers, refilled by the warp when it has read a slot.
//     No other warp is waited for, and an SM has up to 192 KB in flight. Edges of the weight and the k tail are zero-filled;
//   - a lane owns eight rows (MT rows over RG row groups) by CPL columns, the rows in pairs: one 16-byte read of the activations
//     serves 2 * CPL packed fmas, one 16-byte read of a column serves 4 or 8 k-steps. Bodies of 4, 8 and 16 k-steps, eight and
//     twelve warps and twice the cells per lane measured the same or slower, with the items dealt out as below.
//
// Measured (graph replay, several weights in turn, fold included), the plan before -> this: float32 at eight rows [11008, 4096]
// 56 -> 43 us, [10512, 2256] 47 -> 27, at five [50304, 768] 54 -> 41, at sixteen [39296, 6416] 393 -> 248; bf16 [11008, 4096] at
// eight 42.6 -> 35.4, at sixteen 67.4 -> 58.6. Bound: float32 at eight rows HBM (64 % of the measured copy rate at [11008, 4096]);
// otherwise too few warps with work: a CTA's items rarely divide by sixteen ([11008, 4096] in groups of four: 9.3 of them, so 9.2
// warps are active, issue slots 45 % and fma pipe 36 % busy at eight bf16 rows). Under that split int8 weights measured no faster
// than the rows and register skinny kernels (36 against 34 us at eight rows, 87 against 86 at 32), nor did float32 ones at 32 rows
// (79 to 114 against 85 to 108), so those keep theirs; an even split was not tried.
//
// Admission is per leaf and lane: the activations' keys are taken while they are staged, the weights' while they are widened
// (bf16: two words an instruction, a zero passing as 0xFFFF after the subtraction); a lane whose leaf fails runs the defining
// flushed chain again from global memory. Every wait is bounded and decided by the whole warp: where one runs out the warp sets the
// status (10), asks for no further copy, waits for those in flight (stream_ring.cuh) and leaves its items unwritten.
#pragma once
#include <cuda.h>

#include <algorithm>

#include "gemm_int8_tma.cuh"
#include "gemm_skinny.cuh"
#include "stream_ring.cuh"

namespace b200i {

constexpr int SM_SEG = 64;  // bytes of a weight row per ring stage
constexpr int SM_CB = 64;   // columns of an item
constexpr int SM_WARPS = 16;
constexpr int SM_STEPS = 8; // k-steps of an unrolled body
constexpr int SM_LEAF = 128;
constexpr int SM_MAX_ROWS = 16;
constexpr int SM_SMEM_LIMIT = 225 * 1024;
// The swizzled stages start on multiples of 512 bytes, inside an array that asks for no more than its siblings do: the strictest
// alignment of a library's dynamic shared memory is what the static arrays of all its kernels are rounded up to, and the decode
// attention shares out an SM to the last kilobyte (1024 here took its fourth CTA from an SM).
constexpr int SM_ALIGN = 128, SM_RING_ALIGN = 512;
constexpr int SM_SLABS = 2; // leaf groups whose activations a CTA holds
constexpr int SM_LEVELS = 2, SM_MAX_RUN = 1 << SM_LEVELS; // levels of a lane's fold stack, and the leaves of a group that they hold

struct StreamPlan {
    int units;  // column units
    int items;  // units * groups
    int stages; // of a warp's ring
    int key_off, bar_off, ring_off; // bytes into shared memory
};

template <int WK>
struct StreamKind {
    static constexpr int ES = WK == W_F32 ? 4 : 2;
    static constexpr int KC = SM_SEG / ES; // k-steps per stage
    static constexpr int EPQ = 16 / ES;    // k-steps per 16-byte piece
};

// What the row quad numbers of k-step k are permuted by (exclusive or): 32 / MT k-steps fill the banks once.
template <int MT>
__host__ __device__ constexpr int sm_turn(int k) { return (k / (32 / MT)) & (MT / 4 - 1); }

struct StreamWait { // by a whole warp, with one answer
    unsigned long long *full;
    __device__ __forceinline__ bool operator()(int slot, unsigned phase) const { return __all_sync(0xFFFFFFFFu, mbar_wait(&full[slot], phase)) != 0; }
};
// A warp's wait ran out. (Not inlined: its loop would cost the product's loop registers.)
__device__ __noinline__ void sm_lost(unsigned long long *full, StreamRing flow) {
    if ((threadIdx.x & 31) == 0) atomicExch(&g_decode_status, 10);
    flow.drain(StreamWait{full});
}

template <int WK, int MT, int RG, int CPL>
__global__ void __launch_bounds__(32 * SM_WARPS, 1) gemm_stream_kernel(const __grid_constant__ CUtensorMap wmap, const GemmArgs g, const StreamPlan p) {
    static_assert(WK == W_F32 || WK == W_BF16, "int8 weights keep their kernels");
    using K = StreamKind<WK>;
    constexpr int LC = 32 / RG, CB = LC * CPL, RL = MT / RG, PAIRS = RL / 2, QUADS = RL / 4, CELLS = RL * CPL, NW = SM_WARPS, UN = SM_STEPS;
    constexpr int STAGE = CB * SM_SEG;
    static_assert(STAGE % SM_RING_ALIGN == 0, "every stage starts on one");
    static_assert(CB == SM_CB && sm_turn<MT>(UN) == 0, "the quads' places inside a body are constants");
    extern __shared__ __align__(SM_ALIGN) unsigned char sm_smem[];
    float *act = reinterpret_cast<float *>(sm_smem);
    unsigned *lkey = reinterpret_cast<unsigned *>(sm_smem + p.key_off);
    const int tid = threadIdx.x, lane = tid & 31, stages = p.stages;
    const int warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0); // one value a warp: what follows from it lies in uniform registers
    unsigned long long *full = reinterpret_cast<unsigned long long *>(sm_smem + p.bar_off) + warp * stages;
    const unsigned off = smem_u32(sm_smem) + (unsigned)p.ring_off;
    unsigned char *ring = sm_smem + p.ring_off + ((0u - off) & (SM_RING_ALIGN - 1)) + (size_t)warp * stages * STAGE;

    const int lo = (int)((long long)p.items * blockIdx.x / gridDim.x), hi = (int)((long long)p.items * (blockIdx.x + 1) / gridDim.x);
    const int slab0 = lo / p.units, gl = g.group_leaves;

    if (lane == 0) {
        for (int s = 0; s < stages; s++) mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();

    // ---- the copy stream of this warp: (item, chunk of its leaves) ----
    int p_item = lo + warp, p_k = 0, p_row = 0, p_end = 0;
    auto p_enter = [&]() {
        if (p_item < hi) {
            const int slab = p_item / p.units;
            p_row = (p_item - slab * p.units) * CB;
            p_k = slab * gl * SM_LEAF;
            p_end = min(p_k + gl * SM_LEAF, g.k);
        }
    };
    auto fill = [&](int slot) { // false where the warp's items have no more
        if (p_item >= hi) return false;
        if (lane == 0) {
            mbar_expect_tx(&full[slot], STAGE);
            t8_tma_load(ring + (size_t)slot * STAGE, &wmap, &full[slot], p_k, p_row);
        }
        p_k += K::KC;
        if (p_k >= p_end) {
            p_item += NW;
            p_enter();
        }
        return true;
    };
    StreamRing flow{stages};
    p_enter();
    flow.start(fill);

    // ---- activations of the CTA's leaf groups, rows past m zero; one key per leaf ----
    const int k_first = slab0 * gl * SM_LEAF, k_last = min(min((hi - 1) / p.units + 1, g.groups) * gl * SM_LEAF, g.k), klen = k_last - k_first;
    for (int i = tid; i < SM_SLABS * gl; i += 32 * NW) lkey[i] = 0xFFFFFFFFu;
    __syncthreads();
    for (int k0 = warp * 32; k0 < klen; k0 += 32 * NW) {
        const int kk = k0 + lane;
        float x[MT];
#pragma unroll
        for (int r = 0; r < MT; r++) x[r] = (kk < klen && r < g.m) ? __ldg(g.a + (size_t)r * g.k + k_first + kk) : 0.f;
        unsigned key = 0xFFFFFFFFu;
#pragma unroll
        for (int r = 0; r < MT; r++) key = min(key, admit_key(x[r]));
        if (kk < klen) {
#pragma unroll
            for (int q = 0; q < MT / 4; q++)
                *reinterpret_cast<float4 *>(act + (size_t)kk * MT + (q ^ sm_turn<MT>(kk)) * 4) = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        }
        key = __reduce_min_sync(0xFFFFFFFFu, key);
        if (lane == 0) atomicMin(&lkey[k0 / SM_LEAF], key);
    }
    __syncthreads();

    const int lc = lane % LC, rg = lane / LC;
    const int wswz = (lc >> 1) & 3; // the copy's swizzle: 16-byte pieces of row r lie at piece ^ (r / 2 % 4)
    unsigned long long acc[PAIRS][CPL];
    float stack[SM_LEVELS][CELLS];

    for (int item = lo + warp; item < hi; item += NW) {
        const int slab = item / p.units, col0 = (item - slab * p.units) * CB;
        const int t0 = slab * gl, t1 = min(t0 + gl, g.leaves);
        for (int t = t0; t < t1; t++) {
            const int leaf_len = min(SM_LEAF, g.k - t * SM_LEAF);
            const float *ak = act + (size_t)(t * SM_LEAF - k_first) * MT;
            unsigned key = 0xFFFFFFFFu; // bf16: of two words at a time
#pragma unroll
            for (int i = 0; i < PAIRS; i++)
#pragma unroll
                for (int j = 0; j < CPL; j++) acc[i][j] = 0ull;
            for (int koff = 0; koff < leaf_len; koff += K::KC) {
                if (!StreamWait{full}(flow.slot, flow.phase)) { // (no barrier of the block follows)
                    sm_lost(full, flow);
                    return;
                }
                const unsigned char *st = ring + (size_t)flow.slot * STAGE + lc * SM_SEG;
                const int len = min(K::KC, leaf_len - koff);
#pragma unroll 1
                for (int s = 0; s * UN < len; s++) { // len is a multiple of sixteen
                    const float *arow = ak + (size_t)(koff + s * UN) * MT;
#pragma unroll
                    for (int pp = 0; pp < UN / K::EPQ; pp++) {
                        float v[CPL][K::EPQ];
                        const int place = ((s * (UN / K::EPQ) + pp) ^ wswz) * 16;
#pragma unroll
                        for (int j = 0; j < CPL; j++) {
                            const uint4 w4 = *reinterpret_cast<const uint4 *>(st + j * LC * SM_SEG + place);
                            const unsigned word[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                if (WK == W_F32) {
                                    v[j][e] = __uint_as_float(word[e]);
                                    key = min(key, admit_key(v[j][e]));
                                } else {
                                    v[j][(2 * e) % K::EPQ] = __uint_as_float(word[e] << 16);
                                    v[j][(2 * e + 1) % K::EPQ] = __uint_as_float(word[e] & 0xFFFF0000u);
                                    key = __viaddmin_u16x2(word[e] & 0x7FFF7FFFu, 0xFFFFFFFFu, key);
                                }
                            }
                        }
#pragma unroll
                        for (int e = 0; e < K::EPQ; e++) {
                            const int kk = pp * K::EPQ + e, turn = sm_turn<MT>(kk), low = turn & (QUADS - 1), high = turn - low;
                            const float *row = arow + kk * MT + ((rg * QUADS) ^ high) * 4;
                            unsigned long long a2[PAIRS];
#pragma unroll
                            for (int i = 0; i < QUADS; i++) {
                                const ulonglong2 tt = *reinterpret_cast<const ulonglong2 *>(row + (i ^ low) * 4);
                                a2[2 * i] = tt.x;
                                a2[2 * i + 1] = tt.y;
                            }
#pragma unroll
                            for (int j = 0; j < CPL; j++) {
                                const unsigned long long w2 = pack2(v[j][e], v[j][e]);
#pragma unroll
                                for (int i = 0; i < PAIRS; i++) acc[i][j] = fma2_bare(a2[i], w2, acc[i][j]);
                            }
                        }
                    }
                }
                __syncwarp(); // every lane has read the slot
                flow.release(fill);
            }
            // ---- the leaf's nodes ----
            float v[CELLS];
#pragma unroll
            for (int i = 0; i < PAIRS; i++)
#pragma unroll
                for (int j = 0; j < CPL; j++) unpack2(ftz2_hw(acc[i][j]), v[2 * i * CPL + j], v[(2 * i + 1) * CPL + j]);
            bool ok = lkey[t - slab0 * gl] >= ADMIT_MIN;
            if (WK == W_F32) {
                ok = ok && key >= ADMIT_MIN;
            } else {
                constexpr unsigned least = ADMIT_EXP ? (ADMIT_EXP << 7) - 1u : 0u;
                ok = ok && (key & 0xFFFFu) >= least && (key >> 16) >= least;
            }
            if (!ok) { // this lane's columns again, by the defining step, from global memory
#pragma unroll 1
                for (int j = 0; j < CPL; j++) {
                    const int c = col0 + lc + j * LC;
                    if (c >= g.n) continue;
                    float slow[RL];
#pragma unroll
                    for (int r = 0; r < RL; r++) slow[r] = 0.f;
#pragma unroll 1
                    for (int kk = 0; kk < leaf_len; kk++) {
                        const size_t off = (size_t)c * g.k + (size_t)t * SM_LEAF + kk;
                        const float w = WK == W_F32 ? ftz_bits(__ldg(static_cast<const float *>(g.b) + off))
                                                    : ftz_bits(bf16_bits_to_f32(__ldg(static_cast<const unsigned short *>(g.b) + off)));
#pragma unroll
                        for (int r = 0; r < RL; r++) {
                            const int q = (rg * QUADS + r / 4) ^ sm_turn<MT>(kk);
                            slow[r] = step_flush(ftz_bits(ak[(size_t)kk * MT + q * 4 + (r & 3)]), w, slow[r]);
                        }
                    }
#pragma unroll
                    for (int r = 0; r < RL; r++)
#pragma unroll
                        for (int jj = 0; jj < CPL; jj++)
                            if (jj == j) v[r * CPL + jj] = ftz_hw(slow[r]);
                }
            }
            // the fold of the group's leaves: the binary counter's stack, in local memory
            const int i_leaf = t - t0, last = t1 - t0 - 1;
            if (i_leaf != last) {
                int lvl = 0;
                for (int bits = i_leaf; bits & 1; bits >>= 1, lvl++)
#pragma unroll
                    for (int c = 0; c < CELLS; c++) v[c] = fold_add(stack[lvl][c], v[c]);
#pragma unroll
                for (int c = 0; c < CELLS; c++) stack[lvl][c] = v[c];
            } else {
#pragma unroll 1
                for (int lvl = 0; (last >> lvl) != 0; lvl++)
                    if ((last >> lvl) & 1) {
#pragma unroll
                        for (int c = 0; c < CELLS; c++) v[c] = fold_add(stack[lvl][c], v[c]);
                    }
                float *out = g.groups > 1 ? g.ws + (size_t)slab * (size_t)g.m * (size_t)g.n : g.c;
                const bool pairs = g.groups == 1 && epilogue_pairs(g.epi), on = g.groups == 1 && epilogue_on(g.epi);
#pragma unroll
                for (int r = 0; r < RL; r++) {
                    const int row = rg * RL + r;
#pragma unroll
                    for (int j = 0; j < CPL; j++) {
                        const int c = col0 + lc + j * LC;
                        const float x = nan_canon(v[r * CPL + j]);
                        if (pairs) { // gate and up of a pair are neighbouring lanes
                            const float other = __shfl_xor_sync(0xFFFFFFFFu, x, 1);
                            if (!(lane & 1) && row < g.m && c + 1 < g.n) g.c[(size_t)row * (g.n / 2) + c / 2] = epilogue_pair_apply(x, other, g.epi.bias, g.epi.act, c / 2);
                        } else if (row < g.m && c < g.n) {
                            out[(size_t)row * g.n + c] = on ? epilogue_apply(x, g.epi.bias, g.epi.act, c) : x;
                        }
                    }
                }
            }
        }
    }
}

inline bool sm_make_map(CUtensorMap *map, const GemmArgs &g) {
    T8EncodeFn fn = t8_encode_fn();
    if (!fn) return false;
    const int es = g.wkind == W_F32 ? 4 : 2;
    const cuuint64_t dims[2] = {(cuuint64_t)g.k, (cuuint64_t)g.n}, strides[1] = {(cuuint64_t)g.k * es};
    const cuuint32_t box[2] = {(cuuint32_t)(SM_SEG / es), (cuuint32_t)SM_CB}, estr[2] = {1u, 1u};
    return fn(map, g.wkind == W_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(g.b), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline int stream_mt(long long m) { return m <= 8 ? 8 : 16; }
// leaves in groups of at most SM_MAX_RUN (the lanes' fold stacks), at most two groups of which a CTA meets (groups <= SMs); the
// column units and items are counted in 32 bits
inline bool stream_plan_fits(long long m, long long n, long long k, int op, int wkind, int group_leaves, int sms) {
    const long long leaves = leaf_count(k), run = std::min<long long>(group_leaves, leaves);
    return m <= SM_MAX_ROWS && n <= (1ll << 26) && skinny_plan_fits(m, n, k, op) && leaf_size(k) <= SM_LEAF && (wkind == W_F32 || wkind == W_BF16) &&
           run <= SM_MAX_RUN && (leaves + run - 1) / run <= sms;
}

template <int WK, int MT, int RG, int CPL>
inline void launch_stream_cfg(const CUtensorMap &map, const GemmArgs &g, int sms, cudaStream_t st) {
    StreamPlan p;
    p.units = (g.n + SM_CB - 1) / SM_CB;
    p.items = p.units * g.groups;
    p.key_off = std::min(g.groups, SM_SLABS) * g.group_leaves * SM_LEAF * MT * 4; // at most 64 KB
    p.bar_off = (p.key_off + SM_SLABS * g.group_leaves * 4 + 15) / 16 * 16;
    p.stages = 3; // two where the activations leave no room for three; a stage is 64 KB over the warps
    auto ring = [&](int s) { return (p.bar_off + SM_WARPS * s * 8 + SM_ALIGN - 1) / SM_ALIGN * SM_ALIGN; };
    auto total = [&](int s) { return ring(s) + SM_RING_ALIGN - SM_ALIGN + SM_WARPS * s * SM_CB * SM_SEG; };
    while (total(p.stages) > SM_SMEM_LIMIT) p.stages--;
    p.ring_off = ring(p.stages);
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaFuncSetAttribute(gemm_stream_kernel<WK, MT, RG, CPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, SM_SMEM_LIMIT);
        configured[dev] = true;
    }
    gemm_stream_kernel<WK, MT, RG, CPL><<<std::min(p.items, sms), 32 * SM_WARPS, total(p.stages), st>>>(map, g, p);
}

// false where no tensor map can be made
inline bool launch_stream(const GemmArgs &g, int sms, cudaStream_t st) {
    alignas(64) CUtensorMap map;
    if (!sm_make_map(&map, g)) return false;
    if (g.wkind == W_F32) {
        if (stream_mt(g.m) == 8) launch_stream_cfg<W_F32, 8, 1, 2>(map, g, sms, st);
        else launch_stream_cfg<W_F32, 16, 2, 4>(map, g, sms, st);
    } else {
        if (stream_mt(g.m) == 8) launch_stream_cfg<W_BF16, 8, 1, 2>(map, g, sms, st);
        else launch_stream_cfg<W_BF16, 16, 2, 4>(map, g, sms, st);
    }
    return true;
}

} // namespace b200i
