// The int8i32.v1 product on SM pairs: gemm_int8_tma.cuh with two CTAs of a cluster working on one 256 x 256 tile.
//
// A pair issues tcgen05.mma.cta_group::2 (M 256, N 256, K 32): each CTA brings its own 128 rows of A and HALF of the 256 rows
// of B, and both tensor cores read both halves, so a 128 x 256 x 128 block of products costs an SM 32 KB of L2 reads where a
// lone CTA reads 48, and six stages fit where four did. Both kernels were bound by their store until it was cut to a
// conversion and two products per cell (i8_store_block): 4096^3 then takes 60 us = 2.30 POP/s (96 before), 62 with one CTA
// per tile; 8192^2 x 4096 2.69 POP/s against 2.55.
//
//   - warp 0, one lane, in both CTAs: the producer of that CTA's rows; its copies complete on the LEADER's mbarrier.
//   - warp 1, one lane, in the leader (rank 0): the MMA issuer for both; its commits arrive in both CTAs.
//   - warps 2 to 9 in both CTAs: the store of that CTA's 128 rows; they release the accumulator to the leader.
// Pairs walk the units of work blockIdx.x / 2, + number of pairs, ...: whole tiles first; when the last round would leave
// half of the pairs without a tile, its tiles are cut into 256 x 128 halves (N 128), so the round takes half the time.
// Every wait is bounded (status 9); the cluster barriers at entry and exit keep a CTA's shared memory alive while its
// partner can still signal into it, and every thread reaches them whatever ran out.
#pragma once
#include "gemm_int8_tma.cuh"

namespace b200i {

constexpr int P8_BM = 256, P8_BN = 256, P8_STAGES = 6;
constexpr int P8_BOX_B = 64; // rows of B per copy: one for a half unit, two for a whole one
constexpr int P8_A_BYTES = (P8_BM / 2) * T8_BK, P8_B_BYTES = (P8_BN / 2) * T8_BK, P8_STAGE_BYTES = P8_A_BYTES + P8_B_BYTES;
constexpr int P8_SMEM_BYTES = 1024 + P8_STAGES * P8_STAGE_BYTES + T8_TURN_BYTES + 256;
static_assert(P8_SMEM_BYTES <= 232448, "shared memory of one CTA");

__host__ __device__ constexpr unsigned p8_idesc(int tn) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(tn >> 3) << 17) | ((unsigned)(P8_BM >> 4) << 24);
}
__device__ __forceinline__ unsigned p8_leader_addr(const void *p) { // the same shared variable in the cluster's rank 0
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void p8_tma_load(void *dst, const CUtensorMap *map, unsigned leader_bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(reinterpret_cast<unsigned long long>(map)), "r"(leader_bar), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void p8_mma(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void p8_commit_both(unsigned long long *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((unsigned short)3)
                 : "memory");
}
__device__ __forceinline__ void p8_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(T8_THREADS, 1)
    gemm_int8_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, float *__restrict__ c,
                          const int *__restrict__ ea, const int *__restrict__ eb, int m, int n, int k, int tiles_n, int whole, int units) {
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *ring = smem + ((1024u - (smem_u32(smem) & 1023u)) & 1023u); // the same offset in both CTAs
    unsigned *turn_all = reinterpret_cast<unsigned *>(ring + P8_STAGES * P8_STAGE_BYTES);
    unsigned long long *full = reinterpret_cast<unsigned long long *>(ring + P8_STAGES * P8_STAGE_BYTES + T8_TURN_BYTES);
    unsigned long long *empty = full + P8_STAGES, *tfull = empty + P8_STAGES, *tempty = tfull + 2;
    unsigned *tmem_slot = reinterpret_cast<unsigned *>(tempty + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int kt_count = (k + T8_BK - 1) / T8_BK;

    if (tid == 0) {
        for (int s = 0; s < P8_STAGES; s++) {
            mbar_init(&full[s], 1);  // the leader's: its own expect, the bytes of both CTAs
            mbar_init(&empty[s], 1); // the issuer's commit, in both CTAs
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], 2 * T8_STORE_WARPS); // the leader's: the store warps of both CTAs
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T8_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    p8_cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *tmem_slot;

    // unit u: rows 256 * tm, columns col0 .. col0 + width
    auto unit = [&](int u, int &tm, int &col0, int &width) {
        const int tile = u < whole ? u : whole + ((u - whole) >> 1);
        tm = tile / tiles_n;
        col0 = (tile - tm * tiles_n) * P8_BN;
        width = P8_BN;
        if (u >= whole) {
            width = P8_BN / 2;
            col0 += ((u - whole) & 1) * width;
        }
    };

    if (warp == 0) {
        if (lane == 0) { // ---------------- producer of this CTA's rows ----------------
            int it = 0;
            bool alive = true;
            for (int u = pair; u < units && alive; u += pairs) {
                int tm, col0, width;
                unit(u, tm, col0, width);
                const int brow = col0 + rank * (width / 2);
                for (int kt = 0; kt < kt_count; kt++, it++) {
                    const int s = it % P8_STAGES;
                    const unsigned ph = (unsigned)(it / P8_STAGES) & 1u;
                    if (!mbar_wait(&empty[s], ph ^ 1u)) { // a fresh barrier counts as released
                        atomicExch(&g_decode_status, 9);
                        alive = false;
                        break;
                    }
                    unsigned char *st = ring + s * P8_STAGE_BYTES;
                    const unsigned bar = p8_leader_addr(&full[s]);
                    if (rank == 0) mbar_expect_tx(&full[s], 2u * (unsigned)(P8_A_BYTES + (width / 2) * T8_BK));
                    p8_tma_load(st, &map_a, bar, kt * T8_BK, tm * P8_BM + rank * (P8_BM / 2));
                    p8_tma_load(st + P8_A_BYTES, &map_b, bar, kt * T8_BK, brow);
                    if (width == P8_BN) p8_tma_load(st + P8_A_BYTES + P8_BOX_B * T8_BK, &map_b, bar, kt * T8_BK, brow + P8_BOX_B);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) { // ---------------- MMA issuer of the pair ----------------
            int it = 0, ti = 0;
            bool alive = true;
            for (int u = pair; u < units && alive; u += pairs, ti++) {
                int tm, col0, width;
                unit(u, tm, col0, width);
                const int acc = ti & 1;
                const unsigned aph = (unsigned)(ti >> 1) & 1u, idesc = p8_idesc(width);
                if (!mbar_wait(&tempty[acc], aph ^ 1u)) {
                    atomicExch(&g_decode_status, 9);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned d = tmem + (unsigned)(acc * P8_BN);
                for (int kt = 0; kt < kt_count; kt++, it++) {
                    const int s = it % P8_STAGES;
                    const unsigned ph = (unsigned)(it / P8_STAGES) & 1u;
                    if (!mbar_wait(&full[s], ph)) {
                        atomicExch(&g_decode_status, 9);
                        alive = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned a0 = smem_u32(ring + s * P8_STAGE_BYTES), b0 = a0 + P8_A_BYTES;
#pragma unroll
                    for (int j = 0; j < T8_BK / 32; j++)
                        p8_mma(d, t8_smem_desc(a0 + j * 32), t8_smem_desc(b0 + j * 32), idesc, (kt > 0 || j > 0) ? 1u : 0u);
                    p8_commit_both(&empty[s]); // the stage is free in both CTAs when these MMAs have read it
                }
                if (alive) p8_commit_both(&tfull[acc]);
            }
        }
    } else { // ---------------- store warps: this CTA's 128 rows ----------------
        const int q = warp & 3, half = (warp - 2) >> 2;
        unsigned *turn = turn_all + (warp - 2) * (32 * 33);
        int ti = 0;
        for (int u = pair; u < units; u += pairs, ti++) {
            int tm, col0, width;
            unit(u, tm, col0, width);
            const int acc = ti & 1;
            const unsigned aph = (unsigned)(ti >> 1) & 1u;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(&tfull[acc], aph))) {
                if (lane == 0) atomicExch(&g_decode_status, 9);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int rbase = tm * P8_BM + rank * (P8_BM / 2) + q * 32;
            const int ea_mine = rbase + lane < m ? ea[rbase + lane] : 0;
#pragma unroll 1
            for (int cb = half * (width / 2); cb < (half + 1) * (width / 2); cb += 32) {
                if (col0 + cb >= n) break; // uniform over the warp
                i8_store_block(tmem + ((unsigned)(q * 32) << 16) + (unsigned)(acc * P8_BN + cb), turn, c, eb, ea_mine, rbase, col0 + cb, m, n, lane);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(p8_leader_addr(&tempty[acc])) : "memory");
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    p8_cluster_sync(); // nothing signals into the partner's shared memory any more
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T8_TMEM_COLS) : "memory");
}

// Pairs that can be resident at once on the current device (0: none).
inline int p8_resident_pairs() {
    static std::atomic<int> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int v = known[dev].load();
    if (v == 0) {
        if (cudaFuncSetAttribute(gemm_int8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, P8_SMEM_BYTES) != cudaSuccess) { cudaGetLastError(); return 0; }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2);
        cfg.blockDim = dim3(T8_THREADS);
        cfg.dynamicSmemBytes = P8_SMEM_BYTES;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&v, gemm_int8_pair_kernel, &cfg) != cudaSuccess) { cudaGetLastError(); v = 0; }
        if (v <= 0) return 0;
        known[dev].store(v);
    }
    return v;
}

// Returns false when the device holds no pair or the tensor maps cannot be made (the caller then takes the one-CTA kernels).
inline bool launch_gemm_int8_pair(float *c, const signed char *qa, const int *ea, const signed char *qb, const int *eb, int m, int n, int k, cudaStream_t st) {
    const int pairs = p8_resident_pairs();
    if (pairs <= 0) return false;
    alignas(64) CUtensorMap map_a, map_b;
    if (!t8_make_map(&map_a, qa, m, k, P8_BM / 2) || !t8_make_map(&map_b, qb, n, k, P8_BOX_B)) return false;
    const int tiles_n = (n + P8_BN - 1) / P8_BN, tiles = ((m + P8_BM - 1) / P8_BM) * tiles_n;
    const int rest = tiles % pairs, whole = 2 * rest <= pairs ? tiles - rest : tiles;
    const int units = whole + 2 * (tiles - whole);
    gemm_int8_pair_kernel<<<2 * (units < pairs ? units : pairs), T8_THREADS, P8_SMEM_BYTES, st>>>(map_a, map_b, c, ea, eb, m, n, k, tiles_n, whole, units);
    return true;
}

} // namespace b200i
