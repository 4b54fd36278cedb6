// C[m, n] = A[m, k] . W[n, k]^T for 9 to 32 rows of activations on a large float32 weight: a band of all rows by 256
// columns per CTA.
//
// The float32 skinny kernel gives a thread all rows of two columns, so each k-step costs it eight broadcast reads of the
// activations for 32 packed multiply-adds, and its weight window goes through registers with a load in flight at a time.
// Here a thread owns TM x 8 cells, as in the large products (four 128-bit reads and eight doubled words for 32 packed fmas
// at 32 rows), and the weight arrives by cp.async:
//
//   ring    three stages of 64 bytes (16 k-steps) of each of the tile's 256 weight rows (four lanes per row, 16-byte pieces
//           permuted by the row against bank conflicts);
//   turn    thread t takes the 16 k-steps of rows t and t + 128 and stores them k-major as 64-bit pairs, columns t and
//           t + 128 side by side: ready fma.rn.f32x2 operands; this runs between the multiply-adds of the window before;
//   barrier one per window; it publishes the window and its admission verdict.
// Leaves of a CTA's group are folded by a per-thread counter stack, groups by fold_groups as in the other plans.
// Measured (graph replay, fold included) against the skinny kernel: [16384, 2048] 88 against 108 us at 32 rows, 62 against
// 82 at 16 (45 in the streaming kernel, which takes such calls up to sixteen rows); [50304, 2048] 242 against 297; [11008, 4096] 120 against 130; [2304, 768] 23 against 18, hence the rule's size.
// The same kernel with low-bit weights widened on the way lost to the register kernel (int8 [11008, 4096] 111 against 95).
#pragma once
#include "gemm_skinny.cuh"

namespace b200i {

constexpr int BD_THREADS = 128, BD_BN = 256, BD_SEG = 64, BD_STAGES = 3;
constexpr int BD_CHUNK = 2 * K_LEAF_MIN;                // k-steps of activations staged at a time
constexpr int BD_STAGE_BYTES = BD_BN * BD_SEG;
constexpr int bd_smem_bytes(int bm) { return BD_STAGES * BD_STAGE_BYTES + 2 * KS * BD_BN * 4 + BD_CHUNK * bm * 4 + (BD_CHUNK / KS) * 4; }

template <int BM>
__global__ void __launch_bounds__(BD_THREADS, 2) gemm_band_kernel(const GemmArgs g) {
    constexpr int TM = BM / 4, TN = 8, PAIRS = TM * TN / 2, CELLS = TM * TN;
    extern __shared__ __align__(128) unsigned char bd_smem[];
    unsigned char *ring = bd_smem;
    float (*Bs)[KS][BD_BN] = reinterpret_cast<float (*)[KS][BD_BN]>(bd_smem + BD_STAGES * BD_STAGE_BYTES);
    float *As = reinterpret_cast<float *>(bd_smem + BD_STAGES * BD_STAGE_BYTES + 2 * KS * BD_BN * 4); // [BD_CHUNK][BM]
    unsigned *akey = reinterpret_cast<unsigned *>(As + BD_CHUNK * BM);                                 // per window of the chunk

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int bn0 = blockIdx.x * BD_BN;
    const int t_first = blockIdx.y * g.group_leaves, t_end = min(t_first + g.group_leaves, g.leaves);
    const int kbase = t_first * g.leaf, klen = min(g.k, t_end * g.leaf) - kbase, windows = klen / KS; // k is a multiple of 16
    const int wpl = g.leaf / KS;
    const float *wb = static_cast<const float *>(g.b);

    auto issue = [&](int s) { // window s of the CTA's range; one commit always
        if (s < windows) {
            unsigned char *st = ring + (size_t)(s % BD_STAGES) * BD_STAGE_BYTES;
#pragma unroll
            for (int v = 0; v < BD_BN * 4 / BD_THREADS; v++) {
                const int r = v * (BD_THREADS / 4) + (tid >> 2), c = tid & 3;
                const bool in = bn0 + r < g.n;
                const float *src = in ? wb + (size_t)(bn0 + r) * g.k + kbase + s * KS + c * 4 : wb;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(st + r * BD_SEG + ((c ^ ((r >> 1) & 3)) * 16))), "l"(src), "r"(in ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < BD_STAGES; s++) issue(s);

    auto stage_chunk = [&](int w0) { // activations of windows w0 .. w0 + 15, k-major, rows past m zero
        if (tid < BD_CHUNK / KS) akey[tid] = 0xFFFFFFFFu;
        __syncthreads();
#pragma unroll
        for (int kq = 0; kq < BD_CHUNK / 32; kq += 2) { // a warp covers 32 k-steps of a quarter of the rows, twice at a time
            float x[2][BM / 4];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int kk = w0 * KS + (kq + u) * 32 + lane;
#pragma unroll
                for (int r = 0; r < BM / 4; r++) {
                    const int row = warp * (BM / 4) + r;
                    x[u][r] = (kk < klen && row < g.m) ? __ldg(g.a + (size_t)row * g.k + kbase + kk) : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                unsigned key = 0xFFFFFFFFu;
#pragma unroll
                for (int r = 0; r < BM / 4; r += 4) {
                    const float4 v = make_float4(x[u][r], x[u][r + 1], x[u][r + 2], x[u][r + 3]);
                    key = key4(v, key);
                    *reinterpret_cast<float4 *>(As + (size_t)((kq + u) * 32 + lane) * BM + warp * (BM / 4) + r) = v;
                }
                atomicMin(&akey[(kq + u) * 2 + (lane >> 4)], key);
            }
        }
    };

    unsigned key = 0xFFFFFFFFu; // of the window this thread turned last
    auto turn = [&](int w) {    // window w of the CTA's range, into Bs[w & 1]
        const unsigned char *st = ring + (size_t)(w % BD_STAGES) * BD_STAGE_BYTES;
        float (*out)[BD_BN] = Bs[w & 1];
        const int r0 = tid, r1 = tid + 128, sw = (r0 >> 1) & 3; // (r1 >> 1) & 3 is the same
        key = 0xFFFFFFFFu;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float4 a = *reinterpret_cast<const float4 *>(st + r0 * BD_SEG + ((c ^ sw) * 16)), b = *reinterpret_cast<const float4 *>(st + r1 * BD_SEG + ((c ^ sw) * 16));
            key = key4(a, key4(b, key));
            *reinterpret_cast<float2 *>(&out[4 * c + 0][2 * tid]) = make_float2(a.x, b.x);
            *reinterpret_cast<float2 *>(&out[4 * c + 1][2 * tid]) = make_float2(a.y, b.y);
            *reinterpret_cast<float2 *>(&out[4 * c + 2][2 * tid]) = make_float2(a.z, b.z);
            *reinterpret_cast<float2 *>(&out[4 * c + 3][2 * tid]) = make_float2(a.w, b.w);
        }
    };

    // rows ty * TM .. + TM - 1; column places r * 128 + tx * 4 .. + 3
    const int ty = (warp & 1) * 2 + (lane >> 4), tx = (warp >> 1) * 16 + (lane & 15);
    unsigned long long acc[PAIRS]; // [row][pair of places]
#pragma unroll
    for (int i = 0; i < PAIRS; i++) acc[i] = 0ull;
    float stack[FOLD_LEVELS][CELLS];
    auto step = [&](const float *arow, const float *brow, bool flush) {
        float av[TM];
        unsigned long long b2[4];
#pragma unroll
        for (int r = 0; r < TM; r += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(arow + r);
            av[r] = v.x; av[r + 1] = v.y; av[r + 2] = v.z; av[r + 3] = v.w;
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(brow + r * 128);
            b2[2 * r] = v.x;
            b2[2 * r + 1] = v.y;
        }
        if (flush) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float lo, hi;
                unpack2(b2[j], lo, hi);
                b2[j] = pack2(ftz_bits(lo), ftz_bits(hi));
            }
        }
#pragma unroll
        for (int i = 0; i < TM; i++) {
            const float a = flush ? ftz_bits(av[i]) : av[i];
            const unsigned long long a2 = pack2(a, a);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned long long d = fma2_bare(a2, b2[j], acc[i * 4 + j]);
                acc[i * 4 + j] = flush ? ftz2_hw(d) : d;
            }
        }
    };
    auto cells_of = [&](float (&v)[CELLS]) {
#pragma unroll
        for (int i = 0; i < PAIRS; i++) {
            unpack2(ftz2_hw(acc[i]), v[2 * i], v[2 * i + 1]);
            acc[i] = 0ull;
        }
    };

    stage_chunk(0);
    asm volatile("cp.async.wait_group 1;" ::: "memory"); // windows 0 and 1
    __syncthreads();
    turn(0);
    bool admitted = __syncthreads_and(key >= ADMIT_MIN) && akey[0] >= ADMIT_MIN;
    bool clean = true;
    for (int w = 0; w < windows; w++) {
        issue(w + BD_STAGES); // window w was turned before the last barrier: its slot is free
        if (w + 1 < windows) turn(w + 1);
        const float *arow = As + (size_t)((w * KS) % BD_CHUNK) * BM + ty * TM, *brow = &Bs[w & 1][0][tx * 4];
        clean = clean && admitted;
        if (clean) {
#pragma unroll
            for (int kk = 0; kk < KS; kk++) step(arow + kk * BM, brow + kk * BD_BN, false);
        } else {
#pragma unroll 1
            for (int kk = 0; kk < KS; kk++) step(arow + kk * BM, brow + kk * BD_BN, true);
        }
        if ((w + 1) % wpl == 0 && w + 1 < windows) { // a leaf is finished and another follows
            const int leaf = w / wpl;
            float v[CELLS];
            cells_of(v);
            int lvl = 0;
            for (int bits = leaf; bits & 1; bits >>= 1, lvl++) {
#pragma unroll
                for (int c = 0; c < CELLS; c++) v[c] = add_flushed(stack[lvl][c], v[c]);
            }
#pragma unroll
            for (int c = 0; c < CELLS; c++) stack[lvl][c] = v[c];
            clean = true;
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory"); // window w + 2
        if (w + 1 < windows && ((w + 1) * KS) % BD_CHUNK == 0) {
            __syncthreads(); // every thread is through with the chunk
            stage_chunk(w + 1);
        }
        admitted = __syncthreads_and(key >= ADMIT_MIN);
        admitted = admitted && akey[(w + 1) % (BD_CHUNK / KS)] >= ADMIT_MIN;
    }

    float v[CELLS];
    cells_of(v);
    const int last = t_end - t_first - 1;
#pragma unroll 1
    for (int lvl = 0; (last >> lvl) != 0; lvl++)
        if ((last >> lvl) & 1) {
#pragma unroll
            for (int c = 0; c < CELLS; c++) v[c] = add_flushed(stack[lvl][c], v[c]);
        }
    // places r*128 + tx*4 + {0, 1, 2, 3} hold columns c, c + 128, c + 1, c + 129 with c = r*64 + tx*2
    float *out = g.groups > 1 ? g.ws + (size_t)blockIdx.y * (size_t)g.m * (size_t)g.n : g.c;
    const bool pairs = g.groups == 1 && epilogue_pairs(g.epi), single = g.groups == 1 && !pairs && epilogue_on(g.epi);
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int row = ty * TM + i;
        if (row >= g.m) break;
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int col = bn0 + r * 64 + tx * 2 + h * 128;
                const float x = nan_canon(v[i * 8 + r * 4 + h]), y = nan_canon(v[i * 8 + r * 4 + 2 + h]);
                if (pairs) { // n is a multiple of 4
                    if (col < g.n) g.c[(size_t)row * (g.n / 2) + col / 2] = epilogue_pair_apply(x, y, g.epi.bias, g.epi.act, col / 2);
                    continue;
                }
                float *dst = out + (size_t)row * g.n + col;
                if (g.vec_c && col + 1 < g.n && !single) {
                    *reinterpret_cast<float2 *>(dst) = make_float2(x, y);
                } else {
                    if (col < g.n) dst[0] = single ? epilogue_apply(x, g.epi.bias, g.epi.act, col) : x;
                    if (col + 1 < g.n) dst[1] = single ? epilogue_apply(y, g.epi.bias, g.epi.act, col + 1) : y;
                }
            }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int BM>
inline void launch_band_rows(const GemmArgs &g, cudaStream_t st) {
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaFuncSetAttribute(gemm_band_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, bd_smem_bytes(BM));
        configured[dev] = true;
    }
    gemm_band_kernel<BM><<<dim3((unsigned)((g.n + BD_BN - 1) / BD_BN), (unsigned)g.groups), BD_THREADS, bd_smem_bytes(BM), st>>>(g);
}
inline void launch_band(const GemmArgs &g, cudaStream_t st) {
    if (g.m <= 16) launch_band_rows<16>(g, st);
    else launch_band_rows<32>(g, st);
}

} // namespace b200i
