// C[m, n] = A[m, k] . W[n, k]^T for a small decode batch (up to 16 rows), any weight storage: the whole contraction of a
// column inside one CTA.
//
// The skinny plans cut k into leaf groups over many CTAs, stage every 16-step window behind a CTA barrier and fold the
// groups in a second launch. With eight rows there is too little arithmetic to hide that: 14 us + 4 us of fold for a
// [2304, 768] float32 product whose bytes take 1 us. Here:
//
//   - a CTA owns a contiguous range of weight rows (output columns), about n * groups / SMs of them (groups of leaves, below;
//     one up to sixteen leaves), so nearly every SM has one CTA and every CTA the same bytes; it walks them in strips of
//     CB = LC * CPL columns;
//   - the activations of the CTA's leaves are staged ONCE, [k][MT] so that pairs of rows are ready fma.rn.f32x2 operands;
//   - a warp takes a unit (strip, aligned run of leaves): its own ring of 128-byte row segments by cp.async (16-byte
//     pieces permuted by the row, so that 32 lanes read 32 rows without a bank conflict), no barrier wider than the warp.
//     A lane is a weight row (CPL of them) and MT * LC / 32 activation rows: one weight read serves 4 to 16 k-steps, one
//     broadcast read of the activations serves all CPL columns;
//   - unit nodes meet in shared memory and are folded there (the same adjacent-pair tree, the runs being aligned
//     subtrees), so no node crosses L2 and there is no second launch up to sixteen leaves; beyond that the leaves are cut
//     into groups (the activations of more would leave too short a ring) and fold_groups finishes as for the other plans.
// Measured at eight rows, float32 (graph replay): [768, 768] 13.1 -> 5.6 us, [2304, 768] 14.1 -> 6.5, [768, 3072] 13.9 -> 8.6,
// [50304, 768] 66 -> 54 (41 in the streaming kernel, which takes most large weights at 5 rows and more). Bound: latency below ten
// million weights (a leaf is 128 dependent steps), above by the warps' own instructions (about six per step and column of 32 lanes)
// and by HBM.
//
// Admission is per leaf: the activations' keys are taken while they are staged, the weights' while they are used; a lane
// whose leaf fails runs the defining flushed chain again from global memory.
#pragma once
#include <algorithm>

#include "gemm_skinny.cuh"

namespace b200i {

constexpr int RW_MAX_WARPS = 16;
constexpr int RW_LEAF = 128;
constexpr int RW_SEG = 128;                 // bytes of a weight row per ring stage
constexpr int RW_SMEM_LIMIT = 225 * 1024;
constexpr int RW_ACT_LIMIT = 128 * 1024;    // activations of one CTA's leaves
constexpr int RW_MAX_ROWS = 16;

struct RowsPlan {
    int cpc;         // columns per CTA
    int warps, stages;
    int run;         // leaves per unit: 1, 2 or 4
    int together;    // strips folded at a time
    int parts_off, factor_off, key_off, ring_off; // bytes into shared memory
};

template <int WK>
struct RowsKind {
    static constexpr int ES = WK == W_F32 ? 4 : (WK == W_BF16 ? 2 : 1);
    static constexpr int KC = RW_SEG / ES; // k-steps per stage: 32, 64, 128
    static constexpr int EPQ = 16 / ES;    // k-steps per 16-byte piece
};

template <int WK, int MT, int LC, int CPL>
__global__ void __launch_bounds__(32 * RW_MAX_WARPS, 1) gemm_rows_kernel(const GemmArgs g, const RowsPlan p) {
    using K = RowsKind<WK>;
    constexpr int CB = LC * CPL, RG = 32 / LC, RL = MT / RG, PAIRS = RL / 2, CELLS = RL * CPL;
    constexpr int STAGE = CB * RW_SEG;
    extern __shared__ __align__(128) unsigned char rw_smem[];
    float *act = reinterpret_cast<float *>(rw_smem);
    float *parts = reinterpret_cast<float *>(rw_smem + p.parts_off);
    float *factors = reinterpret_cast<float *>(rw_smem + p.factor_off);
    unsigned *lkey = reinterpret_cast<unsigned *>(rw_smem + p.key_off);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nw = p.warps, stages = p.stages;
    unsigned char *ring = rw_smem + p.ring_off + (size_t)warp * stages * STAGE;

    const int c_lo = blockIdx.x * p.cpc, c_hi = min(c_lo + p.cpc, g.n);
    const int t_lo = blockIdx.y * g.group_leaves, t_hi = min(t_lo + g.group_leaves, g.leaves);
    const int leaves = t_hi - t_lo, kbase = t_lo * RW_LEAF, klen = min(g.k, t_hi * RW_LEAF) - kbase;
    const int runs = (leaves + p.run - 1) / p.run;                // units (and nodes) per strip
    const int strips = (c_hi - c_lo + CB - 1) / CB;
    const int supers = (strips + p.together - 1) / p.together;
    const unsigned char *wb = static_cast<const unsigned char *>(g.b);
    const size_t row_bytes = (size_t)g.k * K::ES;

    // ---- the warp's walk: (super, strip, run of leaves, leaf of the run, chunk of the leaf); no division on the way ----
    struct Walk {
        int s, strip, run, i, ch; // strip and run: the unit, strip * runs + run of the super
    };
    const int strip_step = nw / runs, run_step = nw % runs, strip_first = warp / runs, run_first = warp % runs;
    auto here = [&](int s) { return min(p.together, strips - s * p.together); };
    auto settle = [&](Walk &w) {
        while (w.s < supers && w.strip >= here(w.s)) { w.s++; w.strip = strip_first; w.run = run_first; }
    };
    auto leaf_of = [&](const Walk &w) { return w.run * p.run + w.i; };
    auto leaf_len = [&](int l) { return min(RW_LEAF, klen - l * RW_LEAF); };
    auto advance = [&](Walk &w) {
        const int l = leaf_of(w);
        if (++w.ch * K::KC < leaf_len(l)) return;
        w.ch = 0;
        if (++w.i < p.run && l + 1 < leaves) return;
        w.i = 0;
        w.strip += strip_step;
        w.run += run_step;
        if (w.run >= runs) { w.run -= runs; w.strip++; }
        settle(w);
    };
    auto issue = [&](const Walk &w, int slot) {
        if (w.s < supers) {
            const int col0 = c_lo + (w.s * p.together + w.strip) * CB, l = leaf_of(w);
            const int k0 = l * RW_LEAF + w.ch * K::KC, pieces = min(K::KC, klen - k0) / K::EPQ; // leaf_len is a multiple of 16
            const int r0 = lane >> 3, q = lane & 7, left = c_hi - col0 - r0;
            unsigned st = smem_u32(ring + (size_t)slot * STAGE + r0 * RW_SEG);
            const unsigned char *src = wb + (size_t)(col0 + r0) * row_bytes + (size_t)(kbase + k0) * K::ES + q * 16;
            const size_t four_rows = 4 * row_bytes;
#pragma unroll
            for (int v = 0; v < CB / 4; v++) { // rows r0 + 4v: the piece's place alternates between two values
                const bool in = v * 4 < left && q < pieces;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(st + v * 4 * RW_SEG + ((q ^ ((r0 + v * 4) & 7)) * 16)), "l"(in ? src : wb),
                             "r"(in ? 16 : 0)
                             : "memory");
                src += four_rows;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    Walk ahead{0, strip_first, run_first, 0, 0}, now{0, strip_first, run_first, 0, 0};
    settle(ahead);
    settle(now);
    int in_slot = 0, out_slot = 0;
    for (int i = 0; i < stages - 1; i++) {
        issue(ahead, in_slot);
        if (++in_slot == stages) in_slot = 0;
        if (ahead.s < supers) advance(ahead);
    }

    // ---- activations: [k][MT], rows past m zero; one key per leaf ----
    for (int i = tid; i < leaves; i += blockDim.x) lkey[i] = 0xFFFFFFFFu;
    if (WK == W_INT8_EXP || WK == W_INT8_SCALE)
        for (int i = tid; i < c_hi - c_lo; i += blockDim.x)
            factors[i] = WK == W_INT8_EXP ? pow2_f32(__ldg(static_cast<const int *>(g.bscale) + c_lo + i)) : __ldg(static_cast<const float *>(g.bscale) + c_lo + i);
    __syncthreads();
    constexpr int AU = MT <= 8 ? 4 : 2; // groups of 32 k-steps whose loads are in flight together
    for (int k0 = warp * (32 * AU); k0 < klen; k0 += nw * (32 * AU)) {
        float x[AU][MT];
#pragma unroll
        for (int u = 0; u < AU; u++)
#pragma unroll
            for (int r = 0; r < MT; r++) {
                const int kk = k0 + u * 32 + lane;
                x[u][r] = (kk < klen && r < g.m) ? __ldg(g.a + (size_t)r * g.k + kbase + kk) : 0.f;
            }
        unsigned key = 0xFFFFFFFFu; // 32 * AU steps lie inside one leaf
#pragma unroll
        for (int u = 0; u < AU; u++) {
            const int kk = k0 + u * 32 + lane;
#pragma unroll
            for (int r = 0; r < MT; r++) key = min(key, admit_key(x[u][r]));
            if (kk < klen) {
#pragma unroll
                for (int r = 0; r < MT; r += 4) *reinterpret_cast<float4 *>(act + (size_t)kk * MT + r) = make_float4(x[u][r], x[u][r + 1], x[u][r + 2], x[u][r + 3]);
            }
        }
        key = __reduce_min_sync(0xFFFFFFFFu, key);
        if (lane == 0) atomicMin(&lkey[k0 / RW_LEAF], key);
    }
    __syncthreads();

    const int lc = lane % LC, rg = lane / LC;
    unsigned long long acc[PAIRS][CPL];
    float stack[2][CELLS];
    unsigned key = 0xFFFFFFFFu;
    float f[CPL], nbias[CPL];

    for (int s = 0; s < supers; s++) {
        while (now.s == s) {
            const int col0 = c_lo + (s * p.together + now.strip) * CB, l = leaf_of(now);
            const int k0 = l * RW_LEAF + now.ch * K::KC, len = min(K::KC, leaf_len(l) - now.ch * K::KC);
            if (now.ch == 0) { // a new leaf
                key = lkey[l];
#pragma unroll
                for (int i = 0; i < PAIRS; i++)
#pragma unroll
                    for (int j = 0; j < CPL; j++) acc[i][j] = 0ull;
                if (WK == W_INT8_EXP || WK == W_INT8_SCALE) {
#pragma unroll
                    for (int j = 0; j < CPL; j++) {
                        const int c = col0 + lc + j * LC;
                        f[j] = c < c_hi ? factors[c - c_lo] : 1.f;
                        const unsigned fexp = (__float_as_uint(f[j]) >> 23) & 0xFFu;
                        if (fexp < ADMIT_EXP || fexp < 27u || fexp > 227u) key = 0u; // the short spellings below would not be exact, or not admitted
                        nbias[j] = -8388736.0f * f[j];
                    }
                }
            }
            if (stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory"); // three stages: the newest group may still be in flight
            __syncwarp(); // the stage is visible to the warp, and every lane has left the one before it: refill that
            issue(ahead, in_slot);
            if (++in_slot == stages) in_slot = 0;
            if (ahead.s < supers) advance(ahead);
            const unsigned char *st = ring + (size_t)out_slot * STAGE;
            const float *ak = act + (size_t)k0 * MT + rg * RL;
            auto quad = [&](int q) { // the k-steps of one 16-byte piece
                uint4 wv[CPL];
#pragma unroll
                for (int j = 0; j < CPL; j++) wv[j] = *reinterpret_cast<const uint4 *>(st + (lc + j * LC) * RW_SEG + ((q ^ (lc & 7)) * 16));
                float v[CPL][K::EPQ];
#pragma unroll
                for (int j = 0; j < CPL; j++) {
                    const unsigned word[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (WK == W_F32) {
                            v[j][e] = __uint_as_float(word[e]);
                            key = min(key, admit_key(v[j][e]));
                        } else if (WK == W_BF16) {
                            v[j][(2 * e) % K::EPQ] = __uint_as_float(word[e] << 16);
                            v[j][(2 * e + 1) % K::EPQ] = __uint_as_float(word[e] & 0xFFFF0000u);
                            key = min(key, min(admit_key(v[j][(2 * e) % K::EPQ]), admit_key(v[j][(2 * e + 1) % K::EPQ])));
                        } else {
                            const unsigned x = word[e] ^ 0x80808080u;
                            const float b0 = biased_code<0>(x), b1 = biased_code<1>(x), b2 = biased_code<2>(x), b3 = biased_code<3>(x);
                            float *o = &v[j][(4 * e) % K::EPQ];
                            if (WK == W_INT8_EXP) {
                                const unsigned long long ff = pack2(f[j], f[j]), nb = pack2(nbias[j], nbias[j]);
                                unpack2(fma2_bare(pack2(b0, b1), ff, nb), o[0], o[1]);
                                unpack2(fma2_bare(pack2(b2, b3), ff, nb), o[2 % K::EPQ], o[3 % K::EPQ]);
                            } else {
                                o[0] = __fmul_rn(__fsub_rn(b0, 8388736.0f), f[j]);
                                o[1] = __fmul_rn(__fsub_rn(b1, 8388736.0f), f[j]);
                                o[2 % K::EPQ] = __fmul_rn(__fsub_rn(b2, 8388736.0f), f[j]);
                                o[3 % K::EPQ] = __fmul_rn(__fsub_rn(b3, 8388736.0f), f[j]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int e = 0; e < K::EPQ; e++) {
                    unsigned long long a2[PAIRS];
                    const float *row = ak + (size_t)(q * K::EPQ + e) * MT;
                    if (PAIRS == 1) {
                        a2[0] = *reinterpret_cast<const unsigned long long *>(row);
                    } else {
#pragma unroll
                        for (int i = 0; i < PAIRS; i += 2) {
                            const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(row + 2 * i);
                            a2[i] = t.x;
                            a2[(i + 1) % PAIRS] = t.y;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < CPL; j++) {
                        const unsigned long long w2 = pack2(v[j][e], v[j][e]);
#pragma unroll
                        for (int i = 0; i < PAIRS; i++) acc[i][j] = fma2_bare(a2[i], w2, acc[i][j]);
                    }
                }
            };
            if (len == K::KC) {
#pragma unroll 4
                for (int q = 0; q < 8; q++) quad(q);
            } else {
#pragma unroll 1
                for (int q = 0; q < len / K::EPQ; q++) quad(q);
            }
            if (++out_slot == stages) out_slot = 0;

            Walk next = now;
            advance(next);
            if (next.ch == 0) { // the leaf is finished
                float v[CELLS];
#pragma unroll
                for (int i = 0; i < PAIRS; i++)
#pragma unroll
                    for (int j = 0; j < CPL; j++) unpack2(ftz2_hw(acc[i][j]), v[2 * i * CPL + j], v[(2 * i + 1) * CPL + j]);
                if (key < ADMIT_MIN) { // this lane's columns again, by the defining step, from global memory
#pragma unroll 1
                    for (int j = 0; j < CPL; j++) {
                        const int c = col0 + lc + j * LC;
                        if (c >= c_hi) continue;
                        const float fj = (WK == W_INT8_EXP || WK == W_INT8_SCALE) ? factors[c - c_lo] : 1.f;
                        float slow[RL];
#pragma unroll
                        for (int r = 0; r < RL; r++) slow[r] = 0.f;
                        const int lk = l * RW_LEAF, ll = leaf_len(l);
#pragma unroll 1
                        for (int kk = 0; kk < ll; kk++) {
                            const size_t off = (size_t)c * g.k + kbase + lk + kk;
                            float w;
                            if (WK == W_F32) w = ftz_bits(__ldg(static_cast<const float *>(g.b) + off));
                            else if (WK == W_BF16) w = ftz_bits(bf16_bits_to_f32(__ldg(static_cast<const unsigned short *>(g.b) + off)));
                            else w = dequant_int8_pow2((int)__ldg(static_cast<const signed char *>(g.b) + off), fj);
#pragma unroll
                            for (int r = 0; r < RL; r++) slow[r] = step_flush(ftz_bits(act[(size_t)(lk + kk) * MT + rg * RL + r]), w, slow[r]);
                        }
#pragma unroll
                        for (int r = 0; r < RL; r++)
#pragma unroll
                            for (int jj = 0; jj < CPL; jj++)
                                if (jj == j) v[r * CPL + jj] = ftz_hw(slow[r]);
                    }
                }
                const int last = min(p.run, leaves - now.run * p.run) - 1; // the run's last leaf
                fold_push<CELLS, 2>(stack, v, now.i, last);
                if (now.i == last) {
                    float *node = parts + (size_t)((now.strip * runs + now.run) * MT + rg * RL) * CB + lc;
#pragma unroll
                    for (int r = 0; r < RL; r++)
#pragma unroll
                        for (int j = 0; j < CPL; j++) node[r * CB + j * LC] = v[r * CPL + j];
                }
            }
            now = next;
        }
        __syncthreads(); // the nodes of these strips are whole
        const int pairs_total = here(s) * MT * (CB / 2);
        for (int x = tid; x < pairs_total; x += blockDim.x) {
            const int strip = x / (MT * (CB / 2)), r = (x / (CB / 2)) % MT, c = (x % (CB / 2)) * 2;
            const int col = c_lo + (s * p.together + strip) * CB + c;
            if (r >= g.m || col >= c_hi) continue;
            const float *node = parts + (size_t)(strip * runs * MT + r) * CB + c;
            float st2[5][2], v[2];
            for (int n0 = 0; n0 < runs; n0 += 8) {
                float2 y[8];
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if (n0 + e < runs) y[e] = *reinterpret_cast<const float2 *>(node + (size_t)(n0 + e) * MT * CB);
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if (n0 + e < runs) {
                        v[0] = y[e].x;
                        v[1] = y[e].y;
                        fold_push<2, 5>(st2, v, n0 + e, runs - 1);
                    }
            }
            v[0] = nan_canon(ftz_hw(v[0]));
            v[1] = nan_canon(ftz_hw(v[1]));
            if (g.groups > 1) {
                float *dst = g.ws + ((size_t)blockIdx.y * g.m + r) * g.n + col;
                dst[0] = v[0];
                if (col + 1 < c_hi) dst[1] = v[1];
            } else if (epilogue_pairs(g.epi)) { // columns per CTA are even, and so is n: both columns of a pair are here
                g.c[(size_t)r * (g.n / 2) + col / 2] = epilogue_pair_apply(v[0], v[1], g.epi.bias, g.epi.act, col / 2);
            } else {
                float *dst = g.c + (size_t)r * g.n + col;
                const bool on = epilogue_on(g.epi);
                dst[0] = on ? epilogue_apply(v[0], g.epi.bias, g.epi.act, col) : v[0];
                if (col + 1 < c_hi) dst[1] = on ? epilogue_apply(v[1], g.epi.bias, g.epi.act, col + 1) : v[1];
            }
        }
        if (s + 1 < supers) __syncthreads(); // the nodes may be overwritten
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

inline bool rows_plan_fits(long long m, long long n, long long k, int op) { return m <= RW_MAX_ROWS && skinny_plan_fits(m, n, k, op); }
inline int rows_mt(long long m) { return m <= 8 ? 8 : 16; }
// leaves per CTA whose activations fit: a power of two (32 at eight rows, 16 at sixteen)
inline int rows_group_leaves(long long m) { return RW_ACT_LIMIT / (rows_mt(m) * RW_LEAF * 4); }

// A launch of the rows plan: the kernel's strip shape, its plan, and its dynamic shared memory.
struct RowsLaunch {
    int lc, cpl, smem, groups;
    int rounds;  // leaves that a CTA's busiest warp walks one after the other
    int act_bytes;
    RowsPlan p;
};
// Lays out a CTA's shared memory; false where it does not hold two stages of a ring for four warps, which is what the kernel's
// waits need (one stage would be read while its copy is in flight). The factors of int8 weights are what can fill it: four
// bytes for each of a CTA's n * groups / SMs columns, so about n * k above four billion codes. The rule and the launch
// both ask here.
inline bool rows_layout(long long m, long long n, long long k, int wkind, int group_leaves, int sms, RowsLaunch &r) {
    const int leaves = (int)leaf_count(k), gl = group_leaves < leaves ? group_leaves : leaves, mt = rows_mt(m);
    if (gl > rows_group_leaves(m)) return false;
    const int groups = (leaves + gl - 1) / gl, ctas = sms / groups > 0 ? sms / groups : 1;
    long long cpc = (n + ctas - 1) / ctas;
    cpc = (cpc + 1) / 2 * 2;
    r.lc = cpc <= 8 ? 8 : (cpc <= 16 ? 16 : 32);
    r.cpl = mt > 8 || cpc <= 48 ? 1 : 2;
    if (cpc <= 16) cpc = r.lc;
    const int cb = r.lc * r.cpl, stage = cb * RW_SEG;
    const long long strips = (cpc + cb - 1) / cb, factors = wkind == W_INT8_EXP || wkind == W_INT8_SCALE ? (cpc * 4 + 127) / 128 * 128 : 0;
    if (factors > RW_SMEM_LIMIT) return false;
    const long long act = std::min((long long)gl * RW_LEAF, k) * mt * 4;
    RowsPlan &p = r.p;
    p.cpc = (int)cpc;
    // sixteen warps with single leaves, then pairs and fours; eight and four warps when the ring would be shorter than two stages
    for (int most = RW_MAX_WARPS; most >= 4; most /= 2) {
        p.run = 1;
        while (p.run < 4 && (gl + p.run - 1) / p.run > most) p.run *= 2;
        const int runs = (gl + p.run - 1) / p.run;
        p.together = 1;
        while (p.together * 2 <= strips && p.together * runs < 2 * most && (p.together * runs) % most != 0) p.together *= 2;
        const int total = p.together * runs;
        p.warps = total < most ? total : most;
        p.parts_off = (int)((act + 127) / 128 * 128);
        p.factor_off = p.parts_off + total * mt * cb * 4;
        p.key_off = p.factor_off + (int)factors;
        p.ring_off = (p.key_off + gl * 4 + 127) / 128 * 128;
        p.stages = p.ring_off < RW_SMEM_LIMIT ? (RW_SMEM_LIMIT - p.ring_off) / (p.warps * stage) : 0;
        if (p.stages < 2) continue;
        if (p.stages > 3) p.stages = 3;
        r.smem = p.ring_off + p.warps * p.stages * stage;
        r.groups = groups;
        r.act_bytes = (int)act;
        const int rest = (int)(strips % p.together);
        r.rounds = (int)std::min<long long>((strips / p.together * ((total + p.warps - 1) / p.warps) + (rest * runs + p.warps - 1) / p.warps) * p.run, 1 << 30);
        return true;
    }
    return false;
}

template <int WK, int MT, int LC, int CPL>
inline void launch_rows_cfg(const GemmArgs &g, const RowsLaunch &r, cudaStream_t st) {
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaFuncSetAttribute(gemm_rows_kernel<WK, MT, LC, CPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, RW_SMEM_LIMIT);
        configured[dev] = true;
    }
    const dim3 grid((unsigned)((g.n + r.p.cpc - 1) / r.p.cpc), (unsigned)g.groups);
    gemm_rows_kernel<WK, MT, LC, CPL><<<grid, 32 * r.p.warps, r.smem, st>>>(g, r.p);
}

template <int WK, int MT>
inline void launch_rows_mt(const GemmArgs &g, const RowsLaunch &r, cudaStream_t st) {
    if (r.lc == 8) launch_rows_cfg<WK, MT, 8, 1>(g, r, st);
    else if (r.lc == 16) launch_rows_cfg<WK, MT, 16, 1>(g, r, st);
    else if (r.cpl == 1) launch_rows_cfg<WK, MT, 32, 1>(g, r, st);
    else launch_rows_cfg<WK, 8, 32, 2>(g, r, st);
}
template <int WK>
inline void launch_rows_wk(const GemmArgs &g, const RowsLaunch &r, cudaStream_t st) {
    if (g.m <= 8) launch_rows_mt<WK, 8>(g, r, st);
    else launch_rows_mt<WK, 16>(g, r, st);
}
inline void launch_rows(const GemmArgs &g, const RowsLaunch &r, cudaStream_t st) {
    switch (g.wkind) {
    case W_F32: launch_rows_wk<W_F32>(g, r, st); break;
    case W_BF16: launch_rows_wk<W_BF16>(g, r, st); break;
    case W_INT8_EXP: launch_rows_wk<W_INT8_EXP>(g, r, st); break;
    default: launch_rows_wk<W_INT8_SCALE>(g, r, st); break;
    }
}

} // namespace b200i
