// The C ABI of libb200i.so: argument checks, plan selection, launches.
// Declarations and the reference interfaces they replace are in include/b200i.h.
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/b200i.h"
#include "comm.cuh"
#include "decode.cuh"
#include "decode_pair.cuh"
#include "gemm_int8_mma.cuh"
#include "gemm_int8_tma.cuh"
#include "gemm_int8_pair.cuh"
#include "gemm_int15.cuh"
#include "decoder.cuh"
#include "gemm_tile.cuh"
#include "gemm_skinny.cuh"
#include "gemm_packed.cuh"
#include "gemm_tall.cuh"
#include "host_copy.cuh"
#include "gemm_skinny_reg.cuh"
#include "gemm_rows.cuh"
#include "gemm_band.cuh"
#include "gemm_stream.cuh"
#include "lowbit.cuh"

using namespace b200i;

namespace {

std::atomic<long long> g_launches{0};

int64_t fail(char *err, int64_t cap, const char *fmt, ...) {
    if (err && cap > 0) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(err, (size_t)cap, fmt, ap);
        va_end(ap);
    }
    return 1;
}
void clear(char *err, int64_t cap) {
    if (err && cap > 0) err[0] = 0;
}

#define CUDA_TRY(expr)                                                                                      \
    do {                                                                                                    \
        cudaError_t e_ = (expr);                                                                            \
        if (e_ != cudaSuccess) return fail(err, err_cap, "b200i: %s failed: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

constexpr int MAX_DEVICES = 64;
struct DeviceInfo {
    int sms = 148;
    bool known = false;
};
DeviceInfo g_info[MAX_DEVICES];
std::mutex g_mu;

int sm_count(int device) {
    if (device < 0 || device >= MAX_DEVICES) return 148;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_info[device].known) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && v > 0) g_info[device].sms = v;
        g_info[device].known = true;
    }
    return g_info[device].sms;
}

int select_device(int64_t device, char *err, int64_t err_cap, int *out) {
    int dev = 0;
    if (device >= 0) {
        dev = (int)device;
        CUDA_TRY(cudaSetDevice(dev));
    } else {
        CUDA_TRY(cudaGetDevice(&dev));
    }
    if (dev < 0 || dev >= MAX_DEVICES) return fail(err, err_cap, "b200i: device %d is outside the %d devices this library tracks", dev, MAX_DEVICES);
    *out = dev;
    return 0;
}

// The status word of the bounded device-side waits, read and cleared. Every host-pointer entry calls this after its
// final synchronise, so a wait that ran out can never return as a silent success; device-pointer callers read it
// through b200i_decode_status when they next synchronise.
int64_t check_wait_status(char *err, int64_t err_cap, const char *who) {
    int v = 0, zero = 0;
    CUDA_TRY(cudaMemcpyFromSymbol(&v, g_decode_status, sizeof(int)));
    if (v == 0) return 0;
    CUDA_TRY(cudaMemcpyToSymbol(g_decode_status, &zero, sizeof(int)));
    return fail(err, err_cap, "%s: a bounded device-side wait ran out (status %d); the output is incomplete", who, v);
}

// ---- plans -----------------------------------------------------------------------------
enum { PLAN_AUTO = -1, PLAN_FLAT = 0, PLAN_T128 = 1, PLAN_T64 = 2, PLAN_DECODE = 3, PLAN_T32 = 4, PLAN_T128X64 = 5, PLAN_SKINNY = 6, PLAN_PACKED = 7, PLAN_TALL = 8, PLAN_ROWS = 9, PLAN_BAND = 10, PLAN_STREAM = 11 };

// Up to this many rows the weight-streaming decode plan is preferred to the skinny plan; float32 weights at four rows then take
// the rows plan where their call's workspace holds its nodes (rows_preferred: [11008, 4096] 55 us). Low-bit weights switch
// earlier unless the leaf-pair kernel fits (up to four rows): at three and four rows decode_kernel's serial chains cost more
// than the register skinny kernel's eight-row tile (int8 [11008, 4096]: 44 us against 37 us at four rows, 40 against 36 at
// three), except on a very wide weight, where its row streams run at their best
// ([50304, 2048]: bf16 79 us against 98 at four rows, int8 60 against 69 at three).
constexpr int DECODE_PREFER_M = 4;
constexpr long long DECODE_WIDE_N = 32768;
constexpr int DECODE_PREFER_M_LOWBIT = 2;

struct Plan {
    int kind;
    int group_leaves; // S
    int groups;       // G
};

struct TileCfg {
    int kind, bm, bn, per_sm;
    double eff; // fraction of the fused-multiply-add peak the kernel sustains on a full tile (measured)
};
const TileCfg TILE_CFGS[] = {
    {PLAN_T128, 128, 128, 2, 0.55},
    {PLAN_T64, 64, 64, 3, 0.33},
    {PLAN_T32, 32, 128, 4, 0.40},
};

int pow2_floor(int v) {
    int p = 1;
    while (p * 2 <= v) p *= 2;
    return p;
}

// Modelled time of a tiled plan in SM cycles: waves of CTAs over the SM slots,
// each CTA running its share of the leaves, plus the traffic of the group nodes
// and the second launch when the leaves are split.
double tiled_cost(const TileCfg &cfg, long long m, long long n, int leaf, int leaves, int s, int sms) {
    const long long tiles = ((m + cfg.bm - 1) / cfg.bm) * ((n + cfg.bn - 1) / cfg.bn);
    const int groups = (leaves + s - 1) / s;
    const long long ctas = tiles * groups;
    const long long slots = (long long)sms * cfg.per_sm;
    const long long waves = (ctas + slots - 1) / slots;
    const double cta = (double)cfg.bm * cfg.bn * (double)leaf * s * cfg.per_sm / (128.0 * cfg.eff);
    double t = (double)waves * cta + 4000.0;
    if (groups > 1) t += (double)groups * m * n * 8.0 / 2500.0 + 6000.0; // node write + read at HBM rate, second launch
    return t;
}

Plan choose_plan(long long m, long long n, long long k, int sms) {
    const int leaf = (int)leaf_size(k), leaves = (int)leaf_count(k);
    Plan best{PLAN_T128, leaves > 0 ? leaves : 1, 1};
    double best_t = 1e300;
    const int max_s = pow2_floor(leaves > 0 ? leaves : 1) * ((leaves & (leaves - 1)) ? 2 : 1);
    for (const TileCfg &cfg : TILE_CFGS) {
        for (int s = max_s; s >= 1; s /= 2) {
            const int groups = (leaves + s - 1) / s;
            if (groups > MAX_GROUPS) break;
            const double t = tiled_cost(cfg, m, n, leaf, leaves, s, sms);
            if (t < best_t) { best_t = t; best = Plan{cfg.kind, s, groups}; }
        }
    }
    if (best.groups <= 1) best.group_leaves = leaves > 0 ? leaves : 1;
    return best;
}

// The skinny plan's leaf split. Float32 weights (shared-memory kernel): the largest
// power-of-two group that still gives every CTA slot of the device a CTA, else
// single leaves. Low-bit weights (register kernel): the split minimises a modelled
// time in microseconds fitted to measurements on B200 -- rounds of CTAs per SM times
// (leaves per CTA at the kernel's sustained rate, slower while an SM holds fewer than
// three CTAs, plus a fixed cost per CTA), plus the second launch and the L2-resident
// node traffic of the group fold.
Plan choose_skinny(long long m, long long n, long long k, int sms, bool lowbit) {
    const int leaves = (int)leaf_count(k) > 0 ? (int)leaf_count(k) : 1;
    const int max_s = pow2_floor(leaves) * ((leaves & (leaves - 1)) ? 2 : 1);
    int min_s = 1;
    while ((leaves + min_s - 1) / min_s > MAX_GROUPS) min_s *= 2;
    int best = min_s;
    if (lowbit) {
        const int bm = skr_bm((int)m), bn = skr_bn((int)m);
        const long long tiles = ((n + bn - 1) / bn) * ((m + bm - 1) / bm);
        const double rate = bm >= 32 ? 0.25e6 : (bm >= 16 ? 0.20e6 : 0.15e6); // flops per microsecond per SM
        // a CTA's leaf: its multiply-adds at that rate, or its weight bytes at an SM's share of the HBM stream
        const double leaf_us = std::max(2.0 * bm * bn * (double)leaf_size(k) / rate, (double)bn * (double)leaf_size(k) / 40.0e3);
        double best_t = 1e300;
        for (int s = max_s; s >= min_s; s /= 2) {
            const int groups = (leaves + s - 1) / s;
            const long long ctas = tiles * groups;
            const long long rounds = (ctas + sms - 1) / sms;
            double thin = ctas <= sms ? 1.25 : (ctas <= 2 * sms ? 1.08 : 1.0);
            double t = (double)rounds * (s * leaf_us * thin + 0.4);
            if (groups > 1) t += 2.5 + (double)groups * m * n * 8.0 / 7.5e6;
            if (t < best_t) { best_t = t; best = s; }
        }
    } else {
        const long long col_ctas = (n + skinny_bn((int)m) - 1) / skinny_bn((int)m);
        const long long want = (long long)sms * skinny_per_sm((int)m) * 9 / 10;
        for (int s = max_s; s >= min_s; s /= 2)
            if (col_ctas * ((leaves + s - 1) / s) >= want) { best = s; break; }
    }
    Plan p{PLAN_SKINNY, best, (leaves + best - 1) / best};
    if (p.groups <= 1) p.group_leaves = leaves;
    return p;
}

bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// ---- optional device timing of the product's main kernel ------------------------------------
// While enabled, every product call records a CUDA event pair on its stream around its main
// kernel (the tile / packed / skinny / decode kernel; not the packing passes, not the group fold).
struct KernelTiming {
    bool on = false;
    int used = 0;
    std::vector<cudaEvent_t> ev; // pairs
};
KernelTiming g_timing;
std::mutex g_timing_mu;
constexpr int TIMING_MAX_PAIRS = 4096;
thread_local bool t_no_timing = false; // set by the allocation-free entry: creating an event may allocate
int timing_begin(cudaStream_t st) {
    if (t_no_timing) return -1;
    std::lock_guard<std::mutex> lock(g_timing_mu);
    if (!g_timing.on || g_timing.used >= TIMING_MAX_PAIRS) return -1;
    const int slot = g_timing.used++;
    while ((int)g_timing.ev.size() < 2 * (slot + 1)) {
        cudaEvent_t e;
        if (cudaEventCreate(&e) != cudaSuccess) { cudaGetLastError(); g_timing.used = slot; return -1; }
        g_timing.ev.push_back(e);
    }
    cudaEventRecord(g_timing.ev[2 * slot], st);
    return slot;
}
void timing_end(int slot, cudaStream_t st) {
    if (slot < 0) return;
    std::lock_guard<std::mutex> lock(g_timing_mu);
    cudaEventRecord(g_timing.ev[2 * slot + 1], st);
}

size_t round256(size_t v) { return (v + 255) / 256 * 256; }

// rows below which packing the operands costs more than the bulk-copy pipeline returns
constexpr long long PACKED_MIN_EXTENT = 256;
// The packed plan replaces the 128 x 128 tile plan from 256 rows and columns up, and any tile plan when the rows
// are one or two (nearly) full rows of 128 x 128 tiles over a wide, deep product (128 x 11008 x 4096: 305 us
// against 370 us for the 32 x 128 tiles).
inline bool packed_candidate(int tile_kind, long long m, long long n, long long k) {
    if (tile_kind == PLAN_T128 && m >= PACKED_MIN_EXTENT && n >= PACKED_MIN_EXTENT) return true;
    const long long padded = (m + PK_TILE - 1) / PK_TILE * PK_TILE;
    return tile_kind != PLAN_FLAT && m >= 117 && m <= 256 && padded * 10 <= m * 11 && n >= 2048 && k >= 1024;
}
size_t packed_need(long long m, long long n, long long k, int groups) {
    return round256(groups > 1 ? (size_t)groups * m * n * 4 : 0) + pk_workspace_bytes(m, n, k);
}

// A small decode batch with a column's whole contraction in one CTA (gemm_rows.cuh) up to sixteen leaves. Past that the
// activations of all leaves leave too short a ring, and groups of eight leaves on as many more CTAs win in spite of the
// second launch (float32 [11008, 4096] at 8 rows: 57 us against 67 in sixteens and 140 whole).
Plan choose_rows(long long k) {
    const int leaves = (int)leaf_count(k);
    if (leaves <= 16) return Plan{PLAN_ROWS, leaves, 1};
    int run = 8;
    while ((leaves + run - 1) / run > MAX_GROUPS) run *= 2;
    return Plan{PLAN_ROWS, run, (leaves + run - 1) / run};
}
// Modelled microseconds of a rows launch, its fold included: what a warp walks one leaf after the other at the rate of its strip
// shape, slower while more than eight warps share the SM, plus staging and start. Fitted to 6600 launches of 300 to 50304
// columns by 768 to 8192 steps (nine in ten within 10 %; ragged depths and strips are where the plan's time jumps).
double rows_us(const RowsLaunch &r, long long m, long long n, int wkind) {
    static const double leaf_us[3][5][2] = { // [float32, bf16, int8][8 rows: 8 or 16, 32, 64 columns; 16 rows: 8 or 16, 32][to 8 warps, at 16]
        {{2.2, 4.2}, {4.9, 8.8}, {10.2, 13.2}, {4.0, 6.7}, {12.4, 16.4}},
        {{1.8, 3.4}, {3.6, 7.1}, {7.5, 10.7}, {3.3, 5.5}, {9.6, 14.1}},
        {{1.3, 2.6}, {2.7, 5.6}, {5.4, 7.7}, {2.6, 4.8}, {5.8, 10.6}}};
    const int columns = r.lc * r.cpl, shape = (columns <= 16 ? 0 : (columns == 32 ? 1 : 2)) + (m <= 8 ? 0 : 3);
    const double *rate = leaf_us[wkind == W_F32 ? 0 : (wkind == W_BF16 ? 1 : 2)][shape];
    const double crowd = std::max(0, r.p.warps - 8) / 8.0;
    double t = 2.95 + 0.72 * r.act_bytes / 32768.0 + r.rounds * (rate[0] + (rate[1] - rate[0]) * crowd);
    if (r.groups > 1) t += 2.4 + (double)r.groups * m * n * 8.0 / 7.5e6;
    return t;
}
// The same for the plan that the call would take otherwise (`before`: decode or skinny), fitted to the same sizes.
double before_rows_us(const Plan &before, long long m, long long n, long long k, int wkind, int sms) {
    const double words = (double)n * k / 1e6, steps = k / 1000.0;
    if (before.kind == PLAN_DECODE && wkind == W_F32) { // a warp walks 32 rows: to 32 rows an SM, to 64, above
        if (n <= 32ll * sms) return 3.6 + 3.73 * steps + 0.6 * words + 0.27 * n / 1000.0;
        return n <= 64ll * sms ? 4.3 + 6.0 * steps + 0.74 * words : 4.5 + 3.5 * steps + 1.27 * words;
    }
    if (before.kind == PLAN_DECODE) { // the leaf-pair kernel, eight leaves of a row at a time (bf16 past 2048 and int8 past 4096
        const double turns = (double)((k + 1023) / 1024); // steps: more than one copy a row, too short a ring)
        return wkind == W_BF16 ? 4.6 + 1.8 * turns + 0.56 * words + (k > 2048 ? 2.0 : 0.0) : 5.4 + (1.78 * turns + 0.28 * words) * (k > 4096 ? 1.5 : 1.0);
    }
    // leaves that an SM walks, a few CTAs beyond a whole number per SM not showing; a CTA alone takes longer over its own
    const long long ctas = (n + 255) / 256 * before.groups - sms / 20;
    const int own = std::min(before.group_leaves, (int)leaf_count(k));
    const double walk = (double)std::max<long long>((ctas + sms - 1) / sms, 1) * own;
    if (wkind == W_F32)
        return m <= 8 ? 9.1 + std::max(4.08 * walk, 9.5 * own - 5.0) + 0.68 * words : 8.7 + std::max(6.4 * walk, 12.0 * own - 6.0) + 0.59 * words;
    return wkind == W_BF16 ? 6.2 + std::max(2.38 * walk, 5.2 * own - 3.0) + 0.3 * words : 6.1 + std::max(2.34 * walk, 4.4 * own - 2.5) + 0.135 * words;
}
// Float32 weights at 4 to 8 rows and, while a CTA has one strip of sixteen columns, at 9 to 16; int8 ones at 4 rows to 3072
// columns, at 5 to 8 rows also where they are deep; bf16 ones to 3072 columns; low-bit ones at 9 to 16 rows while small enough to
// be bound by latency. Inside these lines the modelled times decide: float32 [2304, 768] at eight rows 6.5 against 14 us,
// [11008, 4096] 57 against 80, but [32000, 1792] 138 against 96 and [1536, 6160] 28 against 21 (a strip of 64 columns for ten).
// (At 5 to 8 float32 rows from nine million words the answer stands where strips come out even, stream_preferred, where the depth
// is past 32768 steps, and where a call's workspace is too small for the stream plan.)
inline bool rows_preferred(const Plan &before, long long m, long long n, long long k, int wkind, int sms) {
    RowsLaunch r;
    if (m < 4 || !rows_layout(m, n, k, wkind, choose_rows(k).group_leaves, sms, r)) return false;
    if (m > 8 && (n > 16ll * sms || (wkind != W_F32 && k > 1024))) return false;
    if (m <= 8 && wkind != W_F32 && n > 3072 && (wkind == W_BF16 || m <= 4 || k < 4096)) return false;
    if (m > 8 && wkind != W_F32) return true;
    if (before.kind != PLAN_DECODE && before.kind != PLAN_SKINNY) return true;
    return rows_us(r, m, n, wkind) < before_rows_us(before, m, n, k, wkind, sms);
}

// 9 to 16 rows: modelled microseconds of the band kernel (fitted like rows_us, within 5 % from two million words up). Up to one CTA
// an SM a leaf takes 8.4 us, above that two share an SM and every round of 2 * SMs takes 13 a leaf, however few CTAs the last
// one has (they start beside the others). Ragged groups count by their leaves.
double band_us(long long m, long long n, long long k, int group_leaves, int sms) {
    const int leaves = (int)leaf_count(k), sl = std::min(group_leaves, leaves), groups = (leaves + sl - 1) / sl;
    const long long ctas = ((n + BD_BN - 1) / BD_BN * leaves + sl - 1) / sl;
    double t = 2.9 + (ctas <= sms ? 2.0 + 8.37 * sl : (double)((ctas + 2 * sms - 1) / (2 * sms)) * (2.73 + 13.0 * sl));
    if (groups > 1) t += 2.1 + (double)groups * m * n * 8.0 / 7.5e6;
    return t;
}
// 9 to 32 rows: the leaf split of the band kernel. Modelled time in microseconds: band_us up to sixteen rows; above, waves of
// CTAs over two slots per SM (leaves per CTA at the kernel's rate, a last wave that fills at most half the slots counting 0.55
// because its CTAs are alone on their SMs, + 1 us to start), plus the second launch and the L2-resident node traffic of the fold.
Plan choose_band(long long m, long long n, long long k, int sms) {
    const int leaves = (int)leaf_count(k) > 0 ? (int)leaf_count(k) : 1;
    const int max_s = pow2_floor(leaves) * ((leaves & (leaves - 1)) ? 2 : 1);
    const long long tiles = (n + BD_BN - 1) / BD_BN, slots = 2ll * sms;
    int min_s = 1;
    while ((leaves + min_s - 1) / min_s > MAX_GROUPS) min_s *= 2;
    int best = max_s;
    double best_t = 1e300;
    for (int sl = max_s; sl >= min_s; sl /= 2) {
        const int groups = (leaves + sl - 1) / sl;
        const long long ctas = tiles * groups, whole = ctas / slots, rest = ctas % slots;
        const double waves = (double)whole + (rest == 0 ? 0.0 : (2 * rest <= slots ? 0.55 : 1.0));
        double t = waves * (std::min(sl, leaves) * 9.5 + 1.0);
        if (groups > 1) t += 2.5 + (double)groups * m * n * 8.0 / 7.5e6;
        if (m <= 16) t = band_us(m, n, k, sl, sms);
        if (t < best_t) { best_t = t; best = sl; }
    }
    Plan p{PLAN_BAND, best, (leaves + best - 1) / best};
    if (p.groups <= 1) p.group_leaves = leaves;
    return p;
}
// Float32 weights from ten million words up (the sizes on both sides of the line stand in gemm_band.cuh); up to sixteen rows also
// by the modelled times ([8192, 1792] 35 against 41 us, but [5120, 4096] 55 against 51), which matters past 32768 steps and where a
// call's workspace is too small for the stream plan: that takes the others.
inline bool band_size(long long n, long long k, int wkind) { return wkind == W_F32 && (double)n * (double)k >= 1.0e7; }
inline bool band_preferred(const Plan &skinny, const Plan &band, long long m, long long n, long long k, int sms) {
    return m > 16 || band_us(m, n, k, band.group_leaves, sms) < 0.97 * before_rows_us(skinny, m, n, k, W_F32, sms);
}

// 5 to 16 rows over large weights: modelled microseconds of the streaming kernel, its fold included. A CTA's warps take its items
// in turn; a turn of sixteen runs at the warps' common rate, the last one at its own number of warps or, with few, at the pace of
// one. Fitted to 1800 launches of 1024 to 50304 columns by 768 to 12208 steps in groups of one, two and four leaves (nine in ten
// within 6 % for bf16, 9 for float32).
double stream_us(long long m, long long n, long long k, int wkind, int group_leaves, int sms) {
    static const double fit[2][2][5] = { // [float32, bf16][8 rows, 16]: start, a leaf of one warp among many, alone, fold, a turn's start
        {{5.5, 0.85, 3.6, 2.4, 1.0}, {8.8, 1.06, 4.5, 3.3, 1.6}}, {{8.2, 0.566, 3.65, 3.2, 0.74}, {10.3, 0.959, 4.2, 3.9, 2.1}}};
    const double *f = fit[wkind == W_F32 ? 0 : 1][m <= 8 ? 0 : 1];
    const long long leaves = leaf_count(k), run = std::min<long long>(group_leaves, leaves), groups = (leaves + run - 1) / run;
    const long long items = (n + SM_CB - 1) / SM_CB * groups, ctas = std::min<long long>(items, sms), own = (items + ctas - 1) / ctas;
    const long long turns = own / SM_WARPS, rest = own % SM_WARPS;
    const double walk = groups > 1 ? (double)run : k / 128.0; // leaves of an item
    double t = f[0] + (double)turns * (SM_WARPS * f[1] * walk + f[4]);
    if (rest) t += std::max(f[2], (double)rest * f[1]) * walk + f[4];
    if (groups > 1) t += f[3] + (double)groups * m * n * 8.0 / 7.5e6;
    return t;
}
// Leaves per group, by the weight's words: single ones while every warp has an item or two, more where the items are many, so that
// fewer nodes pass through L2 (float32, 8 rows, groups of one / two / four leaves: [5536, 2208] 20.2 / 23 / 31 us, [10512, 2256]
// 32.6 / 28.9 / 36, [11008, 4096] 45.6 / 49.2 / 42.7). Groups of four want eight leaves at least. For bf16 another split is taken
// where the model has it 4 or 5 % faster: at the words' lines a CTA's items just pass sixteen, and a second turn of one or two warps
// costs as much as a whole one (8 rows, groups of two / four [9600, 4096] 40.2 / 35.9, of four / two / one [33236, 2064] 61 / 49 / 51).
Plan choose_stream(long long m, long long n, long long k, int wkind, int sms) {
    const int leaves = (int)leaf_count(k) > 0 ? (int)leaf_count(k) : 1;
    const double words = (double)n * (double)k;
    auto groups = [&](int run) { return (leaves + run - 1) / run; };
    int run = words < 16.0e6 ? 1 : (words < 42.0e6 || leaves < 8 ? 2 : 4);
    while (run < SM_MAX_RUN && groups(run) > MAX_GROUPS) run *= 2;
    if (wkind == W_BF16) {
        double least = (m <= 8 ? 0.96 : 0.95) * stream_us(m, n, k, wkind, run, sms);
        for (int r = 1; r <= SM_MAX_RUN; r *= 2)
            if (groups(r) <= MAX_GROUPS && stream_us(m, n, k, wkind, r, sms) < least) {
                least = stream_us(m, n, k, wkind, r, sms);
                run = r;
            }
    }
    return Plan{PLAN_STREAM, run, groups(run)};
}
// Lines from 57 sizes of 768 to 50304 columns by 768 to 8192 steps at 5, 8, 11 and 16 rows, the plan before -> this one, in
// microseconds: float32 from nine million words (8 rows [4935, 1840] 21.4 -> 16.8, 16 rows 32.7 -> 22.2; below, [1376, 5824]
// 17.4 -> 16.6 but [3776, 1600] 12.5 -> 15.9); bf16 from 30 million at 5 to 8 rows ([7632, 4192] 35.6 -> 30.7; below, [2800, 7472]
// 23.8 -> 25.3) and from 42 million at 9 to 16 ([11008, 4096] 67.4 -> 58.0; below, [18880, 2064] 58.1 -> 62.2). Above the lines the
// modelled times decide: a rows plan whose strips come out even keeps the call (float32, 8 rows: [4736, 1920] 12.9 against 15.7,
// [3072, 3072] 15.5 against 16.1, but [4800, 2000] 23.3 against 16.9), and so does the register skinny kernel where the leaves or
// columns do not divide well (bf16, 9 rows: [44000, 1040] 60.9 against 66.3, [25254, 2064] 67.6 against 72.5).
inline bool stream_preferred(const Plan &before, const Plan &stream, long long m, long long n, long long k, int wkind, int sms) {
    const double words = (double)n * (double)k;
    if (m < 5 || words < (wkind == W_F32 ? 9.0e6 : (m <= 8 ? 30.0e6 : 42.0e6))) return false;
    const double us = stream_us(m, n, k, wkind, stream.group_leaves, sms);
    if (before.kind == PLAN_ROWS && m <= 8) {
        RowsLaunch r;
        return !rows_layout(m, n, k, wkind, before.group_leaves, sms, r) || us < 0.94 * rows_us(r, m, n, wkind);
    }
    if (wkind == W_F32 || before.kind != PLAN_SKINNY) return true;
    if (m <= 8) return us < 0.94 * before_rows_us(before, m, n, k, wkind, sms);
    const long long ctas = (n + 255) / 256 * before.groups - sms / 20; // the same for 9 to 16 rows, fitted to 150 sizes (nine in ten within 9 %)
    const double walk = (double)std::max<long long>((ctas + sms - 1) / sms, 1) * std::min<long long>(before.group_leaves, leaf_count(k));
    return us < 0.94 * (8.7 + 1.21 * walk + 0.958 * words / 1e6 + 0.51 * (double)(m - 8));
}

// A^T B of few cells over many rows: every leaf of every 32 x 32 tile as a warp of its own (gemm_tall.cuh).
constexpr long long TALL_MIN_LEAVES = 16;
inline bool tall_fits(long long m, long long n, long long k, int op, int wkind) {
    return op == OP_TN && wkind == W_F32 && m <= TALL_MAX_EXTENT && n <= TALL_MAX_EXTENT && leaf_count(k) >= 2;
}
inline bool tall_candidate(long long m, long long n, long long k) {
    return m <= TALL_MAX_EXTENT && n <= TALL_MAX_EXTENT && leaf_count(k) >= TALL_MIN_LEAVES;
}

// The packed plan's leaf split: with at least two CTAs per slot of the device the tiles alone keep every SM busy
// (a CTA left alone on an SM in the last wave runs at nearly twice the speed, so a partial wave costs little)
// and a split would only add group nodes; below that, the tile plan's split stands.
Plan packed_split(const Plan &tile_plan, long long m, long long n, long long k, int sms) {
    const long long tiles = ((m + PK_TILE - 1) / PK_TILE) * ((n + PK_TILE - 1) / PK_TILE);
    Plan p = tile_plan;
    p.kind = PLAN_PACKED;
    const int leaves = (int)leaf_count(k) > 0 ? (int)leaf_count(k) : 1;
    if (tiles >= 4ll * sms) { p.groups = 1; p.group_leaves = leaves; return p; }
    // Few tiles: split the leaves so that the CTA slots (two per SM) fill in whole waves. Modelled time in
    // microseconds: waves x (leaves per CTA at 21.8 us per 128-step leaf -- a 128 x 128 tile at the kernel's
    // measured rate -- plus 1 us per CTA), plus the second launch and the L2-resident node traffic of the fold.
    const long long slots = 2ll * sms;
    const double leaf_us = 21.8 * (double)leaf_size(k) / 128.0;
    const int max_s = pow2_floor(leaves) * ((leaves & (leaves - 1)) ? 2 : 1);
    int min_s = 1;
    while ((leaves + min_s - 1) / min_s > MAX_GROUPS) min_s *= 2;
    int best = max_s;
    double best_t = 1e300;
    for (int sl = max_s; sl >= min_s; sl /= 2) {
        const int groups = (leaves + sl - 1) / sl;
        // a last wave that fills at most half the slots leaves its CTAs alone on their SMs, at nearly twice the speed
        const long long ctas = tiles * groups, whole = ctas / slots, rest = ctas % slots;
        const double waves = (double)whole + (rest == 0 ? 0.0 : (2 * rest <= slots ? 0.55 : 1.0));
        double t = waves * (sl * leaf_us + 1.0);
        if (groups > 1) t += 3.0 + (double)groups * m * n * 8.0 / 7.5e6;
        if (t < best_t) { best_t = t; best = sl; }
    }
    p.group_leaves = best;
    p.groups = (leaves + best - 1) / best;
    if (p.groups <= 1) p.group_leaves = leaves;
    return p;
}

// Packs both operands into `scratch` (panels, then flags) and runs the packed kernel.
void packed_configure() {
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaFuncSetAttribute(gemm_packed_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PK_SMEM_BYTES);
        cudaFuncSetAttribute(gemm_packed_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PK_RAW_SMEM_BYTES);
        configured[dev] = true;
    }
}
// The packing passes of two operands as one launch (extent 0: no left operand).
void launch_pack(const PackArgs &a, const PackArgs &b, int wkind, cudaStream_t st) {
    const int ta = (a.extent + PK_TILE - 1) / PK_TILE, tb = (b.extent + PK_TILE - 1) / PK_TILE;
    for (int y0 = 0; y0 < ta + tb; y0 += 65535) { // grid.y holds 65535 tiles (more than 8 million rows need a second launch)
        const dim3 grid((unsigned)(a.leaves * ((a.wpl + 1) / 2)), (unsigned)std::min(ta + tb - y0, 65535));
        if (wkind == W_F32) pack_operands_kernel<W_F32><<<grid, 256, 0, st>>>(a, b, ta, y0);
        else if (wkind == W_BF16) pack_operands_kernel<W_BF16><<<grid, 256, 0, st>>>(a, b, ta, y0);
        else if (wkind == W_INT8_EXP) pack_operands_kernel<W_INT8_EXP><<<grid, 256, 0, st>>>(a, b, ta, y0);
        else pack_operands_kernel<W_INT8_SCALE><<<grid, 256, 0, st>>>(a, b, ta, y0);
    }
}

void launch_pack_one(const PackArgs &x, int wkind, cudaStream_t st) {
    PackArgs none = x;
    none.extent = 0;
    launch_pack(none, x, wkind, st);
}

int launch_packed(const GemmArgs &g, int groups, unsigned char *scratch, cudaStream_t st) {
    packed_configure();
    const int wpl = pk_windows_per_leaf(g.leaf);
    float *pa = reinterpret_cast<float *>(scratch);
    float *pb = pa + pk_panel_floats(g.m, g.k);
    unsigned char *fa = reinterpret_cast<unsigned char *>(pb + pk_panel_floats(g.n, g.k));
    unsigned char *fb = fa + pk_flag_bytes(g.m, g.k);
    // quads: k-contiguous rows need k and the leaves in whole quads, the other layout whole quads of rows
    const bool k4 = (g.k % 4 == 0) && (g.leaves == 1 || g.leaf % 4 == 0);
    const size_t balign = g.wkind == W_F32 ? 16 : (g.wkind == W_BF16 ? 8 : 4);
    const bool a_kc = g.op != OP_TN, b_kc = g.op == OP_NT;
    PackArgs a{pa, fa, g.a, nullptr, g.m, g.k, g.leaf, g.leaves, wpl, a_kc, (a_kc ? k4 : g.m % 4 == 0) && aligned(g.a, 16)};
    PackArgs b{pb, fb, g.b, g.bscale, g.n, g.k, g.leaf, g.leaves, wpl, b_kc, (b_kc ? k4 : g.n % 4 == 0) && aligned(g.b, balign)};
    // one row of tiles over float32 rows of whole quads, and leaves of whole stages: B is read where it lies
    const bool raw = g.m <= PK_TILE && g.wkind == W_F32 && b.kcontig && b.vec && (g.leaves == 1 || g.leaf % PK_SK == 0);
    if (raw) launch_pack_one(a, W_F32, st);
    else launch_pack(a, b, g.wkind, st);
    PackedGemmArgs p{pa, pb, fa, fb, g.c, g.ws, g.m, g.n, g.k, g.leaf, g.leaves, wpl, g.group_leaves, groups,
                     (g.n + PK_TILE - 1) / PK_TILE, g.vec_c};
    dim3 grid((unsigned)(((g.m + PK_TILE - 1) / PK_TILE) * p.tiles_n), (unsigned)groups);
    const int tslot = timing_begin(st);
    p.braw = static_cast<const float *>(g.b);
    if (raw) gemm_packed_kernel<true><<<grid, PK_THREADS, PK_RAW_SMEM_BYTES, st>>>(p);
    else gemm_packed_kernel<false><<<grid, PK_THREADS, PK_SMEM_BYTES, st>>>(p);
    timing_end(tslot, st);
    return 2;
}

template <int BM, int BN, int RM, int RN, int MINB>
void launch_tile(GemmArgs &g, int groups, cudaStream_t st) {
    using S = TileShape<BM, BN, RM, RN>;
    static std::atomic<bool> configured[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaFuncSetAttribute(gemm_tile_kernel<BM, BN, RM, RN, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM_BYTES);
        configured[dev] = true;
    }
    g.tiles_n = (g.n + BN - 1) / BN;
    dim3 grid((unsigned)(((g.m + BM - 1) / BM) * g.tiles_n), (unsigned)groups);
    gemm_tile_kernel<BM, BN, RM, RN, MINB><<<grid, S::THREADS, S::SMEM_BYTES, st>>>(g);
}

unsigned grid_for(long long work_items, int block, int sms) {
    long long blocks = (work_items + block - 1) / block;
    const long long cap = (long long)sms * 16;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return (unsigned)blocks;
}

size_t plan_need(const Plan &p, long long m, long long n, long long k) { // workspace bytes
    if (p.kind == PLAN_PACKED) return packed_need(m, n, k, p.groups);
    if (p.kind == PLAN_TALL) return tall_workspace_bytes(m, n, k);
    return p.groups > 1 ? (size_t)p.groups * m * n * 4 : 0;
}

// The automatic choice. `al16`: both operands start on 16 bytes; `pairs`: a gated store; `nodes`: the caller folds.
// `fits(plan)`: the call's workspace holds what the plan needs; a call whose workspace does not keeps the plan before it.
struct AutoCall {
    long long m, n, k;
    int op, wkind, sms;
    bool al16, pairs, nodes, maps; // maps: tensor maps can be made
};
template <class Fits>
Plan choose_auto(const AutoCall &x, Fits fits) {
    const long long m = x.m, n = x.n, k = x.k;
    Plan plan = choose_plan(m, n, k, x.sms);
    auto take = [&](const Plan &p) { if (fits(p)) plan = p; };
    if (packed_candidate(plan.kind, m, n, k)) take(packed_split(plan, m, n, k, x.sms));
    const bool dec = decode_plan_fits(m, n, k, x.op, x.wkind) && x.al16;
    const bool skinny = skinny_plan_fits(m, n, k, x.op) && x.al16;
    const bool wide = n >= DECODE_WIDE_N && (x.wkind == W_BF16 || m == 3);
    // low-bit weights: the leaf-pair decode kernel wherever it fits (up to four rows), else the rule above
    const bool pair = x.wkind != W_F32 && decode_pair_fits(m, n, k, x.op, x.wkind, x.sms);
    const int prefer_m = pair ? DP_MAX_M : ((x.wkind != W_F32 && skinny && !wide) ? DECODE_PREFER_M_LOWBIT : DECODE_PREFER_M);
    const Plan decode{PLAN_DECODE, (int)leaf_count(k), 1};
    if (dec && m <= prefer_m && !(skinny && x.pairs)) plan = decode; // (a gated store needs the skinny plan)
    else if (skinny) plan = choose_skinny(m, n, k, x.sms, x.wkind != W_F32);
    else if (dec) plan = decode;
    if (skinny && m > 8 && band_size(n, k, x.wkind)) {
        const Plan band = choose_band(m, n, k, x.sms);
        if (band_preferred(plan, band, m, n, k, x.sms)) take(band);
    } else if (rows_plan_fits(m, n, k, x.op) && x.al16 && rows_preferred(plan, m, n, k, x.wkind, x.sms)) {
        take(choose_rows(k));
    }
    if (skinny && x.maps && (x.wkind == W_F32 || x.wkind == W_BF16) && m <= SM_MAX_ROWS) {
        const Plan stream = choose_stream(m, n, k, x.wkind, x.sms);
        if (stream.groups <= MAX_GROUPS && stream_plan_fits(m, n, k, x.op, x.wkind, stream.group_leaves, x.sms) &&
            stream_preferred(plan, stream, m, n, k, x.wkind, x.sms))
            take(stream);
    }
    if (tall_fits(m, n, k, x.op, x.wkind) && tall_candidate(m, n, k) && !x.nodes && !x.pairs) take(Plan{PLAN_TALL, 1, (int)leaf_count(k)});
    return plan;
}

int64_t launch_product(int dev, cudaStream_t st, float *c, const float *a, const void *b, const void *bscale, int wkind,
                       int64_t m, int64_t n, int64_t k, int op, int plan_kind, int64_t group_leaves, void *ws,
                       int64_t ws_bytes, char *err, int64_t err_cap, Epilogue epi = Epilogue{nullptr, EPI_ACT_NONE},
                       int64_t *leave_nodes = nullptr) {
    // leave_nodes: the caller folds the leaf-group nodes itself (the gather that follows a sharded product does); on
    // return it holds the number of nodes per cell left in ws, 1 when c is finished as usual
    if (leave_nodes) *leave_nodes = 1;
    if (m <= 0 || n <= 0 || k <= 0)
        return fail(err, err_cap, "identical gemm: m, n and k must be positive (got m=%lld n=%lld k=%lld)", (long long)m,
                    (long long)n, (long long)k);
    if (op != OP_NN && op != OP_NT && op != OP_TN) return fail(err, err_cap, "identical gemm: unknown op %d", op);
    if (wkind < W_F32 || wkind > W_INT8_SCALE) return fail(err, err_cap, "identical gemm: unknown weight kind %d", wkind);
    if ((wkind == W_INT8_EXP || wkind == W_INT8_SCALE) && op != OP_NT)
        return fail(err, err_cap, "identical gemm: int8 weight storage is row-scaled and needs op NT");
    if ((wkind == W_INT8_EXP || wkind == W_INT8_SCALE) && !bscale)
        return fail(err, err_cap, "identical gemm: int8 weight storage needs its per-row exponents or scales");
    if (!c || !a || !b) return fail(err, err_cap, "identical gemm: null storage");
    if (m > 0x7FFFFFFF || n > 0x7FFFFFFF || k > 0x7FFFFFFF || m * n > 0x7FFFFFFFll * 64)
        return fail(err, err_cap, "identical gemm: extent out of range");
    if (!aligned(c, 4) || !aligned(a, 4) || (wkind == W_F32 && !aligned(b, 4)) || (wkind == W_BF16 && !aligned(b, 2)))
        return fail(err, err_cap, "identical gemm: misaligned storage");

    GemmArgs g;
    g.a = a; g.b = b; g.bscale = bscale; g.c = c; g.ws = static_cast<float *>(ws);
    g.m = (int)m; g.n = (int)n; g.k = (int)k; g.op = op; g.wkind = wkind;
    g.leaf = (int)leaf_size(k);
    g.leaves = (int)leaf_count(k);
    g.epi = epi;

    Plan plan;
    if (plan_kind == PLAN_AUTO) {
        const bool pairs = epilogue_pairs(g.epi);
        const bool al16 = aligned(b, 16) && aligned(a, 16);
        const bool maps = m <= SM_MAX_ROWS && op == OP_NT && t8_encode_fn() != nullptr; // (asked for where it can matter)
        auto fits = [&](const Plan &p) {
            const size_t need = plan_need(p, m, n, k);
            if (need && (!ws || ws_bytes < (int64_t)need || !aligned(ws, p.kind == PLAN_PACKED ? 256 : 4))) return false;
            return !pairs || p.groups <= 1 || (aligned(ws, 16) && aligned(c, 8)); // the fold of a gated store
        };
        plan = choose_auto(AutoCall{m, n, k, op, wkind, sm_count(dev), al16, pairs, leave_nodes != nullptr, maps}, fits);
    } else {
        plan.kind = plan_kind;
        int s = group_leaves > 0 ? (int)group_leaves : g.leaves;
        if (s & (s - 1)) {
            if (s < g.leaves) return fail(err, err_cap, "identical gemm: a leaf group must be a power of two");
        }
        if (s > g.leaves) s = g.leaves;
        plan.group_leaves = s;
        plan.groups = (g.leaves + s - 1) / s;
        if (plan.groups > 1 && (s & (s - 1))) return fail(err, err_cap, "identical gemm: a leaf group must be a power of two");
        if (plan.kind == PLAN_TALL) {
            if (!tall_fits(m, n, k, op, wkind))
                return fail(err, err_cap, "identical gemm: the tall plan needs op TN, float32 operands, m and n up to %d and at least two leaves", TALL_MAX_EXTENT);
            plan.group_leaves = 1;
            plan.groups = g.leaves;
        } else if (plan.groups > MAX_GROUPS) return fail(err, err_cap, "identical gemm: more than %d leaf groups", MAX_GROUPS);
        if (plan.kind == PLAN_FLAT || plan.kind == PLAN_DECODE) { plan.groups = 1; plan.group_leaves = g.leaves; }
    }
    g.group_leaves = plan.group_leaves;
    g.groups = plan.groups;
    if (plan.groups > 1) {
        const int64_t need = (int64_t)plan.groups * m * n * 4;
        if (!ws || ws_bytes < need)
            return fail(err, err_cap, "identical gemm: workspace of %lld bytes needed, %lld given", (long long)need,
                        (long long)ws_bytes);
    }

    // 128-bit access is legal when the contiguous axis keeps every vector inside a row and aligned
    const bool a_kc = (op != OP_TN), b_kc = (op == OP_NT);
    const bool leaf_ok = (g.leaves == 1) || (g.leaf % 4 == 0);
    g.vec_a = a_kc ? (k % 4 == 0 && leaf_ok && aligned(a, 16)) : (m % 4 == 0 && aligned(a, 16));
    const size_t balign = wkind == W_F32 ? 16 : (wkind == W_BF16 ? 8 : 4);
    g.vec_b = b_kc ? (k % 4 == 0 && leaf_ok && aligned(b, balign)) : (n % 4 == 0 && aligned(b, balign));
    g.vec_c = (n % 4 == 0) && aligned(c, 16) && (plan.groups == 1 || aligned(ws, 16));

    if (epilogue_pairs(g.epi)) {
        // a gated activation needs both columns of a pair in one thread: the skinny plans, whose threads own adjacent
        // columns, apply it in their own store or in the group fold; no other plan spells it
        const bool fold_ok = plan.groups == 1 || (((long long)m * n) % 4 == 0 && aligned(ws, 16) && aligned(c, 8));
        if ((plan.kind != PLAN_SKINNY && plan.kind != PLAN_ROWS && plan.kind != PLAN_BAND && plan.kind != PLAN_STREAM) || n % 4 != 0 || !fold_ok)
            return fail(err, err_cap, "identical gemm: the gated store activation needs the skinny plan (up to 32 rows, op NT, k a multiple of 16) and n a multiple of 4");
    }
    int tslot = -1;
    if (plan.kind != PLAN_PACKED) tslot = timing_begin(st);
    if (plan.kind == PLAN_FLAT) {
        const long long cells = (long long)m * n;
        gemm_flat_kernel<<<(unsigned)((cells + 127) / 128), 128, 0, st>>>(g);
        g_launches++;
    } else if (plan.kind == PLAN_DECODE) {
        if (!decode_plan_fits(m, n, k, op, wkind) || !aligned(b, 16) || !aligned(a, 16))
            return fail(err, err_cap, "identical gemm: the decode plan needs op NT, m <= %d, k a multiple of 16 and 16-byte aligned weights", DECODE_MAX_M);
        g_launches += launch_decode_plan(g, sm_count(dev), st);
    } else if (plan.kind == PLAN_ROWS) {
        RowsLaunch rows;
        if (!rows_plan_fits(m, n, k, op) || !aligned(b, 16) || !aligned(a, 16) || !rows_layout(m, n, k, wkind, plan.group_leaves, sm_count(dev), rows))
            return fail(err, err_cap, "identical gemm: the rows plan needs op NT, m <= %d, k a multiple of 16, 16-byte aligned operands, leaf groups of at most %d and "
                        "(int8) a weight whose row factors fit", RW_MAX_ROWS, rows_group_leaves(m));
        launch_rows(g, rows, st);
        g_launches++;
    } else if (plan.kind == PLAN_BAND) {
        if (!skinny_plan_fits(m, n, k, op) || wkind != W_F32 || !aligned(b, 16) || !aligned(a, 16))
            return fail(err, err_cap, "identical gemm: the band plan needs op NT, m <= 32, float32 weights, k a multiple of 16 and 16-byte aligned operands");
        launch_band(g, st);
        g_launches++;
    } else if (plan.kind == PLAN_STREAM) {
        if (!stream_plan_fits(m, n, k, op, wkind, plan.group_leaves, sm_count(dev)) || !aligned(b, 16) || !aligned(a, 16) || !launch_stream(g, sm_count(dev), st))
            return fail(err, err_cap, "identical gemm: the stream plan needs op NT, m <= %d, float32 or bf16 weights, k a multiple of 16, 16-byte aligned operands, leaf "
                        "groups of at most %d and tensor maps", SM_MAX_ROWS, SM_MAX_RUN);
        g_launches++;
    } else if (plan.kind == PLAN_TALL) {
        launch_tall(g, st); // its own fold, the store epilogue included
        g_launches += 2;
        plan.groups = 1;
    } else if (plan.kind == PLAN_T128) {
        launch_tile<128, 128, 2, 2, 2>(g, plan.groups, st);
        g_launches++;
    } else if (plan.kind == PLAN_T64) {
        launch_tile<64, 64, 1, 1, 3>(g, plan.groups, st);
        g_launches++;
    } else if (plan.kind == PLAN_T32) {
        launch_tile<32, 128, 1, 2, 4>(g, plan.groups, st);
        g_launches++;
    } else if (plan.kind == PLAN_T128X64) {
        launch_tile<128, 64, 2, 1, 3>(g, plan.groups, st);
        g_launches++;
    } else if (plan.kind == PLAN_PACKED) {
        const size_t nodes = round256(plan.groups > 1 ? (size_t)plan.groups * m * n * 4 : 0);
        if (!ws || !aligned(ws, 256) || (size_t)ws_bytes < packed_need(m, n, k, plan.groups))
            return fail(err, err_cap, "identical gemm: the packed plan needs a 256-byte aligned workspace of %lld bytes, %lld given",
                        (long long)packed_need(m, n, k, plan.groups), (long long)ws_bytes);
        g_launches += launch_packed(g, plan.groups, static_cast<unsigned char *>(ws) + nodes, st);
    } else if (plan.kind == PLAN_SKINNY) {
        if (!skinny_plan_fits(m, n, k, op) || !aligned(b, 16) || !aligned(a, 16))
            return fail(err, err_cap, "identical gemm: the skinny plan needs op NT, m <= 32, k a multiple of 16 and 16-byte aligned operands");
        // low-bit weights stay in registers; float32 windows are too wide for that and go through shared memory
        if (g.wkind != W_F32) launch_skinny_reg(g, plan.groups, sm_count(dev), st);
        else launch_skinny(g, plan.groups, st);
        g_launches++;
    } else {
        return fail(err, err_cap, "identical gemm: unknown plan %d", plan.kind);
    }
    timing_end(tslot, st);
    if (plan.groups > 1 && leave_nodes && n % 4 == 0 && aligned(ws, 16)) {
        *leave_nodes = plan.groups;
    } else if (plan.groups > 1) {
        const long long cells = (long long)m * n;
        launch_fold_groups(g.ws, c, cells, plan.groups, st, g.epi, g.n);
        g_launches++;
    } else if (epilogue_on(g.epi) && plan.kind != PLAN_SKINNY && plan.kind != PLAN_DECODE && plan.kind != PLAN_TALL &&
               plan.kind != PLAN_ROWS && plan.kind != PLAN_BAND && plan.kind != PLAN_STREAM) {
        // the tiled, packed and flat plans store plain product words; their epilogue is a pass of its own
        const long long cells = (long long)m * n;
        if (n % 4 == 0 && aligned(c, 16))
            epilogue_rows4_kernel<<<dim3((unsigned)((n / 4 + 255) / 256), (unsigned)std::min<int64_t>(m, 65535)), 256, 0, st>>>(c, (int)m, (int)n, g.epi);
        else epilogue_rows_kernel<<<grid_for(cells, 256, sm_count(dev)), 256, 0, st>>>(c, cells, (int)n, g.epi);
        g_launches++;
    }
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// Grow-only per-device scratch for the host-pointer twins.
constexpr int HOST_CHUNKS = 8; // row chunks of a pipelined host-pointer product
struct HostPool {
    void *buf[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    size_t cap[6] = {0, 0, 0, 0, 0, 0};
    HostStage stage;                                    // pinned pieces for pageable arrays (host_copy.cuh)
    cudaStream_t stream = nullptr;                      // compute (and the only stream of the unpipelined twins)
    cudaStream_t s_in = nullptr, s_out = nullptr;       // host-to-device and device-to-host copies of the pipelined product
    cudaEvent_t ev[1 + 2 * HOST_CHUNKS] = {};           // weight landed; chunk landed / chunk computed
    bool pipe_ready = false;
};
HostPool g_pool[64];
std::mutex g_pool_mu;

cudaError_t pool_get(int dev, int slot, size_t bytes, void **out) {
    HostPool &p = g_pool[dev];
    if (p.cap[slot] < bytes) {
        if (p.buf[slot]) cudaFree(p.buf[slot]);
        p.buf[slot] = nullptr;
        p.cap[slot] = 0;
        size_t want = bytes + (bytes >> 3) + 256;
        cudaError_t e = cudaMalloc(&p.buf[slot], want);
        if (e != cudaSuccess) return e;
        p.cap[slot] = want;
    }
    *out = p.buf[slot];
    return cudaSuccess;
}

size_t wkind_elem_bytes(int wkind) { return wkind == W_F32 ? 4 : (wkind == W_BF16 ? 2 : 1); }

} // namespace


extern "C" {

int64_t b200i_abi(void) { return 1; }
int64_t b200i_numeric_mode(void) { return 1; }
int64_t b200i_profile_version(void) { return 1; }
int64_t b200i_lowbit_profile_version(void) { return 1; }
const char *b200i_numerical_profile(void) { return "mojolearn.identical.gemm.fp32.v1"; }
const char *b200i_vendor(void) { return "cuda"; }
int64_t b200i_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n;
}
int64_t b200i_launch_count(void) { return g_launches.load(); }
int64_t b200i_decode_plan_fits(int64_t m, int64_t n, int64_t k, int64_t op, int64_t wkind) {
    return decode_plan_fits(m, n, k, (int)op, (int)wkind) ? 1 : 0;
}

int64_t b200i_decode_status(int64_t device) {
    if (device >= 0 && cudaSetDevice((int)device) != cudaSuccess) { cudaGetLastError(); return -1; }
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_decode_status, sizeof(int)) != cudaSuccess) { cudaGetLastError(); return -1; }
    if (v != 0 && cudaMemcpyToSymbol(g_decode_status, &zero, sizeof(int)) != cudaSuccess) { cudaGetLastError(); return -1; }
    return v;
}

int64_t b200i_debug_set_status(int64_t device, int64_t value) {
    if (device >= 0 && cudaSetDevice((int)device) != cudaSuccess) { cudaGetLastError(); return -1; }
    const int v = (int)value;
    if (cudaMemcpyToSymbol(g_decode_status, &v, sizeof(int)) != cudaSuccess) { cudaGetLastError(); return -1; }
    return 0;
}

int64_t b200i_workspace_bytes(int64_t m, int64_t n, int64_t k) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); dev = -1; }
    Plan p = choose_plan(m, n, k, sm_count(dev));
    int groups = p.groups;
    if (tall_candidate(m, n, k) && (int)leaf_count(k) > groups) groups = (int)leaf_count(k);
    if (packed_candidate(p.kind, m, n, k))
        return (int64_t)packed_need(m, n, k, packed_split(p, m, n, k, sm_count(dev)).groups);
    if (skinny_plan_fits(m, n, k, OP_NT)) { // the plan an NT product with aligned operands takes instead
        for (int lowbit = 0; lowbit < 2; lowbit++) {
            const Plan q = choose_skinny(m, n, k, sm_count(dev), lowbit != 0);
            if (q.groups > groups) groups = q.groups;
        }
        if (rows_plan_fits(m, n, k, OP_NT)) groups = std::max(groups, choose_rows(k).groups);
        groups = std::max(groups, choose_band(m, n, k, sm_count(dev)).groups);
        for (const int wkind : {W_F32, W_BF16}) {
            const Plan q = choose_auto(AutoCall{m, n, k, OP_NT, wkind, sm_count(dev), true, false, false, true}, [](const Plan &) { return true; });
            if (q.kind == PLAN_STREAM) groups = std::max(groups, q.groups);
        }
    }
    return groups > 1 ? (int64_t)groups * m * n * 4 : 0;
}

int64_t b200i_product_workspace_bytes(int64_t m, int64_t n, int64_t k, int64_t op, int64_t wkind) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); dev = -1; }
    size_t most = 0; // of what the choice comes to over operand alignments, stores and tensor maps, and of what it falls back to
    for (const bool al16 : {true, false})
        for (const bool pairs : {false, true})
            for (const bool all : {true, false})
                for (const bool maps : {true, false})
                    most = std::max(most, plan_need(choose_auto(AutoCall{m, n, k, (int)op, (int)wkind, sm_count(dev), al16, pairs, false, maps},
                                                                [&](const Plan &p) { return all || p.kind == PLAN_PACKED; }), m, n, k));
    return (int64_t)most;
}

int64_t b200i_kernel_timing(int64_t enable) {
    std::lock_guard<std::mutex> lock(g_timing_mu);
    g_timing.on = enable != 0;
    if (enable) g_timing.used = 0;
    return 0;
}

int64_t b200i_kernel_timing_read(double *total_ms, int64_t *launches) {
    std::lock_guard<std::mutex> lock(g_timing_mu);
    double sum = 0.0;
    for (int i = 0; i < g_timing.used; i++) {
        float ms = 0.f;
        if (cudaEventSynchronize(g_timing.ev[2 * i + 1]) != cudaSuccess ||
            cudaEventElapsedTime(&ms, g_timing.ev[2 * i], g_timing.ev[2 * i + 1]) != cudaSuccess) {
            cudaGetLastError();
            return 1;
        }
        sum += ms;
    }
    if (total_ms) *total_ms = sum;
    if (launches) *launches = g_timing.used;
    g_timing.used = 0;
    return 0;
}

int64_t b200i_plan_workspace_bytes(int64_t m, int64_t n, int64_t k, int64_t plan, int64_t group_leaves) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    if (plan == PLAN_AUTO) return b200i_workspace_bytes(m, n, k);
    const int64_t leaves = leaf_count(k);
    int64_t s = group_leaves > 0 ? group_leaves : leaves;
    if (s > leaves) s = leaves;
    const int64_t groups = (plan == PLAN_FLAT || plan == PLAN_DECODE) ? 1 : (leaves + s - 1) / s;
    if (plan == PLAN_PACKED) return (int64_t)packed_need(m, n, k, (int)groups);
    if (plan == PLAN_TALL) return (int64_t)tall_workspace_bytes(m, n, k);
    return groups > 1 ? groups * m * n * 4 : 0;
}

int64_t b200i_auto_plan(int64_t m, int64_t n, int64_t k, int64_t op, int64_t wkind, int64_t sms, int64_t ws_bytes, int64_t *group_leaves) {
    if (m <= 0 || n <= 0 || k <= 0 || sms <= 0) return -1;
    const Plan p = choose_auto(AutoCall{m, n, k, (int)op, (int)wkind, (int)sms, true, false, false, true},
                               [&](const Plan &q) { return ws_bytes < 0 || (int64_t)plan_need(q, m, n, k) <= ws_bytes; });
    if (group_leaves) *group_leaves = p.group_leaves;
    return p.kind;
}

int64_t b200i_rows_plan_stages(int64_t m, int64_t n, int64_t k, int64_t wkind, int64_t group_leaves, int64_t sms, int64_t *smem_bytes) {
    RowsLaunch r;
    if (m <= 0 || n <= 0 || k <= 0 || sms <= 0 || !rows_plan_fits(m, n, k, OP_NT) ||
        !rows_layout(m, n, k, (int)wkind, group_leaves > 0 ? (int)group_leaves : (int)leaf_count(k), (int)sms, r))
        return 0;
    if (smem_bytes) *smem_bytes = r.smem;
    return r.p.stages;
}

int64_t b200i_pair_epilogue_fits(int64_t m, int64_t n, int64_t k, int64_t op) {
    return (skinny_plan_fits(m, n, k, (int)op) && n % 4 == 0) ? 1 : 0;
}

int64_t b200i_gemm_w_plan(int64_t device, void *stream, float *c, const float *a, const void *b, const void *bscale,
                          int64_t wkind, int64_t m, int64_t n, int64_t k, int64_t op, int64_t plan, int64_t group_leaves,
                          void *ws, int64_t ws_bytes, char *err, int64_t err_cap) {
    clear(err, err_cap);
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    return launch_product(dev, static_cast<cudaStream_t>(stream), c, a, b, bscale, (int)wkind, m, n, k, (int)op, (int)plan,
                          group_leaves, ws, ws_bytes, err, err_cap);
}

int64_t b200i_gemm_w(int64_t device, void *stream, float *c, const float *a, const void *b, const void *bscale,
                     int64_t wkind, int64_t m, int64_t n, int64_t k, int64_t op, void *ws, int64_t ws_bytes, char *err,
                     int64_t err_cap) {
    return b200i_gemm_w_plan(device, stream, c, a, b, bscale, wkind, m, n, k, op, PLAN_AUTO, 0, ws, ws_bytes, err, err_cap);
}

int64_t b200i_gemm_f32(int64_t device, void *stream, float *c, const float *a, const float *b, int64_t m, int64_t n,
                       int64_t k, int64_t op, void *ws, int64_t ws_bytes, char *err, int64_t err_cap) {
    return b200i_gemm_w_plan(device, stream, c, a, b, nullptr, W_F32, m, n, k, op, PLAN_AUTO, 0, ws, ws_bytes, err, err_cap);
}

int64_t b200i_gemm_w_epilogue(int64_t device, void *stream, float *c, const float *a, const void *b, const void *bscale, int64_t wkind,
                              int64_t m, int64_t n, int64_t k, int64_t op, const float *bias, int64_t act, int64_t plan,
                              int64_t group_leaves, void *ws, int64_t ws_bytes, char *err, int64_t err_cap) {
    clear(err, err_cap);
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    if (act < EPI_ACT_NONE || act > EPI_PAIR_GEGLU_TANH) return fail(err, err_cap, "identical gemm: unknown store activation %lld", (long long)act);
    if (bias && !aligned(bias, 4)) return fail(err, err_cap, "identical gemm: misaligned storage");
    return launch_product(dev, static_cast<cudaStream_t>(stream), c, a, b, bscale, (int)wkind, m, n, k, (int)op, (int)plan, group_leaves, ws,
                          ws_bytes, err, err_cap, Epilogue{bias, (int)act});
}

int64_t b200i_gemm_w_nodes(int64_t device, void *stream, float *c, const float *a, const void *b, const void *bscale, int64_t wkind,
                           int64_t m, int64_t n, int64_t k, int64_t op, const float *bias, int64_t act, void *ws, int64_t ws_bytes,
                           int64_t *nodes, char *err, int64_t err_cap) {
    clear(err, err_cap);
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    if (!nodes) return fail(err, err_cap, "identical gemm: nowhere to report the node count");
    if (act < EPI_ACT_NONE || act > EPI_PAIR_GEGLU_TANH) return fail(err, err_cap, "identical gemm: unknown store activation %lld", (long long)act);
    if (bias && !aligned(bias, 4)) return fail(err, err_cap, "identical gemm: misaligned storage");
    return launch_product(dev, static_cast<cudaStream_t>(stream), c, a, b, bscale, (int)wkind, m, n, k, (int)op, PLAN_AUTO, 0, ws, ws_bytes, err,
                          err_cap, Epilogue{bias, (int)act}, nodes);
}

int64_t b200i_to_bf16(int64_t device, void *stream, uint16_t *dst, const float *src, int64_t count, char *err,
                      int64_t err_cap) {
    clear(err, err_cap);
    if (count < 0 || (count > 0 && (!dst || !src))) return fail(err, err_cap, "to_bf16: null storage or negative count");
    if (count == 0) return 0;
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    to_bf16_kernel<<<grid_for((count + 3) / 4, 256, sm_count(dev)), 256, 0, static_cast<cudaStream_t>(stream)>>>(dst, src, count);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_from_bf16(int64_t device, void *stream, float *dst, const uint16_t *src, int64_t count, char *err,
                        int64_t err_cap) {
    clear(err, err_cap);
    if (count < 0 || (count > 0 && (!dst || !src))) return fail(err, err_cap, "from_bf16: null storage or negative count");
    if (count == 0) return 0;
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    from_bf16_kernel<<<grid_for((count + 3) / 4, 256, sm_count(dev)), 256, 0, static_cast<cudaStream_t>(stream)>>>(dst, src, count);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_quantize_int8(int64_t device, void *stream, int8_t *codes, int32_t *exponents, const float *x, int64_t rows,
                            int64_t cols, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "quantize_int8: rows and cols must be positive");
    if (!codes || !exponents || !x) return fail(err, err_cap, "quantize_int8: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    launch_quantize_int8(reinterpret_cast<signed char *>(codes), exponents, x, rows, cols, sm_count(dev), static_cast<cudaStream_t>(stream));
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_dequantize_int8(int64_t device, void *stream, float *y, const int8_t *codes, const int32_t *exponents,
                              int64_t rows, int64_t cols, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "dequantize_int8: rows and cols must be positive");
    if (!codes || !exponents || !y) return fail(err, err_cap, "dequantize_int8: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    dequantize_int8_kernel<<<grid_for(rows * cols, 256, sm_count(dev)), 256, 0, static_cast<cudaStream_t>(stream)>>>(y, reinterpret_cast<const signed char *>(codes), exponents, rows, cols);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_gemm_int8(int64_t device, void *stream, float *c, const int8_t *qa, const int32_t *ea, const int8_t *qb,
                        const int32_t *eb, int64_t m, int64_t n, int64_t k, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (m <= 0 || n <= 0 || k <= 0) return fail(err, err_cap, "identical int8 gemm: m, n and k must be positive");
    if (k > 131072) return fail(err, err_cap, "identical int8 gemm: k = %lld exceeds INT8_MAX_K = 131072", (long long)k);
    if (!c || !qa || !ea || !qb || !eb) return fail(err, err_cap, "identical int8 gemm: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    const long long cells = m * n;
    // the tensor-core kernels wherever their 16-byte copies are aligned (k a multiple of 16) and tensor maps can be made; one
    // thread per cell otherwise
    const signed char *sa = reinterpret_cast<const signed char *>(qa), *sb = reinterpret_cast<const signed char *>(qb);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    bool launched = false;
    if (gemm_int8_mma_fits(qa, qb, k)) {
        const int sms = sm_count(dev);
        // SM pairs at every size (1024 x 4096 x 4096 in 23 us, 4096^3 60 against 62 for one CTA per tile), except where the
        // contraction is so short that the store is all there is and the one-CTA kernel's wider spread of it wins
        // (2048 x 50304 x 768: 157 against 174 us)
        const long long wide = ((m + T8_BM - 1) / T8_BM) * ((n + T8_BN - 1) / T8_BN);
        const bool single = wide >= 4ll * sms && k < 1024;
        launched = (!single && launch_gemm_int8_pair(c, sa, ea, sb, eb, (int)m, (int)n, (int)k, st)) ||
                   launch_gemm_int8_tma(c, sa, ea, sb, eb, (int)m, (int)n, (int)k, sms, st);
    }
    if (!launched) gemm_int8_flat_kernel<<<(unsigned)((cells + 127) / 128), 128, 0, st>>>(c, sa, ea, sb, eb, (int)m, (int)n, (int)k);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_quantize_int15(int64_t device, void *stream, int8_t *hi, int8_t *lo, int32_t *exponents, const float *x, int64_t rows,
                             int64_t cols, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "quantize_int15: rows and cols must be positive");
    if (!hi || !lo || !exponents || !x) return fail(err, err_cap, "quantize_int15: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    quantize_int15_kernel<<<grid_for(rows * 32, 256, sm_count(dev)), 256, 0, static_cast<cudaStream_t>(stream)>>>(reinterpret_cast<signed char *>(hi), reinterpret_cast<signed char *>(lo), exponents, x, rows, cols);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_dequantize_int15(int64_t device, void *stream, float *y, const int8_t *hi, const int8_t *lo, const int32_t *exponents,
                               int64_t rows, int64_t cols, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "dequantize_int15: rows and cols must be positive");
    if (!hi || !lo || !exponents || !y) return fail(err, err_cap, "dequantize_int15: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    dequantize_int15_kernel<<<grid_for(rows * cols, 256, sm_count(dev)), 256, 0, static_cast<cudaStream_t>(stream)>>>(y, reinterpret_cast<const signed char *>(hi), reinterpret_cast<const signed char *>(lo), exponents, rows, cols);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_gemm_int15(int64_t device, void *stream, float *c, const int8_t *ah, const int8_t *al, const int32_t *ea, const int8_t *bh,
                         const int8_t *bl, const int32_t *eb, int64_t m, int64_t n, int64_t k, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (m <= 0 || n <= 0 || k <= 0) return fail(err, err_cap, "identical int15 gemm: m, n and k must be positive");
    if (k > INT15_MAX_K) return fail(err, err_cap, "identical int15 gemm: k = %lld exceeds INT15_MAX_K = 65536", (long long)k);
    if (!c || !ah || !al || !ea || !bh || !bl || !eb) return fail(err, err_cap, "identical int15 gemm: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    const signed char *sah = reinterpret_cast<const signed char *>(ah), *sal = reinterpret_cast<const signed char *>(al);
    const signed char *sbh = reinterpret_cast<const signed char *>(bh), *sbl = reinterpret_cast<const signed char *>(bl);
    // the tensor-core plan wherever its 16-byte copies are aligned (k a multiple of 16); one thread per cell otherwise
    if (gemm_int15_mma_fits(ah, al, bh, bl, m, n, k)) {
        // enough 128 x 64 tiles for every SM: the persistent kernel fed by tensor-map copies; else the per-tile kernel
        const int sms = sm_count(dev);
        const long long tiles = ((m + T8_BM - 1) / T8_BM) * ((n + I15_TN - 1) / I15_TN);
        if (tiles < 2ll * sms || !launch_gemm_int15_tma(c, sah, sal, ea, sbh, sbl, eb, (int)m, (int)n, (int)k, sms, static_cast<cudaStream_t>(stream)))
            launch_gemm_int15_mma(c, sah, sal, ea, sbh, sbl, eb, (int)m, (int)n, (int)k, static_cast<cudaStream_t>(stream));
    }
    else
        gemm_int15_flat_kernel<<<(unsigned)((m * n + 127) / 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(c, sah, sal, ea, sbh, sbl, eb, (int)m, (int)n, (int)k);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_ffma_probe(int64_t device, void *stream, float *scratch, int64_t blocks, int64_t iters, int64_t packed,
                         char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (!scratch || blocks <= 0 || iters <= 0) return fail(err, err_cap, "ffma_probe: bad arguments");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    ffma_probe_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(scratch, (int)iters, (int)packed, 1.0f);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// ---- the product without any allocation ---------------------------------------------------------
// Scratch for the split plan lives in the library image itself: a fixed device array
// that every GPU loading the library carries until the process exits.
constexpr size_t STATIC_SCRATCH_BYTES = 16u << 20;
static __device__ __align__(256) unsigned char g_static_scratch[STATIC_SCRATCH_BYTES];
static void *g_static_scratch_ptr[MAX_DEVICES]; // per device: the array's DEVICE address (the symbol itself is only a host-side stand-in)
static std::mutex g_static_scratch_mu;

// The plan the allocation-free entry runs: the tile plan the cost model prefers when its leaf-group nodes fit the
// built-in scratch, else the same tiles with the leaves split into fewer, larger groups (powers of two, so every
// group is still a subtree of the contract's fold), down to no split at all, which needs no scratch. The bits do
// not depend on the split; only the number of CTAs does.
static Plan noalloc_plan(int64_t m, int64_t n, int64_t k, int sms) {
    Plan plan = choose_plan(m, n, k, sms);
    const int leaves = (int)leaf_count(k) > 0 ? (int)leaf_count(k) : 1;
    while (plan.groups > 1 && (int64_t)plan.groups * m * n * 4 > (int64_t)STATIC_SCRATCH_BYTES) {
        plan.group_leaves *= 2;
        plan.groups = (leaves + plan.group_leaves - 1) / plan.group_leaves;
    }
    if (plan.groups <= 1) { plan.groups = 1; plan.group_leaves = leaves; }
    return plan;
}

int64_t b200i_noalloc_scratch_bytes(int64_t m, int64_t n, int64_t k) {
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); dev = -1; }
    const Plan plan = noalloc_plan(m, n, k, sm_count(dev));
    return plan.groups > 1 ? (int64_t)plan.groups * m * n * 4 : 0;
}

int64_t b200i_gemm_f32_noalloc(int64_t device, void *stream, float *c, const float *a, const float *b, int64_t m, int64_t n,
                               int64_t k, int64_t op, char *err, int64_t err_cap) {
    clear(err, err_cap);
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    void *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_scratch_mu);
        if (!g_static_scratch_ptr[dev]) {
            // once per device, with that device current: ask the runtime where the array lives on it
            void *p = nullptr;
            CUDA_TRY(cudaGetSymbolAddress(&p, g_static_scratch));
            g_static_scratch_ptr[dev] = p;
        }
        scratch = g_static_scratch_ptr[dev];
    }
    if (m <= 0 || n <= 0 || k <= 0)
        return fail(err, err_cap, "identical gemm: m, n and k must be positive (got m=%lld n=%lld k=%lld)", (long long)m,
                    (long long)n, (long long)k);
    const Plan plan = noalloc_plan(m, n, k, sm_count(dev));
    const int64_t need = plan.groups > 1 ? (int64_t)plan.groups * m * n * 4 : 0;
    if (need > (int64_t)STATIC_SCRATCH_BYTES) // cannot happen while an unsplit plan needs no scratch; kept as the guard of that assumption
        return fail(err, err_cap,
                    "identical gemm: this shape needs %lld bytes of scratch and the built-in scratch holds %lld; "
                    "call b200i_gemm_f32 with scratch of b200i_workspace_bytes(m, n, k) bytes instead",
                    (long long)need, (long long)STATIC_SCRATCH_BYTES);
    t_no_timing = true; // the benchmark's event pairs are created on demand, which may allocate
    const int64_t rc = launch_product(dev, static_cast<cudaStream_t>(stream), c, a, b, nullptr, W_F32, m, n, k, (int)op, plan.kind,
                                      plan.groups > 1 ? plan.group_leaves : 0, scratch, (int64_t)STATIC_SCRATCH_BYTES, err, err_cap);
    t_no_timing = false;
    return rc;
}

// ---- decoder-block seams (device pointers, asynchronous on the caller's stream) ----------------

#define SEAM_PROLOGUE()                                          \
    clear(err, err_cap);                                         \
    int dev;                                                     \
    if (select_device(device, err, err_cap, &dev)) return 1;     \
    cudaStream_t st = static_cast<cudaStream_t>(stream)

// A CTA of four warps per row while that leaves at most two on an SM (a decode step), else a warp per row.
static cudaError_t launch_norm_rows(int dev, cudaStream_t st, float *out, const float *x, const float *w, const float *bias, int64_t rows, int width, float eps,
                                    int kind, const float *delta, float *sum_out, int wpc, size_t smem) {
    static std::atomic<bool> configured[64];
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(norm_rows_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(norm_rows_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    if (rows <= 2 * sm_count(dev)) norm_rows_kernel<4><<<(unsigned)rows, 128, smem, st>>>(out, x, w, bias, rows, width, eps, kind, delta, sum_out);
    else norm_rows_kernel<1><<<(unsigned)((rows + wpc - 1) / wpc), 32 * wpc, smem, st>>>(out, x, w, bias, rows, width, eps, kind, delta, sum_out);
    return cudaSuccess;
}

int64_t b200i_norm(int64_t device, void *stream, float *out, const float *x, const float *w, const float *bias, int64_t rows,
                   int64_t width, double eps, int64_t kind, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rows <= 0 || width <= 0 || !out || !x || !w) return fail(err, err_cap, "norm: bad arguments");
    if (kind < NORM_RMS || kind > NORM_RMS_OFFSET) return fail(err, err_cap, "norm: norm kind %lld is not spelled", (long long)kind);
    if (bias && kind != NORM_LAYER) return fail(err, err_cap, "norm: an RMSNorm carries no bias (norm_bias needs layernorm)");
    const int wpc = rows >= 1024 ? 4 : 1; // rows per CTA: few rows spread over the SMs
    const size_t smem = (size_t)wpc * (size_t)((width + 3) & ~3ll) * sizeof(float);
    if (smem <= 200 * 1024) {
        CUDA_TRY(launch_norm_rows(dev, st, out, x, w, bias, rows, (int)width, (float)eps, (int)kind, nullptr, nullptr, wpc, smem));
    } else {
        const long long threads = rows * 32;
        norm_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(out, x, w, bias, rows, (int)width, (float)eps, (int)kind);
    }
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_add_norm(int64_t device, void *stream, float *out, float *sum_out, const float *x, const float *delta, const float *w,
                       const float *bias, int64_t rows, int64_t width, double eps, int64_t kind, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rows <= 0 || width <= 0 || !out || !sum_out || !x || !delta || !w) return fail(err, err_cap, "add_norm: bad arguments");
    if (kind < NORM_RMS || kind > NORM_RMS_OFFSET) return fail(err, err_cap, "norm: norm kind %lld is not spelled", (long long)kind);
    if (bias && kind != NORM_LAYER) return fail(err, err_cap, "norm: an RMSNorm carries no bias (norm_bias needs layernorm)");
    const int wpc = rows >= 1024 ? 4 : 1;
    const size_t smem = (size_t)wpc * (size_t)((width + 3) & ~3ll) * sizeof(float);
    if (smem <= 200 * 1024) {
        CUDA_TRY(launch_norm_rows(dev, st, out, x, w, bias, rows, (int)width, (float)eps, (int)kind, delta, sum_out, wpc, smem));
        g_launches++;
    } else { // a row too wide for shared memory: the two seams one after the other
        const long long count = rows * width;
        add_kernel<<<grid_for(count, 256, sm_count(dev)), 256, 0, st>>>(sum_out, x, delta, count);
        norm_kernel<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, st>>>(out, sum_out, w, bias, rows, (int)width, (float)eps, (int)kind);
        g_launches += 2;
    }
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_qkv_rope_cache(int64_t device, void *stream, float *qr, float *kcache, float *vcache, const float *q, const float *k,
                             const float *v, int64_t src_ld, const float *cosv, const float *sinv, int64_t b, int64_t l,
                             int64_t n_heads, int64_t n_kv, int64_t head_dim, int64_t cap, int64_t pos0, const int32_t *position,
                             int64_t rope_dim, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rope_dim == 0) rope_dim = head_dim;
    if (rope_dim < 0 || rope_dim > head_dim || (rope_dim & 1))
        return fail(err, err_cap, "transformer: the rotary table's rope_dim %lld does not fit head_dim %lld REFUSED", (long long)rope_dim, (long long)head_dim);
    if (b <= 0 || l <= 0 || n_heads <= 0 || n_kv <= 0 || head_dim <= 0 || (head_dim & 1) || !qr || !kcache || !vcache || !q || !k || !v ||
        qr == q)
        return fail(err, err_cap, "qkv_rope_cache: bad arguments");
    if ((cosv == nullptr) != (sinv == nullptr)) return fail(err, err_cap, "qkv_rope_cache: give both tables or neither");
    if (!position) {
        if (pos0 < 0) return fail(err, err_cap, "qkv_rope_cache: bad arguments");
        if (pos0 + l > cap)
            return fail(err, err_cap, "transformer: this call would use %lld KV slots and the cache holds %lld REFUSED", (long long)(pos0 + l),
                        (long long)cap);
    } else if (l > cap) {
        return fail(err, err_cap, "qkv_rope_cache: bad arguments");
    }
    const long long total = b * l * (n_heads + 2 * n_kv) * head_dim;
    const long long ldq = src_ld ? src_ld : n_heads * head_dim, ldkv = src_ld ? src_ld : n_kv * head_dim;
    if (ldq < n_heads * head_dim || ldkv < n_kv * head_dim) return fail(err, err_cap, "qkv_rope_cache: the row pitch is below the row width");
    const bool quads = (cosv ? (rope_dim == head_dim && head_dim % 8 == 0) : head_dim % 4 == 0) && ldq % 4 == 0 && ldkv % 4 == 0 && aligned(qr, 16) &&
                       aligned(kcache, 16) && aligned(vcache, 16) && aligned(q, 16) && aligned(k, 16) && aligned(v, 16) &&
                       (!cosv || (aligned(cosv, 16) && aligned(sinv, 16)));
    if (quads) {
        const int64_t per_head = cosv ? head_dim / 8 : head_dim / 4, units = (n_heads + n_kv) * per_head + n_kv * (head_dim / 4);
        const QkvArgs g{qr, kcache, vcache, q, k, v, cosv, sinv, ldq, ldkv, b * l, (int)l, (int)n_heads, (int)n_kv, (int)head_dim, (int)cap, (int)pos0,
                        cosv ? 1 : 0, position};
        const int threads = units >= 256 ? 256 : 128;
        qkv_rope_cache4_kernel<<<dim3((unsigned)((units + threads - 1) / threads), (unsigned)std::min<int64_t>(b * l, 65535)), threads, 0, st>>>(g);
    } else
        qkv_rope_cache_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(qr, kcache, vcache, q, k, v, ldq, ldkv, cosv, sinv, (int)b, (int)l,
                                                                           (int)n_heads, (int)n_kv, (int)head_dim, (int)cap, (int)pos0,
                                                                           position, cosv ? 1 : 0, (int)rope_dim);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_rope_table(int64_t device, void *stream, float *cosv, float *sinv, int64_t pos0, int64_t l, int64_t head_dim,
                         double theta, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (l <= 0 || head_dim <= 0 || (head_dim & 1) || !cosv || !sinv) return fail(err, err_cap, "rope_table: bad arguments");
    if (pos0 < 0 || pos0 + l > 8192)
        return fail(err, err_cap, "rope_table: absolute position %lld is at or beyond 8192, the domain of the sine and cosine reduction",
                    (long long)(pos0 + l - 1));
    const long long n = l * (head_dim / 2);
    rope_table_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(cosv, sinv, (int)pos0, (int)l, (int)head_dim, (float)theta, nullptr);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_rope_table_at(int64_t device, void *stream, float *cosv, float *sinv, const int32_t *position, int64_t l,
                            int64_t head_dim, double theta, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (l <= 0 || head_dim <= 0 || (head_dim & 1) || !cosv || !sinv || !position) return fail(err, err_cap, "rope_table: bad arguments");
    const long long n = l * (head_dim / 2);
    rope_table_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(cosv, sinv, 0, (int)l, (int)head_dim, (float)theta, position);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_rope_table_opts(int64_t device, void *stream, float *cosv, float *sinv, int64_t pos0, const int32_t *position, int64_t l,
                              int64_t rope_dim, double theta, int64_t scaling, double factor, double low_freq_factor,
                              double high_freq_factor, int64_t original_max_positions, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (l <= 0 || rope_dim <= 0 || (rope_dim & 1) || !cosv || !sinv) return fail(err, err_cap, "rope_table: bad arguments");
    if (scaling < 0 || scaling > 2) return fail(err, err_cap, "transformer options: rope_scaling %lld is not spelled", (long long)scaling);
    if (!(theta > 0.0) || (scaling != 0 && !(factor > 0.0))) return fail(err, err_cap, "transformer options: rope_theta and the rope_scaling factor must be positive");
    if (scaling == 2 && (!(low_freq_factor > 0.0) || !(high_freq_factor > 0.0) || high_freq_factor == low_freq_factor || original_max_positions <= 0))
        return fail(err, err_cap, "transformer options: llama3 rope_scaling needs positive, distinct frequency factors and original positions");
    if (!position && (pos0 < 0 || pos0 + l > 8192 * (scaling == 1 ? (long long)factor : 1)))
        return fail(err, err_cap, "rope_table: absolute position %lld puts the angle at or beyond 8192, the domain of the sine and cosine reduction",
                    (long long)(pos0 + l - 1));
    const long long n = l * (rope_dim / 2);
    RopeOptions o{(float)theta, (int)scaling, (float)factor, (float)low_freq_factor, (float)high_freq_factor, (int)original_max_positions};
    rope_table_opts_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(cosv, sinv, (int)pos0, (int)l, (int)rope_dim, o, position);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_rope_apply(int64_t device, void *stream, float *out, const float *src, const float *cosv, const float *sinv,
                         int64_t rows, int64_t l, int64_t n_heads, int64_t head_dim, int64_t src_ld, int64_t rope_dim, char *err,
                         int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rope_dim == 0) rope_dim = head_dim;
    if (rope_dim < 0 || rope_dim > head_dim || (rope_dim & 1))
        return fail(err, err_cap, "transformer: the rotary table's rope_dim %lld does not fit head_dim %lld REFUSED", (long long)rope_dim, (long long)head_dim);
    if (rows <= 0 || l <= 0 || n_heads <= 0 || head_dim <= 0 || (head_dim & 1) || !out || !src || out == src)
        return fail(err, err_cap, "rope_apply: bad arguments (the rotation is not in place)");
    if (src_ld == 0) src_ld = n_heads * head_dim;
    if (src_ld < n_heads * head_dim) return fail(err, err_cap, "rope_apply: the row pitch is below the row width");
    const long long n = rows * n_heads * head_dim;
    rope_apply_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, src, cosv, sinv, rows, (int)l, (int)n_heads, (int)head_dim, src_ld, (int)rope_dim);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_kv_append(int64_t device, void *stream, float *cache, const float *src, int64_t b, int64_t l, int64_t n_kv,
                        int64_t head_dim, int64_t cap, int64_t pos0, int64_t src_ld, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (src_ld == 0) src_ld = n_kv * head_dim;
    if (b <= 0 || l <= 0 || n_kv <= 0 || head_dim <= 0 || pos0 < 0 || !cache || !src || src_ld < n_kv * head_dim)
        return fail(err, err_cap, "kv_append: bad arguments");
    if (pos0 + l > cap)
        return fail(err, err_cap, "transformer: this call would use %lld KV slots and the cache holds %lld REFUSED", (long long)(pos0 + l),
                    (long long)cap);
    const long long n = b * l * n_kv * head_dim;
    kv_append_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(cache, src, (int)b, (int)l, (int)n_kv, (int)head_dim, (int)cap, (int)pos0,
                                                                  nullptr, src_ld);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_kv_append_at(int64_t device, void *stream, float *cache, const float *src, int64_t b, int64_t l, int64_t n_kv,
                           int64_t head_dim, int64_t cap, const int32_t *position, int64_t src_ld, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (src_ld == 0) src_ld = n_kv * head_dim;
    if (b <= 0 || l <= 0 || n_kv <= 0 || head_dim <= 0 || l > cap || !cache || !src || !position || src_ld < n_kv * head_dim)
        return fail(err, err_cap, "kv_append: bad arguments");
    const long long n = b * l * n_kv * head_dim;
    kv_append_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(cache, src, (int)b, (int)l, (int)n_kv, (int)head_dim, (int)cap, 0, position,
                                                                  src_ld);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// `s_grid` sizes the launch (the key count, or its upper bound when the position is read on the device)
static int64_t attention_launch(int dev, cudaStream_t st, float *ctx, const float *q, const float *kcache, const float *vcache,
                                float *scores, int64_t b, int64_t l, int64_t n_heads, int64_t n_kv, int64_t head_dim, int64_t cap,
                                int key_lo, int s, int own0, int s_grid, int64_t window, const int32_t *position, float softcap,
                                char *err, int64_t err_cap) {
    if (l >= 2 && l <= ATT_SMALL_Q && head_dim % 4 == 0 && head_dim <= K_LEAF_MIN) {
        // A few query rows per sequence (a chunked prompt's tail, speculative steps): scores, softmax and value sum in
        // one kernel, the score rows in shared memory, every key and value row read once for all the query rows. The
        // fewer CTAs the call has, the more shared memory each one spends on bytes in flight. A single query row
        // stays on the two kernels below: measured on B200 (batch 32, 16 heads, 1030 keys) the fused form is 8 %
        // slower on the whole decode step there, because its CTAs run their score, softmax and value phases in step
        // and the memory system idles through everyone's serial softmax, and with few (sequence, head) pairs the
        // scores kernel's split over key tiles is what keeps all SMs loading.
        const int lq = l == 1 ? 1 : (l == 2 ? 2 : (l <= 4 ? 4 : 8));
        const long long ctas = b * n_heads;
        const long long fixed = (long long)lq * K_LEAF_MIN + (long long)lq * ((s_grid + 3) & ~3);
        const long long room = att_cta_bytes(ctas, sm_count(dev), 6) / 4 - fixed; // floats for the key tiles / the value ring
        int kkeys = 32, nkb = (int)(room / (ATD_WARPS * 32 * ATT_KT_PITCH));
        if (nkb > 3) nkb = 3;
        if (nkb < 1) { // not even one full tile per warp: fewer keys per tile
            nkb = 1;
            kkeys = (int)(room / (ATD_WARPS * ATT_KT_PITCH));
        }
        const int vkeys = room >= 4ll * 32 * head_dim ? 32 : 16;
        int stages = (int)(room / (vkeys * head_dim));
        if (stages > ATD_MAX_STAGES) stages = ATD_MAX_STAGES;
        if (kkeys >= 8 && stages >= 2) {
            const size_t smem = attn_decode_smem(lq, s_grid, (int)head_dim, kkeys, nkb, vkeys, stages);
#define DECODE_FUSED(LQ)                                                                                                          \
    do {                                                                                                                          \
        static std::atomic<bool> configured[64];                                                                                  \
        if (dev >= 0 && dev < 64 && !configured[dev]) {                                                                           \
            CUDA_TRY(cudaFuncSetAttribute(attn_decode_kernel<LQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM_LIMIT));  \
            configured[dev] = true;                                                                                               \
        }                                                                                                                         \
        attn_decode_kernel<LQ><<<(unsigned)ctas, ATD_THREADS, smem, st>>>(ctx, q, kcache, vcache, (int)b, (int)l, (int)n_heads,   \
                                                                          (int)n_kv, (int)head_dim, (int)cap, key_lo, s, own0,   \
                                                                          (int)window, position, s_grid, kkeys, nkb, vkeys,      \
                                                                          stages, softcap);                                      \
    } while (0)
            if (lq == 1) DECODE_FUSED(1);
            else if (lq == 2) DECODE_FUSED(2);
            else if (lq == 4) DECODE_FUSED(4);
            else DECODE_FUSED(8);
#undef DECODE_FUSED
            g_launches++;
            CUDA_TRY(cudaGetLastError());
            return 0;
        }
    }
    if (l <= ATT_SMALL_Q) {
        dim3 gs((unsigned)((s_grid + 127) / 128), (unsigned)(b * n_heads));
#define SCORES_SMALL(LQ)                                                                                                          \
    do {                                                                                                                          \
        static std::atomic<bool> configured[64];                                                                                          \
        if (dev >= 0 && dev < 64 && !configured[dev]) {                                                                           \
            CUDA_TRY(cudaFuncSetAttribute(attn_scores_small_kernel<LQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,              \
                                          attn_scores_small_smem<LQ>(K_LEAF_MIN)));                                               \
            configured[dev] = true;                                                                                               \
        }                                                                                                                         \
        attn_scores_small_kernel<LQ><<<gs, 128, attn_scores_small_smem<LQ>((int)head_dim), st>>>(\
            scores, q, kcache, (int)b, (int)l, (int)n_heads, (int)n_kv, (int)head_dim, (int)cap, key_lo, s, own0, (int)window,    \
            position, softcap);                                                                                                   \
    } while (0)
        if (l == 1) SCORES_SMALL(1);
        else if (l == 2) SCORES_SMALL(2);
        else if (l <= 4) SCORES_SMALL(4);
        else SCORES_SMALL(8);
#undef SCORES_SMALL
    } else {
        dim3 g1((unsigned)((s_grid + ATT_T - 1) / ATT_T), (unsigned)((l + ATT_T - 1) / ATT_T), (unsigned)(b * n_heads));
        attn_scores_kernel<<<g1, 256, 0, st>>>(scores, q, kcache, (int)b, (int)l, (int)n_heads, (int)n_kv, (int)head_dim, (int)cap, key_lo, s,
                                                 own0, (int)window, position, softcap);
    }
    if (l <= ATT_SMALL_Q && (size_t)s_grid * sizeof(float) <= 40 * 1024) {
        static std::atomic<bool> configured[64];
        if (dev >= 0 && dev < 64 && !configured[dev]) {
            CUDA_TRY(cudaFuncSetAttribute(attn_context_row_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM_LIMIT));
            CUDA_TRY(cudaFuncSetAttribute(attn_context_row_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM_LIMIT));
            configured[dev] = true;
        }
        // enough CTAs per SM for one wave (four at most); the shared memory that leaves a CTA becomes ring stages
        const long long rows = b * n_heads * l;
        const int stages = attn_context_row_stages(rows, s_grid, (int)head_dim, sm_count(dev));
        const size_t row_smem = attn_context_row_smem(s_grid, (int)head_dim, stages);
        if (rows <= 2ll * sm_count(dev))
            attn_context_row_kernel<256><<<(unsigned)rows, 256, row_smem, st>>>(ctx, scores, vcache, (int)b, (int)l, (int)n_heads, (int)n_kv, (int)head_dim, (int)cap,
                                                                                key_lo, s, own0, (int)window, position, s_grid, stages);
        else
            attn_context_row_kernel<128><<<(unsigned)rows, 128, row_smem, st>>>(ctx, scores, vcache, (int)b, (int)l, (int)n_heads, (int)n_kv, (int)head_dim, (int)cap,
                                                                                key_lo, s, own0, (int)window, position, s_grid, stages);
    } else {
        dim3 g2((unsigned)((l + CTX_ROWS - 1) / CTX_ROWS), (unsigned)(b * n_heads));
#define CONTEXT_ROWS(DPL)                                                                                                     \
    attn_context_kernel<DPL><<<g2, 32 * CTX_WARPS, attn_context_smem((int)head_dim), st>>>(\
        ctx, scores, vcache, (int)b, (int)l, (int)n_heads, (int)n_kv, (int)head_dim, (int)cap, key_lo, s, own0, (int)window, position)
        if (head_dim <= 32) CONTEXT_ROWS(1);
        else if (head_dim <= 64) CONTEXT_ROWS(2);
        else CONTEXT_ROWS(4);
#undef CONTEXT_ROWS
    }
    g_launches += 2;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

static int64_t attention_check(int64_t b, int64_t l, int64_t n_heads, int64_t n_kv, int64_t head_dim, const void *ctx, const void *q,
                               const void *kcache, const void *vcache, const void *scores, char *err, int64_t err_cap) {
    if (b <= 0 || l <= 0 || n_heads <= 0 || n_kv <= 0 || n_heads % n_kv != 0 || head_dim <= 0 || !ctx || !q || !kcache || !vcache || !scores)
        return fail(err, err_cap, "attention: bad arguments");
    if (head_dim > K_LEAF_MIN || head_dim > CTX_MAX_HD)
        return fail(err, err_cap, "attention: head_dim %lld above 128 needs the leaf partition of the product, which this kernel does not spell",
                    (long long)head_dim);
    if (b * n_heads > 65535) return fail(err, err_cap, "attention: batch x heads above 65535");
    return 0;
}

// A prompt's score block [b * heads, l, s] is consumed by the softmax / value kernel right after it is written, so it
// need not exist for the whole batch at once: above ATT_SCRATCH_FLOATS the batch is walked a few sequences at a time
// through one scratch. The bound only caps the scratch (4 GB): walking the serving benchmark's prompt one sequence at a time
// (a 67 MB block that stays in L2 between the two kernels instead of 2 GB through HBM) measured 5.5 % SLOWER on the whole
// prefill (2242 against 2124 ms), because eight launches of 512 value-chain CTAs have eight tails where one launch of 4096
// has one.
constexpr long long ATT_SCRATCH_FLOATS = 1ll << 30;
static int64_t attention_batch_chunk(int64_t b, int64_t l, int64_t n_heads, int64_t s_grid) {
    if (l <= ATT_SMALL_Q) return b;
    const long long per = (long long)n_heads * l * s_grid;
    long long c = per > 0 ? ATT_SCRATCH_FLOATS / per : b;
    if (c < 1) c = 1;
    return c < b ? c : b;
}
static int64_t attention_chunked(int dev, cudaStream_t st, float *ctx, const float *q, const float *kcache, const float *vcache, float *scores,
                                 int64_t b, int64_t l, int64_t n_heads, int64_t n_kv, int64_t head_dim, int64_t cap, int key_lo, int s, int own0,
                                 int s_grid, int64_t window, const int32_t *position, float softcap, char *err, int64_t err_cap) {
    const int64_t step = attention_batch_chunk(b, l, n_heads, s_grid);
    for (int64_t b0 = 0; b0 < b; b0 += step) {
        const int64_t nb = b - b0 < step ? b - b0 : step;
        const size_t qoff = (size_t)b0 * l * n_heads * head_dim, coff = (size_t)b0 * n_kv * cap * head_dim;
        if (attention_launch(dev, st, ctx + qoff, q + qoff, kcache + coff, vcache + coff, scores, nb, l, n_heads, n_kv, head_dim, cap, key_lo, s,
                             own0, s_grid, window, position, softcap, err, err_cap))
            return 1;
    }
    return 0;
}

int64_t b200i_attention_scratch_floats(int64_t b, int64_t l, int64_t n_heads, int64_t s) {
    if (b <= 0 || l <= 0 || n_heads <= 0 || s <= 0) return 0;
    return attention_batch_chunk(b, l, n_heads, s) * n_heads * l * s;
}

int64_t b200i_attention(int64_t device, void *stream, float *ctx, const float *q, const float *kcache, const float *vcache,
                        float *scores, int64_t b, int64_t l, int64_t n_heads, int64_t n_kv, int64_t head_dim, int64_t cap,
                        int64_t used, int64_t window, double softcap, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (attention_check(b, l, n_heads, n_kv, head_dim, ctx, q, kcache, vcache, scores, err, err_cap)) return 1;
    if (used < l || used > cap) return fail(err, err_cap, "attention: the cache holds %lld positions, this call's %lld included", (long long)used, (long long)l);
    const int64_t pos0 = used - l;
    int64_t key_lo = 0;
    if (window > 0 && pos0 - (window - 1) > 0) key_lo = pos0 - (window - 1);
    const int s = (int)(used - key_lo), own0 = (int)(pos0 - key_lo);
    return attention_chunked(dev, st, ctx, q, kcache, vcache, scores, b, l, n_heads, n_kv, head_dim, cap, (int)key_lo, s, own0, s, window,
                             nullptr, (float)softcap, err, err_cap);
}

int64_t b200i_attention_at(int64_t device, void *stream, float *ctx, const float *q, const float *kcache, const float *vcache,
                           float *scores, int64_t b, int64_t l, int64_t n_heads, int64_t n_kv, int64_t head_dim, int64_t cap,
                           const int32_t *position, int64_t window, double softcap, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (attention_check(b, l, n_heads, n_kv, head_dim, ctx, q, kcache, vcache, scores, err, err_cap)) return 1;
    if (!position || l > cap) return fail(err, err_cap, "attention: bad arguments");
    int64_t s_max = cap; // the most keys any position can see
    if (window > 0 && window - 1 + l < s_max) s_max = window - 1 + l;
    return attention_chunked(dev, st, ctx, q, kcache, vcache, scores, b, l, n_heads, n_kv, head_dim, cap, 0, (int)s_max, 0, (int)s_max, window,
                             position, (float)softcap, err, err_cap);
}

int64_t b200i_act_mul(int64_t device, void *stream, float *out, const float *gate, const float *up, int64_t rows, int64_t width,
                      int64_t in_ld, int64_t kind, int64_t interleaved, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    const bool gated = kind == ACT_SWIGLU || kind == ACT_GEGLU_ERF || kind == ACT_GEGLU_TANH;
    if (interleaved) {
        if (!gated || !gate) return fail(err, err_cap, "act_mul: the interleaved layout is the gated MLP's");
        if (in_ld == 0) in_ld = 2 * width;
        if (in_ld < 2 * width) return fail(err, err_cap, "act_mul: bad arguments");
        up = gate + 1;
    } else if (in_ld == 0) {
        in_ld = width;
    }
    if (rows <= 0 || width <= 0 || (!interleaved && in_ld < width) || !out || !up || kind < ACT_SWIGLU || kind > ACT_GEGLU_TANH)
        return fail(err, err_cap, "act_mul: bad arguments");
    if (gated && !gate) return fail(err, err_cap, "act_mul: a gated MLP needs its gate projection");
    if (interleaved && width % 4 == 0 && in_ld % 4 == 0 && width <= 0x3FFFFFFF && aligned(out, 16) && aligned(gate, 16))
        act_mul_pairs_kernel<<<dim3((unsigned)((width / 4 + 255) / 256), (unsigned)std::min<int64_t>(rows, 65535)), 256, 0, st>>>(out, gate, rows, (int)width,
                                                                                                                            in_ld, (int)kind);
    else act_mul_kernel<<<grid_for(rows * width, 256, sm_count(dev)), 256, 0, st>>>(out, gate, up, rows, width, in_ld, (int)kind, interleaved ? 2 : 1);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_add(int64_t device, void *stream, float *out, const float *a, const float *b, int64_t count, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (count <= 0 || !out || !a || !b) return fail(err, err_cap, "add: bad arguments");
    add_kernel<<<grid_for(count, 256, sm_count(dev)), 256, 0, st>>>(out, a, b, count);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_bias_add(int64_t device, void *stream, float *buf, const float *bias, int64_t rows, int64_t width, char *err,
                       int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rows <= 0 || width <= 0 || !buf || !bias) return fail(err, err_cap, "bias_add: bad arguments");
    bias_add_kernel<<<grid_for(rows * width, 256, sm_count(dev)), 256, 0, st>>>(buf, bias, rows, (int)width);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_embedding(int64_t device, void *stream, float *y, const float *table, const int32_t *ids, int64_t n, int64_t vocab,
                        int64_t width, int32_t *status, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (n <= 0 || vocab <= 0 || width <= 0 || !y || !table || !ids || !status) return fail(err, err_cap, "embedding: bad arguments");
    embedding_kernel<<<grid_for(n * width, 256, sm_count(dev)), 256, 0, st>>>(y, table, ids, n, (int)vocab, (int)width, status);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_add_positions(int64_t device, void *stream, float *x, const float *pos, int64_t rows, int64_t l, int64_t pos0,
                            int64_t width, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rows <= 0 || l <= 0 || width <= 0 || pos0 < 0 || !x || !pos) return fail(err, err_cap, "add_positions: bad arguments");
    add_positions_kernel<<<grid_for(rows * width, 256, sm_count(dev)), 256, 0, st>>>(x, pos, rows, (int)l, (int)pos0, (int)width, nullptr);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_add_positions_at(int64_t device, void *stream, float *x, const float *pos, int64_t rows, int64_t l,
                               const int32_t *position, int64_t width, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rows <= 0 || l <= 0 || width <= 0 || !x || !pos || !position) return fail(err, err_cap, "add_positions: bad arguments");
    add_positions_kernel<<<grid_for(rows * width, 256, sm_count(dev)), 256, 0, st>>>(x, pos, rows, (int)l, 0, (int)width, position);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_advance_position(int64_t device, void *stream, int32_t *position, int64_t delta, char *err, int64_t err_cap) {
    SEAM_PROLOGUE();
    if (!position) return fail(err, err_cap, "advance_position: bad arguments");
    advance_position_kernel<<<1, 1, 0, st>>>(position, (int)delta);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_argmax(int64_t device, void *stream, int32_t *out, const float *logits, int64_t rows, int64_t vocab, char *err,
                     int64_t err_cap) {
    SEAM_PROLOGUE();
    if (rows <= 0 || vocab <= 0 || !out || !logits) return fail(err, err_cap, "argmax: bad arguments");
    argmax_kernel<<<(unsigned)rows, ARGMAX_THREADS, 0, st>>>(out, logits, (int)vocab);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// ---- exchange of finished output columns between the GPUs of one node (see comm.cuh) ---------------

namespace {
struct Comm {
    int dev = 0, rank = 0, world = 1;
    size_t bytes = 0;          // the exchange buffer: the receive areas of every site
    unsigned char *base = nullptr;
    int *epoch = nullptr;      // this rank's epoch word
    CommPeers peers{};
    bool mapped[COMM_MAX_WORLD] = {};
    bool local[COMM_MAX_WORLD] = {}; // attached by pointer inside this process (tests), not through an IPC handle
};
constexpr unsigned long long COMM_WAIT_NS = 4000000000ull; // a peer that has not delivered after 4 s is reported, not awaited
} // namespace

int64_t b200i_comm_create(int64_t device, int64_t rank, int64_t world, int64_t bytes, void **comm, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (!comm || world < 1 || world > COMM_MAX_WORLD || rank < 0 || rank >= world || bytes <= 0 || bytes % 16)
        return fail(err, err_cap, "comm_create: bad arguments (1 <= world <= %d, bytes a positive multiple of 16)", COMM_MAX_WORLD);
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    Comm *c = new Comm();
    c->dev = dev; c->rank = (int)rank; c->world = (int)world;
    c->bytes = (size_t)bytes;
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&c->base), c->bytes);
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void **>(&c->epoch), 256);
    if (e == cudaSuccess) e = cudaMemset(c->base, 0, c->bytes); // tag 0 everywhere: no epoch ever has it
    if (e == cudaSuccess) e = cudaMemset(c->epoch, 0, 256);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        if (c->base) cudaFree(c->base);
        if (c->epoch) cudaFree(c->epoch);
        delete c;
        return fail(err, err_cap, "comm_create: %s", cudaGetErrorString(e));
    }
    c->peers.base[rank] = c->base;
    c->mapped[rank] = true;
    *comm = c;
    return 0;
}

int64_t b200i_comm_export(void *comm, void *handle, int64_t handle_bytes, char *err, int64_t err_cap) {
    clear(err, err_cap);
    Comm *c = static_cast<Comm *>(comm);
    if (!c || !handle || handle_bytes < (int64_t)sizeof(cudaIpcMemHandle_t)) return fail(err, err_cap, "comm_export: the handle buffer must hold %d bytes", (int)sizeof(cudaIpcMemHandle_t));
    CUDA_TRY(cudaSetDevice(c->dev));
    cudaIpcMemHandle_t h;
    CUDA_TRY(cudaIpcGetMemHandle(&h, c->base));
    memcpy(handle, &h, sizeof(h));
    return 0;
}

int64_t b200i_comm_attach(void *comm, int64_t peer, const void *handle, char *err, int64_t err_cap) {
    clear(err, err_cap);
    Comm *c = static_cast<Comm *>(comm);
    if (!c || !handle || peer < 0 || peer >= c->world || peer == c->rank || c->mapped[peer]) return fail(err, err_cap, "comm_attach: bad peer %lld", (long long)peer);
    CUDA_TRY(cudaSetDevice(c->dev));
    cudaIpcMemHandle_t h;
    memcpy(&h, handle, sizeof(h));
    void *p = nullptr;
    CUDA_TRY(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
    c->peers.base[peer] = static_cast<unsigned char *>(p);
    c->mapped[peer] = true;
    return 0;
}

int64_t b200i_comm_attach_local(void *comm, int64_t peer, void *other, char *err, int64_t err_cap) {
    clear(err, err_cap);
    Comm *c = static_cast<Comm *>(comm), *o = static_cast<Comm *>(other);
    if (!c || !o || peer < 0 || peer >= c->world || peer == c->rank || c->mapped[peer] || o->rank != peer || o->world != c->world ||
        o->bytes != c->bytes || o->dev != c->dev)
        return fail(err, err_cap, "comm_attach_local: the other exchange must be rank %lld of the same world, size and device", (long long)peer);
    c->peers.base[peer] = o->base;
    c->mapped[peer] = c->local[peer] = true;
    return 0;
}

int64_t b200i_comm_advance(void *comm, void *stream, char *err, int64_t err_cap) {
    clear(err, err_cap);
    Comm *c = static_cast<Comm *>(comm);
    if (!c) return fail(err, err_cap, "comm_advance: no exchange");
    CUDA_TRY(cudaSetDevice(c->dev));
    comm_advance_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(c->epoch);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_comm_gather(void *comm, void *stream, int64_t mode, int64_t area_bytes, float *out, int64_t out_ld, const float *src,
                          int64_t m, int64_t w, int64_t src_ld, char *err, int64_t err_cap) {
    clear(err, err_cap);
    Comm *c = static_cast<Comm *>(comm);
    if (!c) return fail(err, err_cap, "comm_gather: no exchange");
    if (mode < COMM_SEND_RECV || mode > COMM_RECV) return fail(err, err_cap, "comm_gather: bad mode");
    for (int p = 0; p < c->world; p++)
        if (!c->mapped[p]) return fail(err, err_cap, "comm_gather: rank %d's buffer is not attached", p);
    if (!out || m <= 0 || w <= 0 || area_bytes < 0 || area_bytes % 16 || (mode != COMM_RECV && !src)) return fail(err, err_cap, "comm_gather: bad arguments");
    if (src_ld == 0) src_ld = w;
    if (out_ld == 0) out_ld = w * c->world;
    if (src_ld < w || out_ld < w * c->world) return fail(err, err_cap, "comm_gather: a row pitch is below its row width");
    if ((size_t)area_bytes + (size_t)m * (size_t)w * c->world * 8 > c->bytes)
        return fail(err, err_cap, "comm_gather: the site's receive areas do not fit the exchange buffer");
    CUDA_TRY(cudaSetDevice(c->dev));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool pair = w % 2 == 0 && src_ld % 2 == 0 && out_ld % 2 == 0 && aligned(out, 8) && (mode == COMM_RECV || aligned(src, 8));
    const long long items = pair ? m * (w / 2) : m * w;
    long long blocks = (items + COMM_THREADS - 1) / COMM_THREADS;
    const long long cap = 2ll * sm_count(c->dev);
    const unsigned grid = (unsigned)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
    if (pair)
        comm_gather_kernel<true><<<grid, COMM_THREADS, 0, st>>>(c->peers, c->epoch, src, src_ld, out, out_ld, area_bytes, (int)m, (int)w, c->world,
                                                                c->rank, (int)mode, COMM_WAIT_NS);
    else
        comm_gather_kernel<false><<<grid, COMM_THREADS, 0, st>>>(c->peers, c->epoch, src, src_ld, out, out_ld, area_bytes, (int)m, (int)w, c->world,
                                                                 c->rank, (int)mode, COMM_WAIT_NS);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_comm_gather_nodes(void *comm, void *stream, int64_t mode, int64_t area_bytes, float *out, int64_t out_ld, const float *ws,
                                int64_t nodes, int64_t m, int64_t n, const float *bias, int64_t act, char *err, int64_t err_cap) {
    clear(err, err_cap);
    Comm *c = static_cast<Comm *>(comm);
    if (!c) return fail(err, err_cap, "comm_gather_nodes: no exchange");
    if (mode != COMM_SEND_RECV && mode != COMM_SEND) return fail(err, err_cap, "comm_gather_nodes: bad mode");
    for (int p = 0; p < c->world; p++)
        if (!c->mapped[p]) return fail(err, err_cap, "comm_gather_nodes: rank %d's buffer is not attached", p);
    if (act < EPI_ACT_NONE || act > EPI_PAIR_GEGLU_TANH) return fail(err, err_cap, "comm_gather_nodes: unknown store activation %lld", (long long)act);
    if (!out || !ws || m <= 0 || n <= 0 || n % 4 || nodes < 2 || nodes > MAX_GROUPS || area_bytes < 0 || area_bytes % 16 || m * n > 0x7FFFFFFFll)
        return fail(err, err_cap, "comm_gather_nodes: bad arguments (n a multiple of 4, 2 to %d nodes)", MAX_GROUPS);
    const int64_t w = act >= EPI_PAIR_SWIGLU ? n / 2 : n;
    if (out_ld == 0) out_ld = w * c->world;
    if (out_ld < w * c->world || out_ld % 2 || !aligned(out, 8) || !aligned(ws, 16) || (bias && !aligned(bias, 4)))
        return fail(err, err_cap, "comm_gather_nodes: misaligned storage or a row pitch below the row width");
    if ((size_t)area_bytes + (size_t)m * (size_t)w * c->world * 8 > c->bytes)
        return fail(err, err_cap, "comm_gather_nodes: the site's receive areas do not fit the exchange buffer");
    CUDA_TRY(cudaSetDevice(c->dev));
    const long long cells = m * n;
    const unsigned subs = (unsigned)((nodes + FOLD_SUB - 1) / FOLD_SUB);
    comm_fold_gather_kernel<<<(unsigned)((cells / 4 + 31) / 32), 32 * subs, 0, static_cast<cudaStream_t>(stream)>>>(
        c->peers, c->epoch, ws, (int)nodes, Epilogue{bias, (int)act}, out, out_ld, area_bytes, (int)m, (int)n, c->world, c->rank, (int)mode, COMM_WAIT_NS);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

int64_t b200i_comm_destroy(void *comm) {
    Comm *c = static_cast<Comm *>(comm);
    if (!c) return 0;
    cudaSetDevice(c->dev);
    cudaDeviceSynchronize();
    for (int p = 0; p < c->world; p++)
        if (p != c->rank && c->mapped[p] && !c->local[p]) cudaIpcCloseMemHandle(c->peers.base[p]);
    cudaFree(c->base);
    cudaFree(c->epoch);
    cudaGetLastError();
    delete c;
    return 0;
}

// ---- host-pointer twins -------------------------------------------------------------------

// The copies of one host-pointer call: through the worker threads for pageable arrays when there are megabytes of them
// (see host_copy.cuh), else plain asynchronous copies: below 8 MB starting the threads costs what they save (256 x 1024 x 1024
// 440 us plain, 480 with them), and without a pipeline to overlap, below 16 MB unless one operand has 8 (1000 cubed 755 us
// plain, 800 to 870 with them; 1 x 4096 x 512 603 against 521).
constexpr size_t HOST_STAGED_MIN = 8u << 20;
struct HostTransfers {
    struct Span {
        const void *p;
        size_t bytes;
    };
    HostTransfers(HostPool &pool, int dev, size_t least, std::initializer_list<Span> spans) {
        size_t total = 0;
        for (const Span &s : spans)
            if (host_is_pageable(s.p)) total += s.bytes;
        if (total < least) return;
        if (host_stage_prepare(pool.stage) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        copier = new (std::nothrow) HostCopier(pool.stage, dev, total);
        if (copier && !copier->ok()) {
            delete copier;
            copier = nullptr;
        }
    }
    ~HostTransfers() { delete copier; } // joins the workers
    HostTransfers(const HostTransfers &) = delete;
    HostTransfers &operator=(const HostTransfers &) = delete;
    cudaError_t to_device(void *dst, const void *src, size_t bytes, cudaStream_t st, int *segment) {
        *segment = -1;
        if (!copier || !host_is_pageable(src)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
        *segment = copier->add(true, dst, const_cast<void *>(src), bytes, bytes, 1, st);
        return cudaSuccess;
    }
    void wait(int segment) { // until the segment's transfers are queued on its stream
        if (copier) copier->wait(segment);
    }
    cudaError_t to_host(void *dst, size_t pitch, size_t width, const void *src, size_t rows, cudaStream_t st) {
        if (!copier || !host_is_pageable(dst)) {
            if (rows == 1) return cudaMemcpyAsync(dst, src, width, cudaMemcpyDeviceToHost, st);
            return cudaMemcpy2DAsync(dst, pitch, src, width, width, rows, cudaMemcpyDeviceToHost, st);
        }
        const int seg = copier->add(false, const_cast<void *>(src), dst, width, rows == 1 ? width : pitch, rows, st);
        if (seg < 0) return cudaErrorInvalidValue;
        return cudaSuccess;
    }
    cudaError_t finish() { return copier ? copier->finish() : cudaSuccess; }
    HostCopier *copier = nullptr;
};

// The host-pointer product, pipelined over three streams (PCIe is full duplex): host-to-device copies, packing and
// multiplying, device-to-host copies. A tall left operand (m >= 1024) is cut by ROWS: the weight crosses and is
// packed once, the rows of A cross in chunks while earlier chunks are multiplied and their rows of C return. A wide
// k-contiguous weight under a short left operand (op NT, n >= 2048) is cut by weight rows, that is by COLUMNS of C:
// A crosses and is packed once, the weight crosses in chunks, each chunk's columns are computed into a dense block
// and return through a strided copy. Every chunk is a product of its own, so the bits are those of the whole
// product (a cell reads one row of A and one row of the weight). Returns 0 done, 1 error, -1 not applicable (the
// caller runs the plain path).
static int64_t host_gemm_pipelined(int dev, HostPool &pool, float *c, const float *a, const void *b, const void *bscale, int wkind,
                                   int64_t m, int64_t n, int64_t k, int op, char *err, int64_t err_cap) {
    // cut the larger operand: its copy is the one worth hiding under the arithmetic and the return copy
    const bool rows_ok = op != OP_TN && m >= 4 * PACKED_MIN_EXTENT && n >= PACKED_MIN_EXTENT;
    const bool cols_ok = op == OP_NT && n >= 8 * PACKED_MIN_EXTENT && m >= 1;
    const bool weight_larger = (double)n * (double)wkind_elem_bytes(wkind) > 2.0 * (double)m * 4.0;
    const bool by_cols = cols_ok && (!rows_ok || weight_larger);
    const bool by_rows = rows_ok && !by_cols;
    if (!by_rows && !by_cols) return -1;
    const int64_t extent = by_rows ? m : n;
    const int64_t per = ((extent + 3) / 4 + PK_TILE - 1) / PK_TILE * PK_TILE; // about four chunks, whole tiles
    const int nch = (int)((extent + per - 1) / per);
    if (nch < 2 || nch > HOST_CHUNKS) return -1;
    if (!pool.pipe_ready) {
        CUDA_TRY(cudaStreamCreateWithFlags(&pool.s_in, cudaStreamNonBlocking));
        CUDA_TRY(cudaStreamCreateWithFlags(&pool.s_out, cudaStreamNonBlocking));
        for (auto &e : pool.ev) CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        pool.pipe_ready = true;
    }
    const size_t es = wkind_elem_bytes(wkind);
    const size_t abytes = (size_t)m * k * 4, bbytes = (size_t)n * k * es, cbytes = (size_t)m * n * 4;
    const size_t sbytes = (wkind >= W_INT8_EXP) ? (size_t)n * 4 : 0;
    const size_t wsbytes = pk_workspace_bytes(m, n, k);
    void *da, *db, *dc, *ds = nullptr, *dw = nullptr;
    CUDA_TRY(pool_get(dev, 0, abytes, &da));
    CUDA_TRY(pool_get(dev, 1, bbytes, &db));
    CUDA_TRY(pool_get(dev, 2, cbytes, &dc));
    if (sbytes) CUDA_TRY(pool_get(dev, 3, sbytes, &ds));
    CUDA_TRY(pool_get(dev, 4, wsbytes, &dw));
    packed_configure();
    const int sms = sm_count(dev);
    const int leaf = (int)leaf_size(k), leaves = (int)leaf_count(k), wpl = pk_windows_per_leaf(leaf);
    float *pa = static_cast<float *>(dw);
    float *pb = pa + pk_panel_floats(m, k);
    unsigned char *fa = reinterpret_cast<unsigned char *>(pb + pk_panel_floats(n, k));
    unsigned char *fb = fa + pk_flag_bytes(m, k);
    const bool k4 = (k % 4 == 0) && (leaves == 1 || leaf % 4 == 0); // the device copies are aligned: whole quads where the extents are
    // a chunk's tiles alone rarely fill the device: its leaves are split like any other product's
    const Plan split = by_rows ? packed_split(Plan{PLAN_PACKED, leaves, 1}, std::min(per, m), n, k, sms)
                               : packed_split(Plan{PLAN_PACKED, leaves, 1}, m, std::min(per, n), k, sms);
    void *dn = nullptr;
    if (split.groups > 1) CUDA_TRY(pool_get(dev, 5, (size_t)split.groups * (by_rows ? std::min(per, m) * n : m * std::min(per, n)) * 4, &dn));
    auto product = [&](const float *pai, const unsigned char *fai, const float *pbi, const unsigned char *fbi, float *out, int64_t mm, int64_t nn) {
        const int tn = (int)((nn + PK_TILE - 1) / PK_TILE);
        PackedGemmArgs p{pai, pbi, fai, fbi, out, static_cast<float *>(dn), (int)mm, (int)nn, (int)k, leaf, leaves, wpl, split.group_leaves, split.groups, tn,
                         (nn % 4 == 0 && aligned(out, 16)) ? 1 : 0};
        gemm_packed_kernel<false><<<dim3((unsigned)(((mm + PK_TILE - 1) / PK_TILE) * tn), (unsigned)split.groups), PK_THREADS, PK_SMEM_BYTES, pool.stream>>>(p);
        if (split.groups > 1) launch_fold_groups(static_cast<const float *>(dn), out, mm * nn, split.groups, pool.stream);
        g_launches += split.groups > 1 ? 3 : 2; // with its packing pass
    };
    // everything queued below waits for whatever the compute stream still holds from an earlier call
    CUDA_TRY(cudaEventRecord(pool.ev[0], pool.stream));
    CUDA_TRY(cudaStreamWaitEvent(pool.s_in, pool.ev[0], 0));
    CUDA_TRY(cudaStreamWaitEvent(pool.s_out, pool.ev[0], 0));
    // the operand that is not cut crosses first and is packed once
    HostTransfers io(pool, dev, HOST_STAGED_MIN, {{a, abytes}, {b, bbytes}, {c, cbytes}});
    const void *first = by_rows ? b : static_cast<const void *>(a);
    int seg_first = -1, seg_in[HOST_CHUNKS + 1];
    CUDA_TRY(io.to_device(by_rows ? db : da, first, by_rows ? bbytes : abytes, pool.s_in, &seg_first));
    if (by_rows && sbytes) CUDA_TRY(cudaMemcpyAsync(ds, bscale, sbytes, cudaMemcpyHostToDevice, pool.s_in));
    auto chunk_in = [&](int i) { // chunk i of the operand that is cut
        const int64_t x0 = i * per, cnt = (extent - x0 < per) ? extent - x0 : per;
        if (by_rows) return io.to_device(static_cast<float *>(da) + (size_t)x0 * k, a + (size_t)x0 * k, (size_t)cnt * k * 4, pool.s_in, &seg_in[i]);
        return io.to_device(static_cast<unsigned char *>(db) + (size_t)x0 * k * es, static_cast<const unsigned char *>(b) + (size_t)x0 * k * es,
                            (size_t)cnt * k * es, pool.s_in, &seg_in[i]);
    };
    auto chunk_out = [&](int i) { // chunk i of C, behind the kernel that wrote it
        const int64_t x0 = i * per, cnt = (extent - x0 < per) ? extent - x0 : per;
        cudaError_t e = cudaStreamWaitEvent(pool.s_out, pool.ev[2 + 2 * i], 0);
        if (e != cudaSuccess) return e;
        if (by_rows) return io.to_host(c + (size_t)x0 * n, (size_t)cnt * n * 4, (size_t)cnt * n * 4, static_cast<float *>(dc) + (size_t)x0 * n, 1, pool.s_out);
        return io.to_host(c + x0, (size_t)n * 4, (size_t)cnt * 4, static_cast<float *>(dc) + (size_t)m * x0, (size_t)m, pool.s_out);
    };
    CUDA_TRY(chunk_in(0));
    io.wait(seg_first);
    CUDA_TRY(cudaEventRecord(pool.ev[0], pool.s_in));
    CUDA_TRY(cudaStreamWaitEvent(pool.stream, pool.ev[0], 0));
    if (by_rows) {
        PackArgs pbargs{pb, fb, db, ds, (int)n, (int)k, leaf, leaves, wpl, op == OP_NT, op == OP_NT ? k4 : n % 4 == 0};
        launch_pack_one(pbargs, wkind, pool.stream);
    } else {
        PackArgs paargs{pa, fa, da, nullptr, (int)m, (int)k, leaf, leaves, wpl, 1, k4};
        launch_pack_one(paargs, W_F32, pool.stream);
    }
    g_launches++;
    for (int i = 0; i < nch; i++) {
        const int64_t x0 = i * per, cnt = (extent - x0 < per) ? extent - x0 : per;
        const int64_t tile0 = x0 / PK_TILE;
        if (i + 1 < nch) CUDA_TRY(chunk_in(i + 1)); // its copies go on while this chunk's kernels are queued
        io.wait(seg_in[i]);
        if (!by_rows && sbytes)
            CUDA_TRY(cudaMemcpyAsync(static_cast<unsigned char *>(ds) + (size_t)x0 * 4, static_cast<const unsigned char *>(bscale) + (size_t)x0 * 4,
                                     (size_t)cnt * 4, cudaMemcpyHostToDevice, pool.s_in));
        CUDA_TRY(cudaEventRecord(pool.ev[1 + 2 * i], pool.s_in));
        CUDA_TRY(cudaStreamWaitEvent(pool.stream, pool.ev[1 + 2 * i], 0));
        if (by_rows) {
            float *pai = pa + (size_t)tile0 * k * PK_TILE;
            unsigned char *fai = fa + (size_t)tile0 * leaves * wpl;
            PackArgs paargs{pai, fai, static_cast<float *>(da) + (size_t)x0 * k, nullptr, (int)cnt, (int)k, leaf, leaves, wpl, 1, k4};
            launch_pack_one(paargs, W_F32, pool.stream);
            product(pai, fai, pb, fb, static_cast<float *>(dc) + (size_t)x0 * n, cnt, n);
        } else {
            float *pbi = pb + (size_t)tile0 * k * PK_TILE;
            unsigned char *fbi = fb + (size_t)tile0 * leaves * wpl;
            PackArgs pbargs{pbi, fbi, static_cast<unsigned char *>(db) + (size_t)x0 * k * es, sbytes ? static_cast<unsigned char *>(ds) + (size_t)x0 * 4 : nullptr,
                            (int)cnt, (int)k, leaf, leaves, wpl, 1, k4};
            launch_pack_one(pbargs, wkind, pool.stream);
            product(pa, fa, pbi, fbi, static_cast<float *>(dc) + (size_t)m * x0, m, cnt); // a dense [m, cnt] block
        }
        CUDA_TRY(cudaEventRecord(pool.ev[2 + 2 * i], pool.stream));
        if (i > 0) CUDA_TRY(chunk_out(i - 1));
    }
    CUDA_TRY(chunk_out(nch - 1));
    CUDA_TRY(io.finish());
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(pool.s_out));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.s_in));
    return check_wait_status(err, err_cap, "identical gemm");
}

int64_t b200i_host_gemm_w(int64_t device, float *c, const float *a, const void *b, const void *bscale, int64_t wkind,
                          int64_t m, int64_t n, int64_t k, int64_t op, char *err, int64_t err_cap) {
    clear(err, err_cap);
    if (m <= 0 || n <= 0 || k <= 0)
        return fail(err, err_cap, "identical gemm: m, n and k must be positive (got m=%lld n=%lld k=%lld)", (long long)m,
                    (long long)n, (long long)k);
    if (wkind < W_F32 || wkind > W_INT8_SCALE) return fail(err, err_cap, "identical gemm: unknown weight kind %lld", (long long)wkind);
    if (!c || !a || !b) return fail(err, err_cap, "identical gemm: null storage");
    int dev;
    if (select_device(device, err, err_cap, &dev)) return 1;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    HostPool &pool = g_pool[dev];
    if (!pool.stream) CUDA_TRY(cudaStreamCreateWithFlags(&pool.stream, cudaStreamNonBlocking));
    if (op != OP_NN && op != OP_NT && op != OP_TN) return fail(err, err_cap, "identical gemm: unknown op %lld", (long long)op);
    if ((wkind == W_INT8_EXP || wkind == W_INT8_SCALE) && (op != OP_NT || !bscale))
        return fail(err, err_cap, "identical gemm: int8 weight storage is row-scaled: it needs op NT and its per-row exponents or scales");
    {
        const int64_t piped = host_gemm_pipelined(dev, pool, c, a, b, bscale, (int)wkind, m, n, k, (int)op, err, err_cap);
        if (piped >= 0) return piped;
    }
    const size_t abytes = (size_t)m * k * 4, bbytes = (size_t)n * k * wkind_elem_bytes((int)wkind), cbytes = (size_t)m * n * 4;
    const size_t sbytes = (wkind >= W_INT8_EXP) ? (size_t)n * 4 : 0;
    const int64_t wsbytes = b200i_product_workspace_bytes(m, n, k, op, wkind);
    void *da, *db, *dc, *ds = nullptr, *dw = nullptr;
    CUDA_TRY(pool_get(dev, 0, abytes, &da));
    CUDA_TRY(pool_get(dev, 1, bbytes, &db));
    CUDA_TRY(pool_get(dev, 2, cbytes, &dc));
    if (sbytes) CUDA_TRY(pool_get(dev, 3, sbytes, &ds));
    if (wsbytes) CUDA_TRY(pool_get(dev, 4, (size_t)wsbytes, &dw));
    HostTransfers io(pool, dev, std::max(abytes, bbytes) >= HOST_STAGED_MIN ? HOST_STAGED_MIN : 2 * HOST_STAGED_MIN, {{a, abytes}, {b, bbytes}, {c, cbytes}});
    int seg_a, seg_b;
    CUDA_TRY(io.to_device(da, a, abytes, pool.stream, &seg_a));
    CUDA_TRY(io.to_device(db, b, bbytes, pool.stream, &seg_b));
    if (sbytes) {
        if (!bscale) return fail(err, err_cap, "identical gemm: int8 weight storage needs its per-row exponents or scales");
        CUDA_TRY(cudaMemcpyAsync(ds, bscale, sbytes, cudaMemcpyHostToDevice, pool.stream));
    }
    io.wait(seg_a);
    io.wait(seg_b);
    if (launch_product(dev, pool.stream, static_cast<float *>(dc), static_cast<const float *>(da), db, ds, (int)wkind, m, n, k,
                       (int)op, PLAN_AUTO, 0, dw, wsbytes, err, err_cap))
        return 1;
    CUDA_TRY(io.to_host(c, cbytes, cbytes, dc, 1, pool.stream));
    CUDA_TRY(io.finish());
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "identical gemm");
}

#define HOST_PREP()                                                                  \
    clear(err, err_cap);                                                             \
    int dev;                                                                         \
    if (select_device(device, err, err_cap, &dev)) return 1;                         \
    std::lock_guard<std::mutex> lock(g_pool_mu);                                     \
    HostPool &pool = g_pool[dev];                                                    \
    if (!pool.stream) CUDA_TRY(cudaStreamCreateWithFlags(&pool.stream, cudaStreamNonBlocking))

int64_t b200i_host_to_bf16(int64_t device, uint16_t *dst, const float *src, int64_t count, char *err, int64_t err_cap) {
    if (count < 0) return fail(err, err_cap, "to_bf16: negative count");
    if (count == 0) { clear(err, err_cap); return 0; }
    HOST_PREP();
    void *ds, *dd;
    CUDA_TRY(pool_get(dev, 0, (size_t)count * 4, &ds));
    CUDA_TRY(pool_get(dev, 1, (size_t)count * 2, &dd));
    CUDA_TRY(cudaMemcpyAsync(ds, src, (size_t)count * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_to_bf16(dev, pool.stream, static_cast<uint16_t *>(dd), static_cast<const float *>(ds), count, err, err_cap)) return 1;
    CUDA_TRY(cudaMemcpyAsync(dst, dd, (size_t)count * 2, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_from_bf16(int64_t device, float *dst, const uint16_t *src, int64_t count, char *err, int64_t err_cap) {
    if (count < 0) return fail(err, err_cap, "from_bf16: negative count");
    if (count == 0) { clear(err, err_cap); return 0; }
    HOST_PREP();
    void *ds, *dd;
    CUDA_TRY(pool_get(dev, 0, (size_t)count * 2, &ds));
    CUDA_TRY(pool_get(dev, 1, (size_t)count * 4, &dd));
    CUDA_TRY(cudaMemcpyAsync(ds, src, (size_t)count * 2, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_from_bf16(dev, pool.stream, static_cast<float *>(dd), static_cast<const uint16_t *>(ds), count, err, err_cap)) return 1;
    CUDA_TRY(cudaMemcpyAsync(dst, dd, (size_t)count * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_quantize_int8(int64_t device, int8_t *codes, int32_t *exponents, const float *x, int64_t rows,
                                 int64_t cols, char *err, int64_t err_cap) {
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "quantize_int8: rows and cols must be positive");
    HOST_PREP();
    void *dx, *dq, *de;
    CUDA_TRY(pool_get(dev, 0, (size_t)rows * cols * 4, &dx));
    CUDA_TRY(pool_get(dev, 1, (size_t)rows * cols, &dq));
    CUDA_TRY(pool_get(dev, 2, (size_t)rows * 4, &de));
    CUDA_TRY(cudaMemcpyAsync(dx, x, (size_t)rows * cols * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_quantize_int8(dev, pool.stream, static_cast<int8_t *>(dq), static_cast<int32_t *>(de), static_cast<const float *>(dx),
                            rows, cols, err, err_cap))
        return 1;
    CUDA_TRY(cudaMemcpyAsync(codes, dq, (size_t)rows * cols, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(exponents, de, (size_t)rows * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_dequantize_int8(int64_t device, float *y, const int8_t *codes, const int32_t *exponents, int64_t rows,
                                   int64_t cols, char *err, int64_t err_cap) {
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "dequantize_int8: rows and cols must be positive");
    HOST_PREP();
    void *dy, *dq, *de;
    CUDA_TRY(pool_get(dev, 0, (size_t)rows * cols * 4, &dy));
    CUDA_TRY(pool_get(dev, 1, (size_t)rows * cols, &dq));
    CUDA_TRY(pool_get(dev, 2, (size_t)rows * 4, &de));
    CUDA_TRY(cudaMemcpyAsync(dq, codes, (size_t)rows * cols, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(de, exponents, (size_t)rows * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_dequantize_int8(dev, pool.stream, static_cast<float *>(dy), static_cast<const int8_t *>(dq),
                              static_cast<const int32_t *>(de), rows, cols, err, err_cap))
        return 1;
    CUDA_TRY(cudaMemcpyAsync(y, dy, (size_t)rows * cols * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_gemm_int8(int64_t device, float *c, const int8_t *qa, const int32_t *ea, const int8_t *qb,
                             const int32_t *eb, int64_t m, int64_t n, int64_t k, char *err, int64_t err_cap) {
    if (m <= 0 || n <= 0 || k <= 0) return fail(err, err_cap, "identical int8 gemm: m, n and k must be positive");
    if (k > 131072) return fail(err, err_cap, "identical int8 gemm: k = %lld exceeds INT8_MAX_K = 131072", (long long)k);
    HOST_PREP();
    void *dqa, *dqb, *dc, *dea, *deb;
    CUDA_TRY(pool_get(dev, 0, (size_t)m * k, &dqa));
    CUDA_TRY(pool_get(dev, 1, (size_t)n * k, &dqb));
    CUDA_TRY(pool_get(dev, 2, (size_t)m * n * 4, &dc));
    CUDA_TRY(pool_get(dev, 3, (size_t)m * 4, &dea));
    CUDA_TRY(pool_get(dev, 4, (size_t)n * 4, &deb));
    CUDA_TRY(cudaMemcpyAsync(dqa, qa, (size_t)m * k, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dqb, qb, (size_t)n * k, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dea, ea, (size_t)m * 4, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(deb, eb, (size_t)n * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_gemm_int8(dev, pool.stream, static_cast<float *>(dc), static_cast<const int8_t *>(dqa), static_cast<const int32_t *>(dea),
                        static_cast<const int8_t *>(dqb), static_cast<const int32_t *>(deb), m, n, k, err, err_cap))
        return 1;
    CUDA_TRY(cudaMemcpyAsync(c, dc, (size_t)m * n * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_quantize_int15(int64_t device, int8_t *hi, int8_t *lo, int32_t *exponents, const float *x, int64_t rows, int64_t cols,
                                  char *err, int64_t err_cap) {
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "quantize_int15: rows and cols must be positive");
    HOST_PREP();
    void *dx, *dh, *dl, *de;
    CUDA_TRY(pool_get(dev, 0, (size_t)rows * cols * 4, &dx));
    CUDA_TRY(pool_get(dev, 1, (size_t)rows * cols, &dh));
    CUDA_TRY(pool_get(dev, 2, (size_t)rows * cols, &dl));
    CUDA_TRY(pool_get(dev, 3, (size_t)rows * 4, &de));
    CUDA_TRY(cudaMemcpyAsync(dx, x, (size_t)rows * cols * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_quantize_int15(dev, pool.stream, static_cast<int8_t *>(dh), static_cast<int8_t *>(dl), static_cast<int32_t *>(de),
                             static_cast<const float *>(dx), rows, cols, err, err_cap))
        return 1;
    CUDA_TRY(cudaMemcpyAsync(hi, dh, (size_t)rows * cols, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(lo, dl, (size_t)rows * cols, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(exponents, de, (size_t)rows * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_dequantize_int15(int64_t device, float *y, const int8_t *hi, const int8_t *lo, const int32_t *exponents, int64_t rows,
                                    int64_t cols, char *err, int64_t err_cap) {
    if (rows <= 0 || cols <= 0) return fail(err, err_cap, "dequantize_int15: rows and cols must be positive");
    HOST_PREP();
    void *dy, *dh, *dl, *de;
    CUDA_TRY(pool_get(dev, 0, (size_t)rows * cols * 4, &dy));
    CUDA_TRY(pool_get(dev, 1, (size_t)rows * cols, &dh));
    CUDA_TRY(pool_get(dev, 2, (size_t)rows * cols, &dl));
    CUDA_TRY(pool_get(dev, 3, (size_t)rows * 4, &de));
    CUDA_TRY(cudaMemcpyAsync(dh, hi, (size_t)rows * cols, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dl, lo, (size_t)rows * cols, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(de, exponents, (size_t)rows * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_dequantize_int15(dev, pool.stream, static_cast<float *>(dy), static_cast<const int8_t *>(dh), static_cast<const int8_t *>(dl),
                               static_cast<const int32_t *>(de), rows, cols, err, err_cap))
        return 1;
    CUDA_TRY(cudaMemcpyAsync(y, dy, (size_t)rows * cols * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

int64_t b200i_host_gemm_int15(int64_t device, float *c, const int8_t *ah, const int8_t *al, const int32_t *ea, const int8_t *bh,
                              const int8_t *bl, const int32_t *eb, int64_t m, int64_t n, int64_t k, char *err, int64_t err_cap) {
    if (m <= 0 || n <= 0 || k <= 0) return fail(err, err_cap, "identical int15 gemm: m, n and k must be positive");
    if (k > INT15_MAX_K) return fail(err, err_cap, "identical int15 gemm: k = %lld exceeds INT15_MAX_K = 65536", (long long)k);
    HOST_PREP();
    // the two planes of an operand share one pool slot, the second one 256-byte aligned behind the first
    const size_t aplane = ((size_t)m * k + 255) / 256 * 256, bplane = ((size_t)n * k + 255) / 256 * 256;
    void *da, *db, *dc, *dea, *deb;
    CUDA_TRY(pool_get(dev, 0, 2 * aplane, &da));
    CUDA_TRY(pool_get(dev, 1, 2 * bplane, &db));
    CUDA_TRY(pool_get(dev, 2, (size_t)m * n * 4, &dc));
    CUDA_TRY(pool_get(dev, 3, (size_t)m * 4, &dea));
    CUDA_TRY(pool_get(dev, 4, (size_t)n * 4, &deb));
    int8_t *dah = static_cast<int8_t *>(da), *dal = dah + aplane, *dbh = static_cast<int8_t *>(db), *dbl = dbh + bplane;
    CUDA_TRY(cudaMemcpyAsync(dah, ah, (size_t)m * k, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dal, al, (size_t)m * k, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dbh, bh, (size_t)n * k, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dbl, bl, (size_t)n * k, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(dea, ea, (size_t)m * 4, cudaMemcpyHostToDevice, pool.stream));
    CUDA_TRY(cudaMemcpyAsync(deb, eb, (size_t)n * 4, cudaMemcpyHostToDevice, pool.stream));
    if (b200i_gemm_int15(dev, pool.stream, static_cast<float *>(dc), dah, dal, static_cast<const int32_t *>(dea), dbh, dbl,
                         static_cast<const int32_t *>(deb), m, n, k, err, err_cap))
        return 1;
    CUDA_TRY(cudaMemcpyAsync(c, dc, (size_t)m * n * 4, cudaMemcpyDeviceToHost, pool.stream));
    CUDA_TRY(cudaStreamSynchronize(pool.stream));
    return check_wait_status(err, err_cap, "b200i host call");
}

} // extern "C"
