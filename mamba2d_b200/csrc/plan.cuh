// Host-side descriptor validation and launch planning (header-only, used by both entry points).
#pragma once

#include <algorithm>
#include <array>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <unordered_map>

#include "common.cuh"

namespace m2d {

constexpr int kMaxDevices = 64;
constexpr size_t kMaxSmem = 227 * 1024;     // shared memory a CTA can have

// Index of the current device for the per-device caches below, or -1 (no device, or one beyond the caches).
inline int device_index() {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return -1; }
    return dev < kMaxDevices ? dev : -1;
}

// SMs of the current device, asked for once per device (plans are made several times per call).
inline int sm_count() {
    static std::atomic<int> cache[kMaxDevices];
    const int dev = device_index();
    int n = dev >= 0 ? cache[dev].load(std::memory_order_relaxed) : 0;
    if (n > 0) return n;
    if (dev < 0 || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
        cudaGetLastError();   // clear; planning still works on a machine without a device
        return 148;
    }
    cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

// Per (kernel, device): the dynamic shared memory it has been allowed, and its resident CTAs per SM for the
// last (block size, shared memory) asked about.  The runtime calls behind both cost a microsecond or more
// each, as much as a launch; they are made once.
struct KernelFacts {
    size_t smem_allowed = 48 * 1024;
    int block = 0, per_sm = 0;
    size_t smem = 0;
};
inline KernelFacts& kernel_facts(const void* kern, std::unique_lock<std::mutex>& lock) {
    static std::mutex m;
    static std::unordered_map<const void*, std::array<KernelFacts, kMaxDevices>> all;
    lock = std::unique_lock<std::mutex>(m);
    const int dev = device_index();
    return all[kern][dev < 0 ? 0 : dev];
}
inline bool allow_smem(const void* kern, size_t smem) {
    std::unique_lock<std::mutex> lock;
    KernelFacts& f = kernel_facts(kern, lock);
    if (smem <= f.smem_allowed) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) { cudaGetLastError(); return false; }
    f.smem_allowed = smem;
    return true;
}
// Resident CTAs per SM (0: the query failed).
inline int resident_ctas(const void* kern, int block, size_t smem) {
    std::unique_lock<std::mutex> lock;
    KernelFacts& f = kernel_facts(kern, lock);
    if (f.block == block && f.smem == smem) return f.per_sm;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, block, smem) != cudaSuccess) { cudaGetLastError(); return 0; }
    f.block = block; f.smem = smem; f.per_sm = n;
    return n;
}

// Test hooks in desc->flags are honoured only when the environment asks for them.
inline bool test_hooks_enabled() {
    const char* e = getenv("M2D_TEST_HOOKS");
    return e && e[0] == '1';
}

inline int check_desc(const m2d_scan_desc* d, bool bwd, bool need_ptrs) {
    if (!d) return M2D_ERR_NULL;
    if (d->struct_bytes != sizeof(m2d_scan_desc)) return M2D_ERR_ABI;
    if (d->dtype != M2D_F32 && d->dtype != M2D_BF16) return M2D_ERR_DTYPE;
    {
        unsigned known = M2D_SCAN_REVERSE | M2D_SCAN_A_LOG | M2D_SCAN_D_F32;
        known |= bwd ? M2D_SCAN_BC_ZEROED : M2D_SCAN_GELU_OUT | M2D_SCAN_WS_CLEARED;      // an output activation exists in the forward only, gradients in the backward
        const unsigned hooks = M2D_SCAN_TEST_WITHHOLD | M2D_SCAN_TEST_REPORT | M2D_SCAN_TEST_SHORT | (bwd ? M2D_SCAN_TEST_WITHHOLD_UP : 0u);
        if ((d->flags & hooks) && test_hooks_enabled()) known |= hooks;
        if (d->flags & ~known) return M2D_ERR_FLAGS;
    }
    if (d->B < 1 || d->E < 1 || d->N < 1 || d->H < 2 || d->W < 2) return M2D_ERR_SHAPE;
    if (d->N > kMaxN) return M2D_ERR_UNSUPPORTED_N;
    if (d->BT_pitch < d->N || d->BL_pitch < d->N || d->C_pitch < d->N) return M2D_ERR_PITCH;
    {
        // the kernels index every tensor with 31-bit element offsets
        long long widest = d->E > 48 ? d->E : 48;
        if (bwd && d->d_BC_pitch > widest) widest = d->d_BC_pitch;
        if (d->BT_pitch > widest) widest = d->BT_pitch;
        if (d->BL_pitch > widest) widest = d->BL_pitch;
        if (d->C_pitch > widest) widest = d->C_pitch;
        if ((long long)d->B * d->H * d->W * widest >= (1ll << 31)) return M2D_ERR_TOO_LARGE;
    }
    if (bwd && d->d_BC_pitch != 0 && d->d_BC_pitch < d->N) return M2D_ERR_PITCH;
    if (need_ptrs) {
        if (!d->x || !d->dT || !d->dL || !d->AT || !d->AL || !d->BT || !d->BL || !d->C || !d->D) return M2D_ERR_NULL;
        if (bwd && (!d->gy || !d->d_x || !d->d_dT || !d->d_dL || !d->d_AT || !d->d_AL || !d->d_BT || !d->d_BL || !d->d_C || !d->d_D))
            return M2D_ERR_NULL;
    }
    return M2D_OK;
}

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// 128-bit (fp32) / 64-bit (bf16) vector loads need channel and state counts that are multiples
// of 4, pitches that are multiples of 4 elements and suitably aligned base pointers.
inline bool vector_ok(const m2d_scan_desc* d, bool bwd) {
    const size_t al = d->dtype == M2D_F32 ? 16 : 8;
    bool ok = (d->E % 4 == 0) && (d->N % 4 == 0) && (d->BT_pitch % 4 == 0) && (d->BL_pitch % 4 == 0) && (d->C_pitch % 4 == 0);
    ok = ok && aligned(d->x, al) && aligned(d->dT, al) && aligned(d->dL, al) && aligned(d->BT, al) && aligned(d->BL, al) && aligned(d->C, al);
    if (bwd) ok = ok && aligned(d->gy, al);
    return ok;
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// CTAs per image that a chained launch may use: at most one per band, and, when CTAs own more than one band
// each, fewer than one row of steps divided by the rows of a band.  `want` is the chain the resident CTA slots allow;
// `steps_per_row` the steps a warp needs for one row.  Every place that picks or shortens a chain goes
// through this rule.
//
// The batch kernels need the second limit: their warps walk a CTA's bands in lock step, so that a first warp that waits for
// its next band holds up the last columns of this one, and with them the bands below it that it waits for.  For the wave
// kernels it is cautious: a CTA finishes a band before it takes its next, bands are taken in ascending order (descending in
// the adjoint sweep) and each waits only for the one before, so that whatever the chain's length some CTA can always go on.
// On narrow maps it leaves SMs idle: 4x200x14x96 gets one CTA per image where six are free, 600 dependent
// steps instead of 384; 3x45x31x192 135 instead of 115.
inline int bound_chain(long long want, int nbands, int steps_per_row, int Rb) {
    if (want > nbands) want = nbands;
    if (want < nbands) {
        const long long lim = steps_per_row / Rb - 1;
        if (want > lim) want = lim;
    }
    return want < 1 ? 1 : (int)want;
}

// Batch mode: one CTA per (image, 16 channels), images chained per CTA; a warp owns two rows of a band.
constexpr int kPairWarps = 8;            // warps per CTA, at most (128 registers: 16 per SM)
enum PairKernel { kPairForward, kPairStates, kPairAdjoint };

// Time of a batch launch, us, as the plans compare it: the steps of the busiest CTA, times a time per step that grows with
// the warps of the busiest SM that have a row and with the share of the steps in which some warp of a CTA starts a row (and,
// where the record is written, with the CTAs), and something per band.  Least squares over 34 shapes of the models' range
// (1 ... 128 images, 5 ... 2400 rows) x 1 ... 8 warps: 5 % mean error; the number of warps taken by it costs 0.6 % (2 % where the
// record is written) on the best one, geometric mean, and 7 ... 15 % at worst.
inline double pair_time(const m2d_scan_desc* d, const Plan& p, PairKernel k, int per_sm, int sms) {
    const int per = (d->B - 1) / p.grid_x + 1;
    const long long ctas = (long long)p.grid_x * p.groups;
    const int fill = (int)((ctas + sms - 1) / sms);
    const double bands = (double)per * p.nbands, steps = bands * d->W + 2 * p.warps + 1, on_sm = fill < per_sm ? fill : per_sm;
    const double w = on_sm * d->H / (2.0 * p.nbands), wrap = 2 * p.warps < d->W ? 2.0 * p.warps / d->W : 1.0;
    const double t = k == kPairForward ? 1.2 + 1.37 * bands + (0.312 + 0.0340 * w + 0.089 * wrap) * steps
                     : k == kPairStates ? 1.5 + 1.38 * bands + (0.338 + 0.0435 * w + 0.024 * wrap + 0.0070 * on_sm) * steps
                                        : 0.5 + 1.86 * bands + (0.601 + 0.0768 * w + 0.075 * wrap) * steps;
    return fill > per_sm ? t * fill / per_sm : t;
}
// The wave kernels' times below are upper bounds, by about this much where they are compared with the batch kernels'.
constexpr double kWaveMargin = 1.08;

// The same for the sweeps of a backward with the bands of an image in `chain` CTAs.  A band starts kPairLag columns behind
// the last row of the one above, and a CTA takes its next one when it has finished one.  8 % mean error over 13 shapes, above for short ones.
constexpr int kPairLag = 5;
inline double pair_chain_time(const m2d_scan_desc* d, const Plan& p, PairKernel k, int sms) {
    const double lag = p.Rb + kPairLag;
    const double start = p.chain * lag >= d->W ? (p.nbands - 1) * lag : (p.nbands - 1) / p.chain * (double)d->W + (p.nbands - 1) % p.chain * lag;
    const double steps = start + d->W + 2 * p.warps + 1, w = (double)(((long long)d->B * p.groups * p.chain + sms - 1) / sms) * p.warps;
    return k == kPairStates ? (0.54 + 0.025 * w) * steps : (0.84 + 0.043 * w) * steps;
}
// Chained sweeps are taken where they come to less than this share of a wave launch, whose time is an upper bound: where the
// bands are more than the CTAs the wave kernels can have resident.  Backward, us, wave / chained: 16x100x112x64 fp32 1064 /
// 769 (of a share of 0.63), 1x400x400x384 fp32 4683 / 3382 (0.66); but 5x37x53x96 154 / 188 (0.86), 3x80x80x96 290 / 339 (0.95),
// 2x200x336x64 bf16 982 / 1079 (0.97): a step of these kernels takes longer where it is the chain that bounds.  (In the
// forward 16x100x112x64 gains 270 / 219; not taken.)
constexpr double kChainShare = 0.80;
// ... and to less than this share of one CTA per image, whose estimate is high by about as much as this one is low.  Backward, us,
// one CTA per image / chained, without clearing: 20x45x31x192 bf16 294 / 332 (0.87), 32x56x56x64 fp32 424 / 414 (0.73),
// 48x64x80x64 bf16 947 / 809 (0.65), 40x100x120x64 fp32 2258 / 1797 (0.63).  What the two lines leave out is that a call waits for a
// chained scan before it returns: 20 ... 40 us of the host's lead.  Whole training calls at the line, back to back, not chained / chained: 8x39x34x320 fp32 573 / 544,
// 47x40x35x64 517 / 508, 4x36x53x320 535 / 487, 15x40x63x96 bf16 588 / 547, 14x39x42x192 bf16 573 / 563, 55x49x30x64 bf16 535 / 555, 23x58x32x128
// bf16 592 / 615; well below it 8x69x49x320 bf16 1061 / 906, 28x89x102x96 bf16 2639 / 2357.  (The two that lose would keep their states in bf16.)
constexpr double kChainShareOfBatch = 0.70;

// Bytes of the rings that carry a band's last row to the next band.
inline size_t pair_ring_bytes(const m2d_scan_desc* d, const Plan& p) {
    return p.nbands > 1 ? (size_t)p.grid_x * p.groups * d->W * kSlotF4 * sizeof(float4) : 0;
}

// Rings beyond this (three quarters of the L2) also cost the trip to DRAM that pair_time leaves out: such a plan is taken only where every
// other has as large ones.
constexpr size_t kRingBytes = 96u << 20;

// Every number of warps is tried; of the plans whose rings take at most `ring_limit` bytes the one with the least time is kept
// (in *time, us).  Fewer warps are more bands, more CTAs and more rings: 18x6x593x892 needs 612 MB of them with one warp per
// CTA and none with three.  Where no plan has room, the one with the smallest rings.
inline Plan plan_pairs(const m2d_scan_desc* d, PairKernel k, double* time, size_t ring_limit = kRingBytes) {
    Plan best{};
    size_t best_over = 0;
    const int sms = sm_count();
    for (int nw = kPairWarps; nw >= 1; --nw) {
        Plan p{};
        p.groups = (d->E + kGroup - 1) / kGroup;
        p.Rb = d->H < 2 * nw ? d->H : 2 * nw;
        // a band boundary must be written two steps before the band below reads it
        if (p.Rb < d->H && p.Rb > d->W - 2) p.Rb = d->W - 2 > 1 ? (d->W - 2) & ~1 : 1;
        p.warps = (p.Rb + 1) / 2;
        p.nbands = (d->H + p.Rb - 1) / p.Rb;
        p.smem = (k == kPairAdjoint ? pairs_bwd_smem_bytes(p.warps) : pairs_fwd_smem_bytes(p.warps)) + kParamF4 * sizeof(float4);
        const int fit = (int)((kMaxSmem + 1024) / (p.smem + 1024)), per_sm = fit < 16 / p.warps ? fit : 16 / p.warps;
        // all CTAs resident at once: CTAs per channel group = floor(slots / groups), images per CTA to match
        int per_group = per_sm * sms / p.groups;
        if (per_group < 1) per_group = 1;
        const int per = (d->B - 1) / per_group + 1;                  // images per CTA
        p.grid_x = (d->B - 1) / per + 1;
        p.chain = 1;
        const double t = pair_time(d, p, k, per_sm, sms);
        const size_t ring = pair_ring_bytes(d, p), over = ring > ring_limit ? ring : 0;
        if (best.warps == 0 || over < best_over || (over == best_over && t < *time)) { best = p; best_over = over; *time = t; }
    }
    return best;
}
// The plan for few images: bands of at least eight rows (the scratch of a band's boundary row), all CTAs resident.
inline Plan plan_pair_chain(const m2d_scan_desc* d, PairKernel k, double* time) {
    Plan best{};
    const int sms = sm_count();
    for (int nw = kPairWarps; nw >= 4; --nw) {
        Plan p{};
        p.groups = (d->E + kGroup - 1) / kGroup;
        p.Rb = 2 * nw;
        if (p.Rb >= d->H || p.Rb > d->W - 2) continue;
        p.warps = nw;
        p.nbands = (d->H + p.Rb - 1) / p.Rb;
        p.smem = (k == kPairAdjoint ? pairs_bwd_smem_bytes(nw) : pairs_fwd_smem_bytes(nw)) + kParamF4 * sizeof(float4);
        const int fit = (int)((kMaxSmem + 1024) / (p.smem + 1024)), per_sm = fit < 16 / nw ? fit : 16 / nw;
        p.chain = bound_chain((long long)per_sm * sms / ((long long)d->B * p.groups), p.nbands, d->W, p.Rb);
        if (p.chain < 2) continue;
        p.grid_x = d->B;
        const double t = pair_chain_time(d, p, k, sms);
        if (best.warps == 0 || t < *time) { best = p; *time = t; }
    }
    return best;
}
inline size_t pair_edge_bytes(const m2d_scan_desc* d, const Plan& p) {
    return align256((size_t)d->B * p.groups * p.nbands * d->W * kSlotF4 * sizeof(float4));
}

// Scratch layout shared by every entry point: [status word, 256 bytes][the rest].
constexpr size_t kStatusBytes = 256;

// Wave kernels (wave.cuh): bands of eight rows, 8 * C channels per CTA, one CTA per SM.  Where images and
// channel groups alone do not fill the GPU every image gets a chain of CTAs; otherwise a CTA walks a list of
// images.
inline Plan plan_wave(const m2d_scan_desc* d, int C) {
    Plan p{};
    p.wave = C;
    p.warps = 8;
    p.Rb = 8;
    p.nbands = (d->H + 7) / 8;
    p.groups = (d->E + 8 * C - 1) / (8 * C);
    const long long slots = sm_count(), ctas = (long long)d->B * p.groups;
    p.chain = ctas <= slots ? bound_chain(slots / ctas, p.nbands, d->W, p.Rb) : 1;
    const long long lists = slots / p.groups > 0 ? slots / p.groups : 1, per = (d->B + lists - 1) / lists;
    p.grid_x = p.chain > 1 ? d->B : (int)((d->B + per - 1) / per);
    return p;
}

// Boundary rows a wave launch keeps per (list, channel group): one per band where another CTA reads them or
// the backward's second sweep comes back to them, else two in turn.
inline int wave_rows(const Plan& p, bool bwd) { return p.nbands == 1 ? 0 : (p.chain == 1 && !bwd ? 2 : p.nbands); }
inline size_t wave_edge_bytes(const m2d_scan_desc* d, const Plan& p, bool bwd) {
    return align256((size_t)p.grid_x * ((d->E + p.wave - 1) / p.wave) * wave_rows(p, bwd) * d->W * 16 * p.wave * sizeof(float));
}

// Steps a wave launch takes, as the plans compare them: bands walked one after the other by the busiest CTA, and the
// start-up of the chain (a band can start when the one above it is about 15 columns in: the eight rows of its wave,
// the chunk of columns being published, the trip through L2).  Too many where a CTA has several bands, because the
// later rounds of the first CTAs run during the start-up: 173 against 128 by the dependences for 5x37x53x96, 951
// against 786 for 2x200x336x64.  The measured times per step in plan_fwd and plan_bwd belong to this count.
inline double wave_steps(const m2d_scan_desc* d, const Plan& p) {
    const long long slots = sm_count(), ctas = (long long)p.grid_x * p.groups * p.chain;
    const long long images = p.chain > 1 ? 1 : ((long long)d->B + p.grid_x - 1) / p.grid_x;
    const long long bands = (ctas + slots - 1) / slots * images * ((p.nbands + p.chain - 1) / p.chain);
    return (double)bands * ((d->W + 12) / 4 * 4) + (p.chain - 1) * 15.0;
}

// Whether a chained forward with four channels per lane hands its boundary rows over in pairs of columns instead of chunks
// of four: a band then starts about 12 columns behind the one above instead of 15, and looks at the boundary twice per
// chunk.  Worth it where the start-up of the chain is a good part of the steps, with bf16 I/O, whose chunks are sent later
// (kGiveAfter), a tenth, in fp32 three tenths.  Chunks / pairs, us, by the start-up's share of the steps:
//   bf16  400x400x384 (7 %) 1143 / 1157, 3x85x96x384 (12 %) 205 / 204, 300x900x192 (16 %) 1125 / 1112, 512x512x192 (18 %) 1011 / 989,
//         4x130x200x128 (22 %) 304 / 293, 300x500x192 (25 %) 680 / 668, 2x336x336x96 (33 %) 561 / 511
//   fp32  512x512x192 (18 %) 1002 / 1051, 300x500x192 (25 %) 686 / 709, 3x200x300x96 (26 %) 420 / 435, 2x300x336x96 (33 %) 531 / 513,
//         250x250x256 (33 %) 432 / 410, 1024x1024x64 (35 %) 1734 / 1626
// With two channels per lane, whose steps are shorter, pairs are slower (2x200x336x64 bf16 286 / 314).
// plan_fwd charges plans with pairs the 15 columns all the same: what it charges the two-channel plans is above their time
// by more.  With 12 columns every 25th shape of the models' range goes from two channels to four and takes 1.14 times as long
// (geometric mean of 90 of them; 2x306x183x96 fp32 346 / 410 us, 1x310x435x64 bf16 396 / 529, 2x502x452x64 fp32 829 / 777).
inline bool edge_pairs(const m2d_scan_desc* d, const Plan& p, size_t element) {
    return p.wave == 4 && p.chain > 1 && (p.chain - 1) * 15.0 * 10.0 >= wave_steps(d, p) * (element == 2 ? 1 : 3);
}

// A thread's last plan of a kind.  A call asks for its plan several times (workspace, chain, launch), at 1 ... 2 us each; the
// plan depends on what is compared here and on nothing else.
template <typename P>
struct LastPlan {
    int device = -2, B, H, W, E, N, dtype;
    P plan;
    template <typename F>
    const P& get(const m2d_scan_desc* d, F make) {
        const int dev = device_index();
        if (dev != device || d->B != B || d->H != H || d->W != W || d->E != E || d->N != N || (int)d->dtype != dtype) {
            plan = make();
            device = dev; B = d->B; H = d->H; W = d->W; E = d->E; N = d->N; dtype = (int)d->dtype;
        }
        return plan;
    }
};

// The fastest plan, or with a `scratch_limit` the fastest that fits it; where none does, one that says how much it needs.
inline Plan make_plan_fwd(const m2d_scan_desc* d, size_t scratch_limit = SIZE_MAX) {
    // The batch kernel runs one CTA per (image, 16 channels) and is at its best when those fill the GPU; the wave kernels
    // split an image over CTAs as well.  Measured times per step of those: 0.62 us with four channels per lane, 0.42 us
    // with two and twice the CTAs.  The batch kernel needs three columns.
    Plan p{};
    double best = 1e30;
    if (d->W >= 3) {
        p = plan_pairs(d, kPairForward, &best, std::min(kRingBytes, scratch_limit - kStatusBytes));
        best *= kWaveMargin;
        p.scratch = kStatusBytes + align256(pair_ring_bytes(d, p));
    }
    auto consider = [&](Plan w, double step) {
        const double t = step * wave_steps(d, w);
        w.scratch = kStatusBytes + wave_edge_bytes(d, w, false);
        const bool room = w.scratch <= scratch_limit, had = best < 1e30 && p.scratch <= scratch_limit;
        if (best == 1e30 || (room && (!had || t < best))) { best = t; p = w; }
    };
    for (const int C : {4, 2}) {
        Plan w = plan_wave(d, C);
        consider(w, C == 4 ? 0.62 : 0.42);
        if (scratch_limit == SIZE_MAX || w.chain == 1) continue;
        w.chain = 1;                     // (two boundary rows in turn, instead of one per band)
        consider(w, C == 4 ? 0.62 : 0.42);
    }
    return p;
}

inline Plan plan_fwd(const m2d_scan_desc* d) {
    static thread_local LastPlan<Plan> last;
    return last.get(d, [&] { return make_plan_fwd(d); });
}

}  // namespace m2d
