// Host-side descriptor validation and launch planning (header-only, used by both entry points).
#pragma once

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
        const unsigned hooks = M2D_SCAN_TEST_WITHHOLD | M2D_SCAN_TEST_REPORT | (bwd ? M2D_SCAN_TEST_WITHHOLD_UP : 0u);
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

// Row-warps per CTA: as many as allowed, traded against rows lost to padding in the last band
// (score = warps x fraction of useful rows; ties go to the better fraction).
inline int pick_warps(int H, int max_warps) {
    if (H <= max_warps) return H;
    int best = max_warps;
    double best_score = -1.0, best_eff = 0.0;
    for (int w = max_warps; w >= 2; --w) {
        const int bands = (H + w - 1) / w;
        const double eff = (double)H / ((double)bands * w);
        const double score = w * eff;
        if (score > best_score + 1e-9 || (score > best_score - 1e-9 && eff > best_eff)) {
            best_score = score; best_eff = eff; best = w;
        }
    }
    return best;
}

// Batch mode: one CTA per (image, 32-channel group), images chained per CTA.
inline Plan plan_common(const m2d_scan_desc* d, int max_warps, int warps_per_sm) {
    Plan p{};
    p.groups = (d->E + kGroup - 1) / kGroup;
    p.warps = pick_warps(d->H, max_warps);
    p.Rb = p.warps;
    p.nbands = (d->H + p.Rb - 1) / p.Rb;
    if (p.nbands > 1 && p.Rb > d->W - 2) {
        // a band boundary must be written two steps before the band below reads it
        p.Rb = d->W - 2 > 1 ? d->W - 2 : 1;
        p.warps = p.Rb;
        p.nbands = (d->H + p.Rb - 1) / p.Rb;
    }
    const int ctas_per_sm = warps_per_sm / p.warps > 0 ? warps_per_sm / p.warps : 1;
    const long long slots = (long long)ctas_per_sm * sm_count();
    // all CTAs resident at once: CTAs per channel group = floor(slots / groups), images per CTA to match
    long long per_group = slots / p.groups;
    if (per_group < 1) per_group = 1;
    const long long per = (d->B + per_group - 1) / per_group;    // images per CTA
    p.grid_x = (int)((d->B + per - 1) / per);
    p.chain = 1;
    return p;
}

// Try every cap on the row-warps per CTA and keep the plan that keeps the most warps resident,
// discounted by the rows lost to padding; ties go to the larger CTA.
inline Plan plan_best(const m2d_scan_desc* d, int max_warps, int warps_per_sm) {
    Plan best = plan_common(d, max_warps, warps_per_sm);
    double best_score = -1.0;
    const double cap = (double)warps_per_sm * sm_count();
    for (int w = max_warps; w >= 2; --w) {
        const Plan p = plan_common(d, w, warps_per_sm);
        double resident = (double)p.grid_x * p.groups * p.warps;
        if (resident > cap) resident = cap;
        const double eff = (double)d->H / ((double)p.nbands * p.Rb);
        const double score = resident * eff;
        if (score > best_score * 1.02) { best_score = score; best = p; }
    }
    return best;
}

// Steps the busiest CTA of a batch launch takes.
inline double batch_steps(const m2d_scan_desc* d, const Plan& p) {
    const long long per = ((long long)d->B + p.grid_x - 1) / p.grid_x;
    return (double)per * p.nbands * d->W + p.Rb;
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Scratch layout shared by every entry point: [status word, 256 bytes][the rest].
constexpr size_t kStatusBytes = 256;

// CTAs per image that a wave launch may use: at most one per band, and, when CTAs own more than one band
// each, fewer than one row of steps divided by the rows of a band.  `want` is the chain the resident CTA slots allow;
// `steps_per_row` the steps a warp needs for one row.  Every place that picks or shortens a chain goes
// through this rule.
//
// The second limit is cautious: the waits end without it.  A CTA finishes a band before it takes its next, bands are
// taken in ascending order (descending in the adjoint sweep) and each waits only for the one before, so that
// whatever the chain's length some CTA can always go on.  (Kernels whose CTAs walk their bands in lock-step need
// it.)  On narrow maps it leaves SMs idle: 4x200x14x96 gets one CTA per image where six are free, 600 dependent
// steps instead of 384; 3x45x31x192 135 instead of 115.
inline int bound_chain(long long want, int nbands, int steps_per_row, int Rb) {
    if (want > nbands) want = nbands;
    if (want < nbands) {
        const long long lim = steps_per_row / Rb - 1;
        if (want > lim) want = lim;
    }
    return want < 1 ? 1 : (int)want;
}

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

inline Plan plan_fwd(const m2d_scan_desc* d, bool allow_chain = true) {
    // The batch kernel runs one CTA per (image, 32 channels) and is at its best when those fill the GPU; the
    // wave kernels split an image over CTAs as well.  Measured times per step: 0.9 us (batch), 0.62 us (wave,
    // four channels per lane) and 0.42 us (two channels, twice the CTAs); they put the lines where the
    // measured times cross within 10 % (56x56x64: wave up to batch 64, 290 against 381 us there; 14x14x320:
    // up to batch 8).  The batch kernel needs three columns.  (fp32 or bf16 I/O differ by less than that.)
    Plan p{};
    double best = 1e30;
    if (d->W >= 3) {
        p = plan_best(d, 8, 16);
        p.smem = rows_fwd_smem_bytes(p.warps) + kParamF4 * sizeof(float4);
        p.scratch = kStatusBytes;
        if (p.nbands > 1) p.scratch += align256((size_t)p.grid_x * p.groups * d->W * kSlotF4 * sizeof(float4));
        best = 0.9 * batch_steps(d, p);
    }
    for (const int C : {4, 2}) {
        if (!allow_chain && d->W >= 3) break;
        Plan w = plan_wave(d, C);
        if (!allow_chain) w.chain = 1;
        const double t = (C == 4 ? 0.62 : 0.42) * wave_steps(d, w);
        if (t < best) { best = t; p = w; p.scratch = kStatusBytes + wave_edge_bytes(d, w, false); }
    }
    return p;
}

}  // namespace m2d
