// Backward entry point of the wavefront scan: recompute sweep and adjoint sweep, two kernels in batch mode (one CTA per
// image and channel group, or a chain of them) and one of the wave kernels, followed with bf16 I/O by a small kernel that casts
// the fp32 accumulators of the reduced gradients.
#include <algorithm>

#include "launch.cuh"
#include "sweep_pairs.cuh"
#include "wave_bwd.cuh"

namespace m2d {

// Workspace layout of the backward pass (all regions 256-byte aligned):
//   status   one word, nonzero if a wait between CTAs gave up
//   acc      bf16 I/O only: fp32 accumulators 3 x [B*H*W][N] | 2 x [E][N] | [E], zeroed before the
//            main kernel (with the status word, in one memset) and cast by a second kernel.  With fp32 I/O
//            the kernel accumulates straight into the caller's (zeroed) gradient tensors and this region is empty.
//   edge     batch: per-CTA band-boundary ring, ctas*W KiB (only if nbands > 1); wave and chained batch sweeps: the
//            boundary rows of the recompute sweep (h, downwards) and of the adjoint sweep (pT, upwards)
//   hs       state record written by the recompute sweep: batch, chained or not, B*groups*H*W KiB (half where it is
//            bf16: BwdPlan::wide), wave 512*C bytes per (list, warp, band, step)
struct BwdLayout {
    size_t edge, hs, acc, acc_bytes, total;
};

// The plans of a backward: `states` (batch mode) is the recompute sweep's, `wide` an fp32 state record.
struct BwdPlan : Plan {
    Plan states;
    bool wide;
};

// With bf16 I/O the batch kernels with one CTA per image keep the states of a large batch in bf16, which halves the traffic that
// the recompute sweep waits for, and those of a few images in fp32, as the wave kernels and the chained sweeps do: the gradients
// are then those of the unrounded states.
//
// This line decides what a call's gradients are, so it stays where it was, whatever today's kernels take: "few" is where a wave
// launch comes to less time than one CTA per image and 32 channels with up to six rows in flight each and twelve on an SM.  The
// times per step are those of that division of the work.
inline bool few_images(const m2d_scan_desc* d) {
    const int sms = sm_count(), g = (d->E - 1) / 32 + 1;
    double best = -1.0, time = 0.0;
    for (int w = 6; w >= 2; --w) {
        int Rb = std::min(w, (int)d->H);
        if (Rb < d->H && Rb > d->W - 2) Rb = std::max(1, (int)d->W - 2);
        const int bands = (d->H - 1) / Rb + 1, lists = std::max(1, 12 / Rb * sms / g), per = (d->B - 1) / lists + 1;
        const double ctas = (double)((d->B - 1) / per + 1) * g, score = std::min(ctas * Rb, 12.0 * sms) * d->H / ((double)bands * Rb);
        if (score > best * 1.02) {
            best = score;
            time = (ctas > sms ? 2.45 : 1.95) * ((double)per * bands * d->W + Rb);
        }
    }
    return 1.2 * wave_steps(d, plan_wave(d, 2)) + 10.0 < time;
}

inline BwdLayout bwd_layout(const m2d_scan_desc* d, const BwdPlan& p) {
    BwdLayout L;
    size_t off = kStatusBytes;
    L.acc = off;
    L.acc_bytes = 0;
    if (d->dtype != M2D_F32) {
        const size_t npn = (size_t)d->B * d->H * d->W * d->N, en = (size_t)d->E * d->N;
        L.acc_bytes = align256((3 * npn + 2 * en + d->E) * sizeof(float));
    }
    off += L.acc_bytes;
    L.edge = off;
    if (p.wave) off += 2 * wave_edge_bytes(d, p, true);
    else if (p.chain > 1) off += pair_edge_bytes(d, p.states) + pair_edge_bytes(d, p);
    else off += align256(std::max(pair_ring_bytes(d, p), pair_ring_bytes(d, p.states)));
    L.hs = off;
    if (p.wave) off += align256((size_t)p.grid_x * p.groups * p.warps * p.nbands * (d->W + 7) * p.wave * 512);
    else off += align256((size_t)d->B * p.groups * d->H * d->W * (p.wide ? 64 : 32) * sizeof(float4));
    L.total = off;
    return L;
}

// Scratch beyond which a call's memory comes before its time, a tenth of the device's.  Three choices that are faster ask for more:
//   - chained sweeps keep an fp32 record, also where one CTA per image keeps a bf16 one, and boundary rows: 40x56x56x64 bf16 666 MB
//     for 290, 8x82x84x384 1.73 GB for 0.70.  (With a bf16 record 409 MB and 1.05 GB, and whole training calls of 850 for 872 us and
//     1863 for 1937; but the weights' gradients differ by 1e-3 then.)
//   - the batch kernels' record, chained or not, holds every image of the call, the wave kernels' those that are under way:
//     316x7x9400x71 fp32 106 GB for 11, 40x900x900x64 bf16 172 for 90.
//   - the wave kernels' record is fp32, with seven columns more than the map has: 5x3470x5x589 bf16 5.2 GB for 1.7.
constexpr size_t kLargeScratch = (size_t)16 << 30;

inline BwdPlan make_plan_bwd(const m2d_scan_desc* d) {
    // Batch or wave, as in plan_fwd: 1.2 us per step of both sweeps in the wave kernel with two channels per lane (four
    // spill and are slower at every size measured), whatever the I/O type.
    BwdPlan p{};
    double best = 1e30;
    if (d->W >= 3) {
        double states = 0.0;
        static_cast<Plan&>(p) = plan_pairs(d, kPairAdjoint, &best);
        p.states = plan_pairs(d, kPairStates, &states);
        p.wide = d->dtype == M2D_F32 || few_images(d);
        best = (best + states) * kWaveMargin;
    }
    BwdPlan small = p;                   // few images: the wave kernels, else one CTA per image
    const Plan w = plan_wave(d, 2);
    if (d->W < 3 || few_images(d)) static_cast<Plan&>(small) = w;
    const double wave = 1.2 * wave_steps(d, w) + 10.0;
    if (wave < best) static_cast<Plan&>(p) = w;
    double adjoint = 0.0, states = 0.0;
    const Plan pa = plan_pair_chain(d, kPairAdjoint, &adjoint), ps = plan_pair_chain(d, kPairStates, &states);
    const double chained = adjoint + states + (pa.warps && ps.warps ? (pair_edge_bytes(d, pa) + pair_edge_bytes(d, ps)) / 5e6 : 1e30);    // (and clearing)
    if (chained < kChainShare * wave && chained < kChainShareOfBatch * best) {
        static_cast<Plan&>(p) = pa;
        p.states = ps;
        p.wide = true;
    }
    p.scratch = bwd_layout(d, p).total;
    if (p.scratch > kLargeScratch) {
        small.scratch = bwd_layout(d, small).total;
        if (small.scratch < p.scratch - p.scratch / 8) return small;
    }
    return p;
}

inline BwdPlan plan_bwd(const m2d_scan_desc* d) {
    static thread_local LastPlan<BwdPlan> last;
    return last.get(d, [&] { return make_plan_bwd(d); });
}

// Few images: several CTAs per image.
template <typename io_t, bool VEC>
__global__ void __launch_bounds__(256, 1) m2d_bwd_wave_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    wave_backward<io_t, 2, VEC>(a, reinterpret_cast<char*>(smem));
}

// Batch mode (one CTA per image and channel group, or a chain of them): the recompute sweep, which writes the state record and d_C, and the
// adjoint sweep, each a kernel of its own: their registers, shared memory and bands need not be the same.
template <typename io_t, typename rec_t, bool VEC, bool CHAIN>
__global__ void __launch_bounds__(kPairWarps * 32, 2) m2d_bwd_states_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    const PairLane ln(a);
    const unsigned params = begin_pairs<io_t>(a, smem, pairs_fwd_smem_bytes(ln.nwarps), ln);
    forward_pairs<io_t, rec_t, VEC, true, false, CHAIN>(a, smem_u32(smem), params, 0.f);
}

template <typename io_t, typename rec_t, bool VEC, bool CHAIN>
__global__ void __launch_bounds__(kPairWarps * 32, 2) m2d_bwd_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    const PairLane ln(a);
    const unsigned params = begin_pairs<io_t>(a, smem, pairs_bwd_smem_bytes(ln.nwarps), ln);
    const int o_ch = ln.ch0 + (ln.nq & 1);
    const float D_lane = o_ch < a.E ? load_D<io_t>(a, o_ch) : 0.f;
    Quad dAT[2], dAL[2];
    clear(dAT);
    clear(dAL);
    float dD = 0.f;
    reverse_pairs<io_t, rec_t, VEC, CHAIN>(a, smem_u32(smem), params, D_lane, dAT, dAL, dD);

    // ---- per-(channel, state) sums: fold the CTA's warps through shared memory, then one atomic per value from warp 0
    constexpr int kSums = 17;
    float s[kSums];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            s[c * 4 + k * 2] = dAT[c][k].x; s[c * 4 + k * 2 + 1] = dAT[c][k].y;
            s[8 + c * 4 + k * 2] = dAL[c][k].x; s[8 + c * 4 + k * 2 + 1] = dAL[c][k].y;
        }
    s[16] = dD;
    float* const red = reinterpret_cast<float*>(smem);     // (2.2 KB per warp, of 12 that it has)
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSums; ++k) red[threadIdx.x * kSums + k] = s[k];
    __syncthreads();
    if (ln.r != 0) return;
    for (int w = 1; w < ln.nwarps; ++w)
#pragma unroll
        for (int k = 0; k < kSums; ++k) s[k] += red[(w * 32 + ln.lane) * kSums + k];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int n = 0; n < 4; ++n)
            if (c < ln.chv && n < ln.nv) {
                const long long idx = (long long)(ln.ch0 + c) * a.N + ln.n0 + n;
                // with A given as A_log the gradient asked for is d_A_log = d_A * A (A = -exp(A_log),
                // models/kernels/wavefront_cuda.py:72-73); the product is linear, so every CTA
                // scales its own partial sum
                const float sT = a.a_log ? load_A<io_t>(a.AT, idx, 1, true) : 1.f;
                const float sL = a.a_log ? load_A<io_t>(a.AL, idx, 1, true) : 1.f;
                atomicAdd(a.accAT + idx, s[c * 4 + n] * sT);
                atomicAdd(a.accAL + idx, s[8 + c * 4 + n] * sL);
            }
    if (o_ch < a.E) atomicAdd(a.accD + o_ch, s[16]);      // (two lanes each: one for each row)
}

// bf16 I/O: cast the fp32 accumulators into the caller's gradient tensors (d_AT / d_AL stay fp32 when
// they are gradients of the fp32 parameter A_log).  VEC: four states at a time (N and the pitch multiples of 4, tensors
// on 8 bytes).  Bound by its traffic then; one state at a time, with a 64-bit division for its pixel, took 11.4 us at
// 128 x 28 x 28 x 128 and 14.4 at 2 x 200 x 336 x 64, 6.6 and 7.2 now.
template <bool VEC>
__global__ void m2d_bwd_finalize(const float* __restrict__ acc, __nv_bfloat16* d_BT, __nv_bfloat16* d_BL, __nv_bfloat16* d_C, void* d_AT, void* d_AL,
                                 void* d_D, long long npn, int N, int pitch, long long en, int E, int a_log, int d_f32) {
    typedef __nv_bfloat16 io_t;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    if (VEC) {
        // (31 bits are enough: check_desc)
        const unsigned quads = (unsigned)(npn / 4), per = (unsigned)N / 4;
        for (unsigned k = (unsigned)tid; k < quads; k += (unsigned)nthreads) {
            const size_t at = pitch == N ? (size_t)k * 4 : (size_t)(k / per) * pitch + k % per * 4;
            const float4 v0 = __ldcs(reinterpret_cast<const float4*>(acc) + k), v1 = __ldcs(reinterpret_cast<const float4*>(acc + npn) + k),
                         v2 = __ldcs(reinterpret_cast<const float4*>(acc + 2 * npn) + k);
            *reinterpret_cast<uint2*>(d_BT + at) = make_uint2(pack_bf16x2(v0.x, v0.y), pack_bf16x2(v0.z, v0.w));
            *reinterpret_cast<uint2*>(d_BL + at) = make_uint2(pack_bf16x2(v1.x, v1.y), pack_bf16x2(v1.z, v1.w));
            *reinterpret_cast<uint2*>(d_C + at) = make_uint2(pack_bf16x2(v2.x, v2.y), pack_bf16x2(v2.z, v2.w));
        }
    } else {
        for (long long k = tid; k < npn; k += nthreads) {
            const long long at = pitch == N ? k : k / N * pitch + k % N;
            store1(d_BT, at, acc[k]);
            store1(d_BL, at, acc[npn + k]);
            store1(d_C, at, acc[2 * npn + k]);
        }
    }
    const float* accA = acc + 3 * npn;
    for (long long k = tid; k < en; k += nthreads) {
        if (a_log) {
            static_cast<float*>(d_AT)[k] = accA[k];
            static_cast<float*>(d_AL)[k] = accA[en + k];
        } else {
            store1(static_cast<io_t*>(d_AT), k, accA[k]);
            store1(static_cast<io_t*>(d_AL), k, accA[en + k]);
        }
    }
    for (long long k = tid; k < E; k += nthreads) {
        if (d_f32) static_cast<float*>(d_D)[k] = accA[2 * en + k];
        else store1(static_cast<io_t*>(d_D), k, accA[2 * en + k]);
    }
}

// Zero the columns of a wider buffer that d_BT, d_BL and d_C are: one pass when they are neighbours.  For callers that
// do not set M2D_SCAN_BC_ZEROED; the native block call does, and clears its whole buffer instead (a pitched memset of
// its 401408 rows at E = 64 takes 220 us more).
static bool zero_columns(const ScanArgs& a, const m2d_scan_desc* d, cudaStream_t st) {
    const size_t rows = (size_t)d->B * d->H * d->W, pitch = (size_t)a.acc_pitch * 4, width = (size_t)d->N * 4;
    if (a.accBL == a.accBT + d->N && a.accC == a.accBL + d->N) return cudaMemset2DAsync(a.accBT, pitch, 0, 3 * width, rows, st) == cudaSuccess;
    return cudaMemset2DAsync(a.accBT, pitch, 0, width, rows, st) == cudaSuccess && cudaMemset2DAsync(a.accBL, pitch, 0, width, rows, st) == cudaSuccess &&
           cudaMemset2DAsync(a.accC, pitch, 0, width, rows, st) == cudaSuccess;
}

typedef void (*SweepKernel)(const ScanArgs);

template <typename io_t>
static int launch_bwd(const m2d_scan_desc* d, const BwdPlan& pl, bool vec, cudaStream_t st) {
    // (a kernel by the type of its record, its kind of loads and whether its CTAs are chained)
    auto pick = [&](auto kernel) -> SweepKernel {
        auto loads = [&](auto rec, auto chain) { return vec ? kernel(rec, std::true_type{}, chain) : kernel(rec, std::false_type{}, chain); };
        if (pl.chain > 1) return loads(float{}, std::true_type{});           // (fp32, whatever few_images says: kLargeScratch)
        return pl.wide || sizeof(io_t) == 4 ? loads(float{}, std::false_type{}) : loads(io_t{}, std::false_type{});
    };
    const BwdLayout L = bwd_layout(d, pl);
    char* ws = static_cast<char*>(d->workspace);
    ScanArgs a;
    fill_common_args(a, d, pl);
    a.status = reinterpret_cast<int*>(ws);
    a.ring = reinterpret_cast<float4*>(ws + L.edge);
    size_t zero_bytes = L.acc_bytes ? kStatusBytes + L.acc_bytes : sizeof(int);
    if (pl.wave) {
        const size_t edge = wave_edge_bytes(d, pl, true);
        a.bnd = reinterpret_cast<float4*>(ws + L.edge);
        a.bnd_up = reinterpret_cast<float4*>(ws + L.edge + edge);
        a.bnd_rows = wave_rows(pl, true);
        if (pl.chain > 1) zero_bytes = L.edge + 2 * edge;
    } else if (pl.chain > 1) {
        const size_t states = pair_edge_bytes(d, pl.states);
        a.bnd = reinterpret_cast<float4*>(ws + L.edge);
        a.bnd_up = reinterpret_cast<float4*>(ws + L.edge + states);
        zero_bytes = L.edge + states + pair_edge_bytes(d, pl);
    }
    if (cudaMemsetAsync(ws, 0, zero_bytes, st) != cudaSuccess) return M2D_ERR_LAUNCH;
    a.gy = d->gy;
    a.hs = reinterpret_cast<float4*>(ws + L.hs);
    a.d_x = d->d_x; a.d_dT = d->d_dT; a.d_dL = d->d_dL;
    const size_t npn = (size_t)d->B * d->H * d->W * d->N, en = (size_t)d->E * d->N;
    if (d->dtype == M2D_F32) {
        a.acc_pitch = d->d_BC_pitch ? (int)d->d_BC_pitch : d->N;
        a.accBT = static_cast<float*>(d->d_BT); a.accBL = static_cast<float*>(d->d_BL); a.accC = static_cast<float*>(d->d_C);
        a.accAT = static_cast<float*>(d->d_AT); a.accAL = static_cast<float*>(d->d_AL); a.accD = static_cast<float*>(d->d_D);
        // the six accumulated outputs start from zero; a caller that carved the three per-pixel ones
        // out of one buffer and the three per-channel ones out of another, in this order, gets two
        // memsets instead of six (they are 3 us each against a 200 us kernel at the smallest stage)
        const bool pitched = a.acc_pitch != d->N;
        const bool big_adjacent = !pitched && a.accBL == a.accBT + npn && a.accC == a.accBL + npn;
        const bool small_adjacent = a.accAL == a.accAT + en && a.accD == a.accAL + en;
        bool ok;
        if (big_adjacent && !(d->flags & M2D_SCAN_BC_ZEROED) && a.accAT == a.accC + npn && small_adjacent) {
            ok = cudaMemsetAsync(a.accBT, 0, (3 * npn + 2 * en + (size_t)d->E) * 4, st) == cudaSuccess;
        } else {
            ok = (d->flags & M2D_SCAN_BC_ZEROED) ? true : pitched ? zero_columns(a, d, st) : big_adjacent ? cudaMemsetAsync(a.accBT, 0, 3 * npn * 4, st) == cudaSuccess
                              : (cudaMemsetAsync(a.accBT, 0, npn * 4, st) == cudaSuccess && cudaMemsetAsync(a.accBL, 0, npn * 4, st) == cudaSuccess &&
                                 cudaMemsetAsync(a.accC, 0, npn * 4, st) == cudaSuccess);
            ok = ok && (small_adjacent ? cudaMemsetAsync(a.accAT, 0, (2 * en + (size_t)d->E) * 4, st) == cudaSuccess
                                       : (cudaMemsetAsync(a.accAT, 0, en * 4, st) == cudaSuccess && cudaMemsetAsync(a.accAL, 0, en * 4, st) == cudaSuccess &&
                                          cudaMemsetAsync(a.accD, 0, (size_t)d->E * 4, st) == cudaSuccess));
        }
        if (!ok) return M2D_ERR_LAUNCH;
    } else {
        float* acc = reinterpret_cast<float*>(ws + L.acc);
        a.acc_pitch = d->N;
        a.accBT = acc; a.accBL = acc + npn; a.accC = acc + 2 * npn;
        a.accAT = acc + 3 * npn; a.accAL = a.accAT + en; a.accD = a.accAL + en;
    }
    Plan p = pl;
    if (pl.wave) {
        a.acc_vec = d->N % 4 == 0 && a.acc_pitch % 4 == 0 && aligned(a.accBT, 16) && aligned(a.accBL, 16) && aligned(a.accC, 16);
        p.smem = WaveSmem<io_t, 2, true>::kBytes;
    }
    if (!pl.wave) {
        a.Rb = pl.states.Rb;
        a.nbands = pl.states.nbands;
        a.chain = pl.states.chain;
        const int rc = launch_sweep_kernel(pick([](auto rec, auto v, auto ch) { return m2d_bwd_states_kernel<io_t, decltype(rec), decltype(v)::value, decltype(ch)::value>; }),
                                           a, pl.states, st);
        if (rc != M2D_OK) return rc;
        a.Rb = pl.Rb;
        a.nbands = pl.nbands;
        a.chain = pl.chain;
    }
    const int rc = launch_sweep_kernel(pl.wave ? (vec ? m2d_bwd_wave_kernel<io_t, true> : m2d_bwd_wave_kernel<io_t, false>)
                                               : pick([](auto rec, auto v, auto ch) { return m2d_bwd_kernel<io_t, decltype(rec), decltype(v)::value, decltype(ch)::value>; }),
                                       a, p, st);
    if (rc != M2D_OK) return rc;
    if constexpr (sizeof(io_t) == 2) {
        const int pitch = d->d_BC_pitch ? (int)d->d_BC_pitch : d->N;
        const bool quads = d->N % 4 == 0 && pitch % 4 == 0 && aligned(d->d_BT, 8) && aligned(d->d_BL, 8) && aligned(d->d_C, 8);
        // a thread per quad of B and C or per (channel, state), whichever are more: a 7x7 image of 512 channels has 196 of those
        // and 8192 of these.  A grid for the quads alone / this one, us: 1x7x7x512 18.4 / 2.8, 1x5x5x576 19.8 / 2.4,
        // 3x7x7x512 7.7 / 2.8, 4x14x14x384 3.5 / 2.8, 128x28x28x128 6.3 / 6.3
        const size_t fit = (size_t)sm_count() * 8, items = std::max(quads ? npn / 4 : npn, en);
        const int fin_blocks = (int)std::min((items + 255) / 256, fit);
        (quads ? m2d_bwd_finalize<true> : m2d_bwd_finalize<false>)<<<fin_blocks, 256, 0, st>>>(
            a.accBT, static_cast<io_t*>(d->d_BT), static_cast<io_t*>(d->d_BL), static_cast<io_t*>(d->d_C), d->d_AT, d->d_AL, d->d_D, (long long)npn,
            d->N, pitch, (long long)en, d->E, a.a_log, a.d_f32);
        if (cudaGetLastError() != cudaSuccess) return M2D_ERR_LAUNCH;
    }
    return M2D_OK;
}

}  // namespace m2d

extern "C" uint64_t m2d_scan_bwd_workspace(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, true, false) != M2D_OK) return 0;
    return m2d::plan_bwd(d).scratch;
}

extern "C" int64_t m2d_scan_bwd_status_offset(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, true, false) != M2D_OK) return -1;
    return 0;
}

extern "C" int m2d_scan_bwd_chain(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, true, false) != M2D_OK) return 0;
    return m2d::plan_bwd(d).chain;
}

extern "C" int m2d_scan_bwd(const m2d_scan_desc* d, void* stream) {
    int rc = m2d::check_desc(d, true, true);
    if (rc != M2D_OK) return rc;
    const m2d::BwdPlan pl = m2d::plan_bwd(d);
    if (!d->workspace || d->workspace_bytes < pl.scratch || (reinterpret_cast<uintptr_t>(d->workspace) & 255))
        return M2D_ERR_WORKSPACE;
    const bool vec = m2d::vector_ok(d, true);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (d->dtype == M2D_F32) return m2d::launch_bwd<float>(d, pl, vec, st);
    return m2d::launch_bwd<__nv_bfloat16>(d, pl, vec, st);
}
