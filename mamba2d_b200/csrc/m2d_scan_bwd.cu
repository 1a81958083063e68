// Backward entry point of the wavefront scan: recompute sweep + adjoint sweep in one kernel,
// followed by a small kernel that casts the fp32 accumulators of the reduced gradients.
#include <algorithm>

#include "launch.cuh"
#include "sweep_rows.cuh"
#include "wave_bwd.cuh"

// Row-warps per CTA of the backward kernel (two CTAs per SM): the register budget per thread follows
// from it (6 warps: 168 registers).
#ifndef M2D_BWD_MAXW
#define M2D_BWD_MAXW 6
#endif
#ifndef M2D_BWD_MINB
#define M2D_BWD_MINB 2
#endif

namespace m2d {

// Workspace layout of the backward pass (all regions 256-byte aligned):
//   status   one word, nonzero if a wait between CTAs gave up
//   acc      bf16 I/O only: fp32 accumulators 3 x [B*H*W][N] | 2 x [E][N] | [E], zeroed before the
//            main kernel (with the status word, in one memset) and cast by a second kernel.  With fp32 I/O
//            the kernel accumulates straight into the caller's (zeroed) gradient tensors and this region is empty.
//   edge     batch: per-CTA band-boundary ring, ctas*W*2 KiB (only if nbands > 1); wave: the boundary rows
//            of the recompute sweep (h, downwards) and of the adjoint sweep (pT, upwards)
//   hs       state record written by the recompute sweep: batch B*groups*H*W*2 KiB (1 KiB with bf16 I/O), wave
//            512*C bytes per (list, warp, band, step)
struct BwdLayout {
    size_t edge, hs, acc, acc_bytes, total;
};

inline BwdLayout bwd_layout(const m2d_scan_desc* d, const Plan& p) {
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
    else if (p.nbands > 1) off += align256((size_t)p.grid_x * p.groups * d->W * kSlotF4 * sizeof(float4));
    L.hs = off;
    if (p.wave) off += align256((size_t)p.grid_x * p.groups * p.warps * p.nbands * (d->W + 7) * p.wave * 512);
    else off += align256((size_t)d->B * p.groups * d->H * d->W * (d->dtype == M2D_F32 ? 128 : 64) * sizeof(float4));
    L.total = off;
    return L;
}

inline Plan plan_bwd(const m2d_scan_desc* d) {
    // Batch or wave, as in plan_fwd.  Measured times per step of both sweeps together, whatever the I/O type: 2.45 us in
    // batch mode with two CTAs per SM, 1.95 us with one, 1.2 us in the wave kernel with two channels per lane (four
    // spill and are slower at every size measured).  56x56x64: wave up to batch 32, 581 against 738 us.
    Plan p{};
    double best = 1e30;
    if (d->W >= 3) {
        p = plan_best(d, M2D_BWD_MAXW, 2 * M2D_BWD_MAXW);
        p.smem = rows_bwd_smem_bytes(p.warps) + kParamF4 * sizeof(float4);
        best = ((long long)p.grid_x * p.groups > sm_count() ? 2.45 : 1.95) * batch_steps(d, p);
    }
    const Plan w = plan_wave(d, 2);
    if (1.2 * wave_steps(d, w) + 10.0 < best) p = w;
    p.scratch = bwd_layout(d, p).total;
    return p;
}

// Few images: several CTAs per image.
template <typename io_t, bool VEC>
__global__ void __launch_bounds__(256, 1) m2d_bwd_wave_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    wave_backward<io_t, 2, VEC>(a, reinterpret_cast<char*>(smem));
}

// Batch mode (one CTA per image and channel group): both sweeps written as nested loops.
template <typename io_t, bool VEC>
__global__ void __launch_bounds__(M2D_BWD_MAXW * 32, M2D_BWD_MINB) m2d_bwd_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    const int lane = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    const int cq = lane >> 2, nq = lane & 3;
    const int g = blockIdx.y;
    const int ch0 = g * kGroup + cq * 4, n0 = nq * 4;
    const int chv = min(4, max(0, a.E - ch0));
    const int nv = min(4, max(0, a.N - n0));

    const int total = (int)(rows_bwd_smem_bytes(nwarps) / sizeof(float4));
    for (int k = threadIdx.x; k < total; k += blockDim.x) smem[k] = make_float4(0.f, 0.f, 0.f, 0.f);

    const int ch_own = g * kGroup + lane;
    const float D_own = ch_own < a.E ? load_D<io_t>(a, ch_own) : 0.f;
    float dAT[4][4], dAL[4][4], dD[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        dD[c] = 0.f;
#pragma unroll
        for (int n = 0; n < 4; ++n) dAT[c][n] = dAL[c][n] = 0.f;
    }
    __syncthreads();
    float4* const params = reinterpret_cast<float4*>(reinterpret_cast<char*>(smem) + rows_bwd_smem_bytes(nwarps));
    if (threadIdx.x < 32) stage_params<io_t>(params, a.AT, a.AL, a.N, ch0, chv, n0, nv, lane, a.a_log);
    __syncthreads();

    for (int b = (int)blockIdx.x; b < a.B; b += (int)gridDim.x) {
        forward_rows<io_t, VEC, true, false>(a, smem, params, D_own, b, 0, 1);
        reverse_rows<io_t, VEC>(a, smem, params, D_own, dAT, dAL, dD, b);
    }

    // ---- per-(channel,state) sums: fold the CTA's row-warps through shared memory, then one
    //      atomic per value from warp 0 ----------------------------------------------------------
    float* red = reinterpret_cast<float*>(smem);        // reuse: needs 36 floats per thread
    const int slot = (int)rows_handoff_f4(nwarps) * 4;   // floats available
    const bool fits = (int)blockDim.x * 36 <= slot;
    if (fits && nwarps > 1) {
        float* mine = red + (size_t)threadIdx.x * 36;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int n = 0; n < 4; ++n) { mine[c * 4 + n] = dAT[c][n]; mine[16 + c * 4 + n] = dAL[c][n]; }
            mine[32 + c] = dD[c];
        }
        __syncthreads();
        if (r == 0) {
            for (int w = 1; w < nwarps; ++w) {
                const float* o = red + (size_t)(w * 32 + lane) * 36;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
#pragma unroll
                    for (int n = 0; n < 4; ++n) { dAT[c][n] += o[c * 4 + n]; dAL[c][n] += o[16 + c * 4 + n]; }
                    dD[c] += o[32 + c];
                }
            }
        }
    }
    if (r == 0 || !(fits && nwarps > 1)) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (c < chv) {
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    if (n < nv) {
                        const long long idx = (long long)(ch0 + c) * a.N + n0 + n;
                        // with A given as A_log the gradient asked for is d_A_log = d_A * A (A = -exp(A_log),
                        // models/kernels/wavefront_cuda.py:72-73); the product is linear, so every CTA
                        // scales its own partial sum
                        const float sT = a.a_log ? load_A<io_t>(a.AT, idx, 1, true) : 1.f;
                        const float sL = a.a_log ? load_A<io_t>(a.AL, idx, 1, true) : 1.f;
                        atomicAdd(a.accAT + idx, dAT[c][n] * sT);
                        atomicAdd(a.accAL + idx, dAL[c][n] * sL);
                    }
                }
                if (nq == 0) atomicAdd(a.accD + ch0 + c, dD[c]);
            }
        }
    }
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

template <typename io_t>
static int launch_bwd(const m2d_scan_desc* d, const Plan& pl, bool vec, cudaStream_t st) {
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
    const int rc = launch_sweep_kernel(pl.wave ? (vec ? m2d_bwd_wave_kernel<io_t, true> : m2d_bwd_wave_kernel<io_t, false>)
                                               : (vec ? m2d_bwd_kernel<io_t, true> : m2d_bwd_kernel<io_t, false>), a, p, st);
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
    const m2d::Plan pl = m2d::plan_bwd(d);
    if (!d->workspace || d->workspace_bytes < pl.scratch || (reinterpret_cast<uintptr_t>(d->workspace) & 255))
        return M2D_ERR_WORKSPACE;
    const bool vec = m2d::vector_ok(d, true);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (d->dtype == M2D_F32) return m2d::launch_bwd<float>(d, pl, vec, st);
    return m2d::launch_bwd<__nv_bfloat16>(d, pl, vec, st);
}
