// What every scan kernel gets: the argument block and the loads of the parameters.
//
// Math per cell (i,j), per channel e and state n (reference: models/kernels/wf_cuda/wf_cuda.cu:41-69
// for the recurrence, models/kernels/wavefront_cuda.py:156 for the readout):
//     gT = exp(dT*AT)   gL = exp(dL*AL)   uT = dT*BT*x   uL = dL*BL*x
//     h  = wL*(gL*h_left + uL) + wT*(gT*h_top + uT)
//     (wL,wT) = (1,0) on row 0, (0,1) on column 0 below row 0, (1/2,1/2) inside
//     y  = sum_n h*C + x*D
// The weights are folded into the exponent (exp2(dT*AT*log2e + log2 wT)).
//
// And its adjoint, with lam the total adjoint of h and kap = c*lam, c the weight of the cell's inputs
// (reference: models/kernels/wf_cuda/wf_cuda.cu:108-160; the reference's omega buffer equals lam/2 and
// carries no extra information):
//     lam[i,j] = gy*C + gL[i,j+1]*kap[i,j+1] + gT[i+1,j]*kap[i+1,j]
// Each cell computes its own gates once and hands pT = gT*kap to the row above and pL = gL*kap to the cell
// on its left.  All gradient arithmetic the reference does afterwards in PyTorch
// (models/kernels/wavefront_cuda.py:97-139, :176-178, :193-194) is fused:
//     dzT = pT*h[i-1,j]                 dzL = pL*h[i,j-1]
//     d_AT[e,n] += dzT*dT               d_AL[e,n] += dzL*dL
//     d_dT = sum_n dzT*AT + mT*x*sum_n kap*BT      (mT = i>0)
//     d_dL = sum_n dzL*AL + mL*x*sum_n kap*BL      (mL = j>0 or i==0)
//     d_x  = mT*dT*sum_n kap*BT + mL*dL*sum_n kap*BL + gy*D
//     d_BT[n] = sum_e mT*kap*dT*x       d_BL[n] = sum_e mL*kap*dL*x        d_C[n] = sum_e gy*h
//     d_D[e] += gy*x
#pragma once

#include <type_traits>

#include "common.cuh"

namespace m2d {

struct ScanArgs {
    int B, H, W, E, N;
    const void *x, *dT, *dL, *AT, *AL, *BT, *BL, *C, *D;
    long long pBT, pBL, pC;   // pixel pitch (elements) of BT, BL, C
    void* y;
    int dir;                  // +1: scan from the top-left corner; -1: from the bottom-right one (same memory, walked backwards)
    float4* ring;             // batch kernels: per-CTA band-boundary ring, [cta][W][2][32] float4
    int Rb, nbands;
    // ---- wave kernels and chained batch sweeps: CTA c of a chain of `chain` CTAs owns the bands q = c, c + chain, ... of
    // its images; the last row of band q reaches band q+1 through `bnd`
    int chain;                // 1 = one CTA per image
    float4* bnd;              // boundary rows, see wave_fwd.cuh; chained batch sweeps: [image][group][band][W][2][32] float4
    int bnd_rows;             // wave kernels: rows kept per (chain, channel group), one per band or two in turn
    int* status;              // nonzero if a wait for a boundary row gave up (results are then invalid); never null
    int* host_flag;           // the same news in host memory, where the next call sees it without synchronising; may be null
    int wait_limit;           // polls before such a wait gives up
    int withhold;             // test hook: the first band of image 0 never hands over its last row
    int mute_up;              // test hook: this band (0: none) hands nothing up in the adjoint sweep
    int shorten;              // test hook: half as many CTAs per image as planned (host side only)
    int act;                  // forward only: 1 = apply GELU (erf form) to y before it is stored
    int a_log;                // AT / AL hold the fp32 parameter A_log (A = -exp(A_log)); d_AT / d_AL are then fp32 d_A_log
    int d_f32;                // D and d_D are fp32 whatever the I/O type
    // ---- backward only ----
    const void* gy;
    float4* hs;               // state record; batch kernels: [group][pixel] blocks of two (fp32) or one (bf16) float4 per lane
    // fp32 accumulators of the reduced gradients, zeroed before the kernel.  For fp32 I/O they are
    // the caller's gradient tensors themselves; for bf16 I/O they live in the workspace.
    float *accBT, *accBL, *accC;   // [B*H*W] rows of N values at a pitch of acc_pitch
    int acc_pitch;
    int acc_vec;                   // wave kernel: rows of accBT, accBL, accC take 16-byte accesses
    float4* bnd_up;                // as bnd, for the adjoint sweep
    float *accAT, *accAL;          // [E][N]
    float* accD;                   // [E]
    void *d_x, *d_dT, *d_dL;
};
// Flat pixel index in memory of scan position (i, j) of image b.  In the reverse direction the
// scan's cell (i, j) is the memory's pixel (H-1-i, W-1-j), i.e. the image's pixels in opposite order.
__device__ __forceinline__ int scan_pixel(const ScanArgs& a, int b, int i, int j) {
    const int p = i * a.W + j;
    return b * a.H * a.W + (a.dir > 0 ? p : a.H * a.W - 1 - p);
}

// float4 units of one (cell, warp) block of the state record
template <typename rec_t> struct HsBlock { static constexpr int f4 = sizeof(rec_t) == 2 ? 32 : 64; };

// Element (e, n) of AT / AL as a float.  With `a_log` the tensors hold the fp32 parameter A_log and
// A = -exp(A_log), rounded to the I/O type the way the reference's cast does
// (models/kernels/wavefront_cuda.py:72-73, :89-90); `exact` skips that rounding (used for the
// gradient d_A_log = d_A * A, where the reference multiplies by the fp32 value).
template <typename io_t>
__device__ __forceinline__ float load_A(const void* A, long long idx, int a_log, bool exact = false) {
    if (!a_log) return load1(static_cast<const io_t*>(A), idx);
    const float v = -expf(__ldg(static_cast<const float*>(A) + idx));
    if (sizeof(io_t) == 2 && !exact) return __bfloat162float(__float2bfloat16_rn(v));
    return v;
}

// D[e] as a float; an fp32 parameter is rounded to the I/O type the way the caller's cast would.
template <typename io_t>
__device__ __forceinline__ float load_D(const ScanArgs& a, int e) {
    if (!a.d_f32) return load1(static_cast<const io_t*>(a.D), e);
    const float v = __ldg(static_cast<const float*>(a.D) + e);
    return sizeof(io_t) == 2 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
}

template <typename io_t>
__device__ __forceinline__ void stage_params(float4* dst, const void* AT, const void* AL, int N, int ch0, int chv, int n0, int nv, int lane,
                                             int a_log) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        float t[4], l[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const bool ok = (c < chv) && (n < nv);
            t[n] = ok ? load_A<io_t>(AT, (long long)(ch0 + c) * N + n0 + n, a_log) * kLog2e : 0.f;
            l[n] = ok ? load_A<io_t>(AL, (long long)(ch0 + c) * N + n0 + n, a_log) * kLog2e : 0.f;
        }
        dst[c * 32 + lane] = make_float4(t[0], t[1], t[2], t[3]);
        dst[64 + c * 32 + lane] = make_float4(l[0], l[1], l[2], l[3]);
    }
}

constexpr int kWaitPolls = 1 << 22;     // polls before a wait for another CTA gives up

}  // namespace m2d
