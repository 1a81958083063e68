// Shared device helpers and the launch plan for the sm_100a wavefront-scan kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "m2d_scan.h"

namespace m2d {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr int kGroup = 16;      // channels owned by one warp of the batch kernels (8 lanes x 2 channels)
constexpr int kMaxN = 16;       // states owned by one warp   (4 lanes x 4 states)
constexpr int kSlotF4 = 64;     // float4 per (cell, warp) block of states: 2 channels x 32 lanes

__device__ __forceinline__ float ex2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Predicated forms (no branch, no reconvergence point): the copy / store happens iff `on`.
__device__ __forceinline__ void cp_async16_if(bool on, unsigned smem_addr, const void* gmem) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}"
                 ::"r"(smem_addr), "l"(gmem), "r"((int)on) : "memory");
}
__device__ __forceinline__ void cp_async8_if(bool on, unsigned smem_addr, const void* gmem) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p cp.async.ca.shared.global [%0], [%1], 8;\n\t}"
                 ::"r"(smem_addr), "l"(gmem), "r"((int)on) : "memory");
}
// Unpredicated forms, for call sites that branch on a loop-invariant condition themselves.
__device__ __forceinline__ void cp_async16(unsigned smem_addr, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(unsigned smem_addr, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr), "l"(gmem) : "memory");
}
// A 1 KiB block: two 16-byte pieces per lane, 512 bytes apart.
__device__ __forceinline__ void cp_async_block(unsigned smem_addr, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n\tcp.async.cg.shared.global [%0+512], [%1+512], 16;"
                 ::"r"(smem_addr), "l"(gmem) : "memory");
}
// gelu(y), erf form: y/2 (1 + erf(y/sqrt 2)) = max(y, 0) - |y|/2 erfc(|y|/sqrt 2), with log2(erfc) as a polynomial on
// [0, 6] (weighted least squares, Lawson's iteration; erfc(6) = 2e-17 stands for what lies beyond).  Largest
// error 2.4e-7 over |y| <= 8, 4.5e-7 with erff and 1e-5 relative for negative y, where 1 + erf cancels; and no
// branch: one value per lane and cell, this is 16 instructions in the readout against about 35.
__device__ __forceinline__ float gelu_erf(float y) {
    const float m = fminf(fabsf(y), 8.4852814f), t = m * 0.70710678f;
    float q = 2.9805828e-6f;
    q = fmaf(q, t, -5.1289102e-5f);
    q = fmaf(q, t, 3.4886587e-4f);
    q = fmaf(q, t, -9.5030182e-4f);
    q = fmaf(q, t, -1.9680441e-3f);
    q = fmaf(q, t, 2.9599719e-2f);
    q = fmaf(q, t, -0.14927331f);
    q = fmaf(q, t, -0.91819334f);
    q = fmaf(q, t, -1.6279321f);
    q = fmaf(q, t, 4.0780279e-7f);
    return fmaf(-0.5f * m, ex2(q), fmaf(0.5f, fabsf(y), 0.5f * y));      // (a NaN stays one: |y| + y, not fmaxf)
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ unsigned pack_bf16x2(float lo, float hi) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// ---- input staging in shared memory (batch kernels) ------------------------------------------------
// A cell: 28 slots of 16 bytes, x[4] dT[4] dL[4] gy[4] (one slot per four channels), BT[4] BL[4] C[4] (one slot per four
// states).  A slot holds four elements of the I/O type (fp32: 16 bytes, bf16: the first 8 bytes).
constexpr int kCellSlots = 28;

// ---- scalar element loads / stores --------------------------------------------------------------
__device__ __forceinline__ float bf16_bits_to_float(unsigned short b) { return __uint_as_float(static_cast<unsigned>(b) << 16); }
__device__ __forceinline__ float load1(const float* __restrict__ p, long long off) { return __ldg(p + off); }
__device__ __forceinline__ float load1(const __nv_bfloat16* __restrict__ p, long long off) {
    return bf16_bits_to_float(__ldg(reinterpret_cast<const unsigned short*>(p) + off));
}
__device__ __forceinline__ void store1(float* p, long long off, float v) { p[off] = v; }
__device__ __forceinline__ void store1(__nv_bfloat16* p, long long off, float v) { p[off] = __float2bfloat16_rn(v); }

// Sum four per-channel partials over the 4 nq lanes.  On return lane nq holds the total of
// channel index nq of its 4-channel block (so lane l of the warp holds channel l of the group).
__device__ __forceinline__ float reduce_states(float v0, float v1, float v2, float v3, int nq) {
    const bool hi2 = (nq & 2) != 0;
    float k0 = hi2 ? v2 : v0, k1 = hi2 ? v3 : v1;
    const float s0 = hi2 ? v0 : v2, s1 = hi2 ? v1 : v3;
    k0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    k1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    const bool hi1 = (nq & 1) != 0;
    const float k = hi1 ? k1 : k0, s = hi1 ? k0 : k1;
    return k + __shfl_xor_sync(0xffffffffu, s, 1);
}

// The per-(channel,state) parameters A*log2(e) of the CTA's 16 channels live in shared memory
// behind everything else: [AT | AL][2 channels][32 lanes] float4 (2 KiB), read block by block.
constexpr int kParamF4 = 2 * 2 * 32;

// Shared memory of the batch kernels (sweep_pairs.cuh), in front of the parameters.
constexpr int kRot = 1024;                                                // one buffer of an area
constexpr int kFwdBlock = 2 * 3 * kRot, kBwdBlock = 4 * 3 * kRot;         // per warp: S, T (, HA, HB)
__host__ __device__ inline size_t pairs_fwd_smem_bytes(int warps) { return (size_t)warps * kFwdBlock + 3 * kRot; }
__host__ __device__ inline size_t pairs_bwd_smem_bytes(int warps) { return (size_t)warps * kBwdBlock + 2 * 3 * kRot; }

// Host-side launch plan shared by the workspace queries and the launches.
struct Plan {
    int groups;        // ceil(E / channels of a CTA)
    int warps;         // warps per CTA
    int Rb;            // rows per band
    int nbands;        // ceil(H / Rb)
    int grid_x;        // image chains per channel group; chain k walks images k, k + grid_x, ...
    int chain;         // CTAs per chain (> 1 when there are far fewer images than SMs)
    int wave;          // channels per lane of the wave kernel (several CTAs per image), or 0
    size_t smem;       // dynamic shared memory per CTA
    size_t scratch;    // workspace bytes
};

}  // namespace m2d
