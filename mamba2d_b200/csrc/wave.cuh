// Pieces shared by the wave kernels: forward and backward for few images on large maps.
//
// Lane layout.  A warp owns C channels x 16 states and EIGHT consecutive rows (a band): lane = (r, nq) =
// (lane >> 2, lane & 3) walks row r of the band and owns C channels x states [4nq, 4nq+4) of it, one
// column per step, r columns behind lane row 0.  The eight rows of a step are cells of one anti-diagonal,
// so the cell above was finished by lane - 4 in the step before and reaches this lane through a slot of
// shared memory that only this warp uses: the wavefront runs inside a warp.  Sums over states finish
// across the four nq lanes, sums over channels across the warps of the CTA.
//
// A CTA is eight such warps on the same band and C * 8 neighbouring channels.  The inputs of kChunk steps
// are staged in shared memory with cp.async, warp w fetching the cells of lane row w for all of them, a
// few chunks ahead; the block barrier that hands a chunk over is the only one.
//
// Bands of an image belong to different CTAs.  The last row of a band reaches the next band through global
// memory that the host has zeroed: states are stored with their bits inverted, and no arithmetic returns the
// NaN that would then read as zero.  The consumer loads the columns it will need one chunk ahead and sees
// from the values themselves whether they are there.
// One trip to L2 per chunk, off the critical path, and no flags, fences or counters.  The wait for a value
// that is not there yet is bounded.
#pragma once

#include "common.cuh"
#include "sweep_fwd.cuh"

namespace m2d {

constexpr int kWaveRows = 8;
constexpr int kWaveWarps = 8;
constexpr int kChunk = 4;      // steps per staged chunk; boundary columns move in the same units
constexpr int kStages = 4;     // chunk buffers: inputs are requested three chunks ahead (a chunk of a lone CTA takes
                               // about as long as a trip to HBM)

template <int C> constexpr int kEdgeFloats = 16 * C;        // boundary state per (warp, column)
template <int C> constexpr int kSlotBytes = (kWaveRows + 1) * kEdgeFloats<C> * 5;

// One staged cell: x | dT | dL (| gy) of the CTA's channels, then BT | BL | C of the 16 states.
template <typename io_t, int C, bool GY> struct StageLayout {
    static constexpr int kCh = C * kWaveWarps;
    static constexpr int kTensors = GY ? 4 : 3;
    static constexpr int kElems = kTensors * kCh + 48;
    // neighbouring rows fall into different banks: an odd multiple of the 16 states' bytes
    static constexpr int kPlain = kElems * (int)sizeof(io_t), kRow = 16 * (int)sizeof(io_t);
    static constexpr int kCellBytes = kPlain / kRow % 2 ? kPlain : kPlain + kRow;
    static constexpr int kStepBytes = kCellBytes * kWaveRows;
    static constexpr int kBytes = kStages * kChunk * kStepBytes;
    static constexpr int kPieces = kElems / 4;                       // pieces of four elements
};

__device__ __forceinline__ float2 bf2_to_float2(unsigned u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }

// K staged elements as floats, channels (or states) in pairs.
template <typename io_t, int K> __device__ __forceinline__ void read_staged(unsigned addr, float2 (&o)[K / 2]);
template <> __device__ __forceinline__ void read_staged<float, 4>(unsigned addr, float2 (&o)[2]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0].x), "=f"(o[0].y), "=f"(o[1].x), "=f"(o[1].y) : "r"(addr));
}
template <> __device__ __forceinline__ void read_staged<float, 2>(unsigned addr, float2 (&o)[1]) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(o[0].x), "=f"(o[0].y) : "r"(addr));
}
template <> __device__ __forceinline__ void read_staged<__nv_bfloat16, 4>(unsigned addr, float2 (&o)[2]) {
    unsigned u, v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(u), "=r"(v) : "r"(addr));
    o[0] = bf2_to_float2(u);
    o[1] = bf2_to_float2(v);
}
template <> __device__ __forceinline__ void read_staged<__nv_bfloat16, 2>(unsigned addr, float2 (&o)[1]) {
    unsigned u;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(u) : "r"(addr));
    o[0] = bf2_to_float2(u);
}

// One row (C channels of one state) of a lane's state block.
__device__ __forceinline__ void lds_vec(unsigned addr, float2 (&o)[2]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0].x), "=f"(o[0].y), "=f"(o[1].x), "=f"(o[1].y) : "r"(addr) : "memory");
}
__device__ __forceinline__ void lds_vec(unsigned addr, float2 (&o)[1]) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(o[0].x), "=f"(o[0].y) : "r"(addr) : "memory");
}
__device__ __forceinline__ void sts_vec(unsigned addr, const float2 (&v)[2]) {
    asm volatile("st.shared.v4.f32 [%4], {%0, %1, %2, %3};" ::"f"(v[0].x), "f"(v[0].y), "f"(v[1].x), "f"(v[1].y), "r"(addr) : "memory");
}
__device__ __forceinline__ void sts_vec(unsigned addr, const float2 (&v)[1]) {
    asm volatile("st.shared.v2.f32 [%2], {%0, %1};" ::"f"(v[0].x), "f"(v[0].y), "r"(addr) : "memory");
}
// One element, stored where `on`, without a branch.
__device__ __forceinline__ void store_if(bool on, float* p, float v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"((int)on) : "memory");
}
__device__ __forceinline__ void store_if(bool on, __nv_bfloat16* p, float v) {
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.b16 [%0], %1;\n\t}" ::"l"(p), "h"(*reinterpret_cast<const unsigned short*>(&b)), "r"((int)on) : "memory");
}
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float lane_of(const float2 (&v)[2], int n) { return (n & 1) ? v[n >> 1].y : v[n >> 1].x; }

// Sum C per-channel partials over the four nq lanes.  C == 4: lane nq returns channel nq; C == 2: lane nq
// returns channel nq >> 1.
__device__ __forceinline__ float wave_reduce(const float2 (&v)[2], int nq) { return reduce_states(v[0].x, v[0].y, v[1].x, v[1].y, nq); }
__device__ __forceinline__ float wave_reduce(const float2 (&v)[1], int nq) {
    const bool hi = (nq & 2) != 0;
    float k = hi ? v[0].y : v[0].x;
    k += __shfl_xor_sync(0xffffffffu, hi ? v[0].x : v[0].y, 2);
    return k + __shfl_xor_sync(0xffffffffu, k, 1);
}

// Load 16 bytes another CTA may be writing, past L1.
__device__ __forceinline__ uint4 load_shared_line(const void* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// Boundary states in global memory have their bits inverted: zero means "not written yet" (it would stand
// for the NaN 0xffffffff; the NaNs of arithmetic are 0x7fffffff).
__device__ __forceinline__ bool is_set(const uint4& v) { return v.x != 0 && v.y != 0 && v.z != 0 && v.w != 0; }
__device__ __forceinline__ uint4 inverted(const uint4& v) { return make_uint4(~v.x, ~v.y, ~v.z, ~v.w); }

// Staging of one lane row's cells by one warp: lanes 0..23 copy x, dT, dL (8 pieces of four channels each
// when C == 4), the others BT and BL; the rest (C, gy) goes with a second copy per step.
template <typename io_t, int C, bool GY, bool VEC>
struct Stager {
    typedef StageLayout<io_t, C, GY> L;
    static constexpr int kCopies = (L::kPieces + 31) / 32;
    const char* base[kCopies];
    int pitch[kCopies], dst[kCopies], nvalid[kCopies];
    __device__ __forceinline__ void init(const ScanArgs& a, int chbase, int lane) {
#pragma unroll
        for (int k = 0; k < kCopies; ++k) {
            const int p = lane + 32 * k;
            constexpr int per = L::kCh / 4;
            dst[k] = p * 4 * (int)sizeof(io_t);
            if (p < L::kTensors * per) {
                const int t = p / per, ch = chbase + (p % per) * 4;
                const void* b = t == 0 ? a.x : (t == 1 ? a.dT : (t == 2 ? a.dL : a.gy));
                base[k] = static_cast<const char*>(b) + (size_t)ch * sizeof(io_t);
                pitch[k] = a.E;
                nvalid[k] = min(4, a.E - ch);
            } else {
                const int s = p - L::kTensors * per, t = s / 4, n = (s % 4) * 4;
                const void* b = t == 0 ? a.BT : (t == 1 ? a.BL : a.C);
                base[k] = static_cast<const char*>(b) + (size_t)n * sizeof(io_t);
                pitch[k] = (int)(t == 0 ? a.pBT : (t == 1 ? a.pBL : a.pC));
                nvalid[k] = p < L::kPieces ? min(4, a.N - n) : 0;
            }
        }
    }
    // One cell.
    __device__ __forceinline__ void copy(unsigned cell, char* cellp, int pix) const {
#pragma unroll
        for (int k = 0; k < kCopies; ++k) {
            const char* src = base[k] + (long long)pix * pitch[k] * (int)sizeof(io_t);
            if (VEC) {
                if (sizeof(io_t) == 4) cp_async16_if(nvalid[k] > 0, cell + dst[k], src);
                else cp_async8_if(nvalid[k] > 0, cell + dst[k], src);
            } else {
                for (int e = 0; e < nvalid[k]; ++e) reinterpret_cast<io_t*>(cellp + dst[k])[e] = reinterpret_cast<const io_t*>(src)[e];
            }
        }
    }
    // kChunk consecutive cells of one row, `step` (+1 or -1) pixels apart (vector path).
    __device__ __forceinline__ void copy_run(unsigned cell, int pix, int step) const {
#pragma unroll
        for (int k = 0; k < kCopies; ++k) {
            const char* src = base[k] + (long long)pix * pitch[k] * (int)sizeof(io_t);
            const long long inc = (long long)(step * pitch[k] * (int)sizeof(io_t));
            if (nvalid[k] > 0) {
#pragma unroll
                for (int s = 0; s < kChunk; ++s) {
                    if (sizeof(io_t) == 4) cp_async16(cell + dst[k] + s * L::kStepBytes, src);
                    else cp_async8(cell + dst[k] + s * L::kStepBytes, src);
                    src += inc;
                }
            }
        }
    }
};

}  // namespace m2d
