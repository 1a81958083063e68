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
#include "scan_args.cuh"

namespace m2d {

constexpr int kWaveRows = 8;
constexpr int kWaveWarps = 8;
constexpr int kChunk = 4;      // steps per staged chunk; boundary columns move in the same units

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
// Three elements at the same place of three tensors.
__device__ __forceinline__ void store3_if(bool on, float* p, float* q, float* s, float a, float b, float c) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t@p st.global.f32 [%0], %3;\n\t@p st.global.f32 [%1], %4;\n\t@p st.global.f32 [%2], %5;\n\t}"
                 ::"l"(p), "l"(q), "l"(s), "f"(a), "f"(b), "f"(c), "r"((int)on) : "memory");
}
__device__ __forceinline__ void store3_if(bool on, __nv_bfloat16* p, __nv_bfloat16* q, __nv_bfloat16* s, float a, float b, float c) {
    const unsigned u = pack_bf16x2(a, b), v = pack_bf16x2(c, c);
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b16 a, b, c, d;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 {a, b}, %3;\n\tmov.b32 {c, d}, %4;\n\t"
                 "@p st.global.b16 [%0], a;\n\t@p st.global.b16 [%1], b;\n\t@p st.global.b16 [%2], c;\n\t}"
                 ::"l"(p), "l"(q), "l"(s), "r"(u), "r"(v), "r"((int)on) : "memory");
}
// A state block from shared memory, where `on`; elsewhere it stays as it is.
__device__ __forceinline__ void lds_block_if(bool on, unsigned addr, float2 (&o)[4][2]) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %17, 0;\n\t"
                 "@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%16];\n\t@p ld.shared.v4.f32 {%4, %5, %6, %7}, [%16+64];\n\t"
                 "@p ld.shared.v4.f32 {%8, %9, %10, %11}, [%16+128];\n\t@p ld.shared.v4.f32 {%12, %13, %14, %15}, [%16+192];\n\t}"
                 : "+f"(o[0][0].x), "+f"(o[0][0].y), "+f"(o[0][1].x), "+f"(o[0][1].y), "+f"(o[1][0].x), "+f"(o[1][0].y), "+f"(o[1][1].x),
                   "+f"(o[1][1].y), "+f"(o[2][0].x), "+f"(o[2][0].y), "+f"(o[2][1].x), "+f"(o[2][1].y), "+f"(o[3][0].x), "+f"(o[3][0].y),
                   "+f"(o[3][1].x), "+f"(o[3][1].y)
                 : "r"(addr), "r"((int)on) : "memory");
}
__device__ __forceinline__ void lds_block_if(bool on, unsigned addr, float2 (&o)[4][1]) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %9, 0;\n\t"
                 "@p ld.shared.v2.f32 {%0, %1}, [%8];\n\t@p ld.shared.v2.f32 {%2, %3}, [%8+32];\n\t"
                 "@p ld.shared.v2.f32 {%4, %5}, [%8+64];\n\t@p ld.shared.v2.f32 {%6, %7}, [%8+96];\n\t}"
                 : "+f"(o[0][0].x), "+f"(o[0][0].y), "+f"(o[1][0].x), "+f"(o[1][0].y), "+f"(o[2][0].x), "+f"(o[2][0].y), "+f"(o[3][0].x),
                   "+f"(o[3][0].y)
                 : "r"(addr), "r"((int)on) : "memory");
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
    bool both[kCopies];    // false: gy and C, which a recompute sweep does not need
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
                both[k] = t < 3;
                nvalid[k] = min(4, a.E - ch);
            } else {
                const int s = p - L::kTensors * per, t = s / 4, n = (s % 4) * 4;
                const void* b = t == 0 ? a.BT : (t == 1 ? a.BL : a.C);
                base[k] = static_cast<const char*>(b) + (size_t)n * sizeof(io_t);
                pitch[k] = (int)(t == 0 ? a.pBT : (t == 1 ? a.pBL : a.pC));
                nvalid[k] = p < L::kPieces ? min(4, a.N - n) : 0;
                both[k] = t < 2;
            }
        }
    }
    // One cell.  RECOMPUTE: without gy and C.
    template <bool RECOMPUTE>
    __device__ __forceinline__ void copy(unsigned cell, char* cellp, int pix) const {
#pragma unroll
        for (int k = 0; k < kCopies; ++k) {
            const char* src = base[k] + (long long)pix * pitch[k] * (int)sizeof(io_t);
            const bool on = nvalid[k] > 0 && (!RECOMPUTE || both[k]);
            if (VEC) {
                if (sizeof(io_t) == 4) cp_async16_if(on, cell + dst[k], src);
                else cp_async8_if(on, cell + dst[k], src);
            } else if (on) {
                for (int e = 0; e < nvalid[k]; ++e) reinterpret_cast<io_t*>(cellp + dst[k])[e] = reinterpret_cast<const io_t*>(src)[e];
            }
        }
    }
    // kChunk consecutive cells of one row, `step` (+1 or -1) pixels apart (vector path).
    template <bool RECOMPUTE>
    __device__ __forceinline__ void copy_run(unsigned cell, int pix, int step) const {
#pragma unroll
        for (int k = 0; k < kCopies; ++k) {
            const char* src = base[k] + (long long)pix * pitch[k] * (int)sizeof(io_t);
            const long long inc = (long long)(step * pitch[k] * (int)sizeof(io_t));
            if (nvalid[k] > 0 && (!RECOMPUTE || both[k])) {
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

// Shared memory of a CTA.
constexpr int kEdgeCols = 4 * kChunk;      // boundary columns per warp: three chunks to read, one to write
template <typename io_t, int C, bool BWD>
struct WaveSmem {
    typedef StageLayout<io_t, C, BWD> Stage;
    // chunk buffers: inputs are requested this many chunks, less one, ahead (a chunk of a CTA that has its SM
    // to itself takes about as long as a trip to HBM)
    static constexpr int kChunks = BWD ? 3 : 4;
    static constexpr int kEdgeBytes = kEdgeFloats<C> * 4;
    static constexpr int kSlots = kChunks * kChunk * Stage::kStepBytes;                   // hand-off slots of each warp
    static constexpr int kEdge = kSlots + kWaveWarps * kSlotBytes<C>;                     // boundary columns of each warp
    static constexpr int kAbove = kEdge + kWaveWarps * kEdgeCols * kEdgeBytes;            // backward: states above the band
    static constexpr int kZeros = kAbove + (BWD ? kWaveWarps * kChunks * kChunk * kEdgeBytes : 0);
    static constexpr int kPart = kZeros + kEdgeBytes;                                     // backward: each warp's share of dB, dC
    static constexpr int kPartBytes = kChunk * 3 * kWaveRows * 16 * 4;                    // ... per warp and chunk
    static constexpr int kBytes = kPart + (BWD ? kWaveWarps * kPartBytes : 0);
};

// What a lane keeps for the whole kernel.
template <typename io_t, int C, bool VEC, bool BWD>
struct WaveLane {
    int lane, r, nq, w, cgroups, cg, ch0, n0, chv, nv;
    unsigned lane_x, lane_b;                   // this lane's first channel / state in the first staged cell
    float2 aT[4][C / 2], aL[4][C / 2];         // A * log2(e) of its states, channels in pairs
    float2 Dm[C / 2];                          // D, in lane nq == 0 only: x*D enters the sum over states once
    Stager<io_t, C, BWD, VEC> stager;

    __device__ __forceinline__ void init(const ScanArgs& a, char* smem) {
        typedef WaveSmem<io_t, C, BWD> S;
        typedef typename S::Stage L;
        lane = threadIdx.x & 31; r = lane >> 2; nq = lane & 3; w = threadIdx.x >> 5;
        cgroups = (a.E + C - 1) / C;
        cg = blockIdx.y * kWaveWarps + w;
        ch0 = cg * C; n0 = nq * 4;
        chv = min(C, a.E - ch0); nv = min(4, max(0, a.N - n0));
        for (int k = threadIdx.x * 16; k < S::kBytes; k += blockDim.x * 16) *reinterpret_cast<float4*>(smem + k) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < C; ++c) {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const bool ok = c < chv && n < nv;
                const long long idx = (long long)(ch0 + c) * a.N + n0 + n;
                const float t = ok ? load_A<io_t>(a.AT, idx, a.a_log) * kLog2e : 0.f, u = ok ? load_A<io_t>(a.AL, idx, a.a_log) * kLog2e : 0.f;
                if (c & 1) { aT[n][c / 2].y = t; aL[n][c / 2].y = u; } else { aT[n][c / 2].x = t; aL[n][c / 2].x = u; }
            }
            const float d = nq == 0 && c < chv ? load_D<io_t>(a, ch0 + c) : 0.f;
            if (c & 1) Dm[c / 2].y = d; else Dm[c / 2].x = d;
        }
        lane_x = smem_u32(smem) + r * L::kCellBytes + w * C * (int)sizeof(io_t);
        lane_b = smem_u32(smem) + r * L::kCellBytes + (L::kTensors * L::kCh + n0) * (int)sizeof(io_t);
        stager.init(a, blockIdx.y * L::kCh, lane);
        __syncthreads();
    }
};

// A lane's block of states in the backward's record.  fp32 whatever the I/O type: the record of the few
// images this kernel is for is small, and the gradients are then those of the unrounded states.
template <int C> struct RecordBlock {
    static constexpr int kVecs = C;      // 16-byte pieces per lane
    float4 v[kVecs];
    __device__ __forceinline__ void pack(const float2 (&h)[4][C / 2]) {
#pragma unroll
        for (int m = 0; m < kVecs; ++m) {
            const float2 a = C == 4 ? h[m][0] : h[2 * m][0], b = C == 4 ? h[m][C / 2 - 1] : h[2 * m + 1][0];
            v[m] = make_float4(a.x, a.y, b.x, b.y);
        }
    }
    __device__ __forceinline__ void unpack(float2 (&h)[4][C / 2]) const {
#pragma unroll
        for (int m = 0; m < kVecs; ++m) {
            (C == 4 ? h[m][0] : h[2 * m][0]) = make_float2(v[m].x, v[m].y);
            (C == 4 ? h[m][C / 2 - 1] : h[2 * m + 1][0]) = make_float2(v[m].z, v[m].w);
        }
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int m = 0; m < kVecs; ++m) v[m] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ void store(float4* rec, int lane) const {
#pragma unroll
        for (int m = 0; m < kVecs; ++m) __stcg(rec + m * 32 + lane, v[m]);
    }
    __device__ __forceinline__ void load(const float4* rec, int lane) {
#pragma unroll
        for (int m = 0; m < kVecs; ++m) v[m] = __ldcg(rec + m * 32 + lane);
    }
};

}  // namespace m2d
