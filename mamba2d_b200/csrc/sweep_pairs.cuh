// Wavefront sweeps of the batch mode (one CTA per image and 16 channels), written as nested loops.
//
// A CTA owns 16 channels x 16 states and walks `nb` images; each image is cut into bands of `Rb` rows; warp r owns the
// rows 2r and 2r+1 of a band, "A" and "B", and walks them together: in one step it computes cell (A, col) and cell
// (B, col-1), which lie on one anti-diagonal and do not depend on each other.  Warp r runs two steps behind warp r-1.
// A lane owns 2 channels x 4 states of both rows, so
//   - A's state of the last step is B's state above: half of the hand-offs between rows never leave the registers;
//   - the parameters A_T, A_L of a lane and its sums of their gradients serve two cells: 16 values each instead of 32;
//   - sums over lanes take both cells through one exchange.
// The other hand-offs (B of warp r to A of warp r+1) go through shared memory; one __syncthreads per step keeps the warps
// in lock step.  The last row of a band reaches the first row of the next one through a per-CTA ring in global memory.  The
// recompute sweep of the backward also accumulates d_C = sum_e gy*h, while h is in registers;
// the adjoint sweep mirrors the forward one (bands last to first, the bottom row leads, columns right to left): B is a
// column ahead of A, and the block h[A][j] is B's state above and A's state on the left in the same step.
//
// Everything that arrives asynchronously from global memory (the staged inputs, ring blocks, blocks of the state record)
// is requested TWO steps before the cell that uses it and lands in one of three rotating buffers; a step ends with
// cp.async.wait_group 1, i.e. it waits for the copies issued one step earlier, never for its own.  (With one step of
// lead and two buffers the wait at the end of a step was for copies issued at its start, and a step is shorter than a
// trip to HBM on this part.)  The blocks handed from warp to warp rotate through the same three buffers, so that a step
// reads whatever it reads from buffer `rd`, requests into `wr` and hands over through `ho`, which is the next step's `rd`.
// A band boundary must be written at least two steps before the band below reads it: the plan keeps Rb <= W - 2.
//
// Against one row of 32 channels per warp, a lane 4 x 4 of it (us, kernel times, before / now): 128x56x56x64 fp32 forward
// 364 / 312, backward 1400 / 507 + 684 (its two sweeps are kernels of their own now); 128x28x28x128 bf16 190 / 171 and
// 656 / 183 + 402; 128x14x14x320 bf16 129 / 121 and 403 / 137 + 252; 128x7x7x512 fp32 64 / 52 and 199 / 63 + 116.  Instructions
// per 512 states (56x56x64 fp32): forward 224 -> 189, both sweeps of the backward 803 -> 217 + 521; wavefronts of the
// shared-memory pipe, which was half busy, 250 -> 56 + 152.  What bounds them now: the forward and the adjoint the latency of
// a warp's instructions at 16 warps per SM (128 registers; an instruction every 2.0 and 1.7 cycles of a scheduler), and
// that 512 CTAs put four on some SMs and three on others; the recompute sweep in fp32 the writing of the record (2.5 GB
// through DRAM in 507 us; with a bf16 record, 369).  Blocks of one anti-diagonal side by side in the record, blocks copied out
// of shared memory in bulk (505 / 509, 231 / 245 at 28x28x128), and inputs
// requested into L2 four columns ahead, did not change the last.
#pragma once

#include "scan_args.cuh"

namespace m2d {

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_prev() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }


// ---- what a lane is ----------------------------------------------------------------------------------------------
// lane = (cq, nq) = (lane >> 2, lane & 3): channels ch0 = 16 g + 2 cq, +1 and states 4 nq ... 4 nq + 3 of rows A and B.
// In copies and in sums over channels the upper half of the warp stands for row B (or d_BL); in sums over states, the
// lanes with nq & 2 do.
struct PairLane {
    int lane, r, nwarps, cq, nq, g, ch0, n0, chv, nv;
    __device__ __forceinline__ PairLane(const ScanArgs& a) {
        lane = threadIdx.x & 31; r = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0); nwarps = blockDim.x >> 5;
        cq = lane >> 2; nq = lane & 3; g = blockIdx.x;
        ch0 = g * kGroup + cq * 2; n0 = nq * 4;
        chv = min(2, max(0, a.E - ch0)); nv = min(4, max(0, a.N - n0));
    }
};

// ---- shared memory -----------------------------------------------------------------------------------------------
// A block per warp, and in it areas of three 1 KiB buffers (kRot apart):
//   S   states (forward) or pT (adjoint) of the row before this warp's, resp. of its own row A
//   T   staged inputs: cells A and B, kCellSlots slots of 16 bytes each
//   HA  adjoint: h[A][j]          HB  adjoint: h[B][j-1]
// The first warp's block follows an HB area (adjoint), the last one's is followed by an S area, then by the parameters.
__device__ __forceinline__ float4 lds4(unsigned p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p) : "memory");
    return v;
}
__device__ __forceinline__ void sts4(unsigned p, const float4& v) {
    asm volatile("st.shared.v4.f32 [%4], {%0, %1, %2, %3};" ::"f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(p) : "memory");
}
__device__ __forceinline__ float2 bf2_pair(unsigned u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
// two or four staged elements as floats
template <typename io_t> __device__ __forceinline__ float2 lds_in2(unsigned p);
template <> __device__ __forceinline__ float2 lds_in2<float>(unsigned p) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(p) : "memory");
    return v;
}
template <> __device__ __forceinline__ float2 lds_in2<__nv_bfloat16>(unsigned p) {
    unsigned u;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(u) : "r"(p) : "memory");
    return bf2_pair(u);
}
template <typename io_t> __device__ __forceinline__ float lds_in1(unsigned p) {
    if constexpr (sizeof(io_t) == 4) {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p) : "memory");
        return v;
    } else {
        unsigned short v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p) : "memory");
        return bf16_bits_to_float(v);
    }
}
typedef float2 Quad[2];         // four states of one channel
template <typename io_t> __device__ __forceinline__ void lds_in4(Quad& o, unsigned p);
template <> __device__ __forceinline__ void lds_in4<float>(Quad& o, unsigned p) {
    const float4 v = lds4(p);
    o[0] = make_float2(v.x, v.y);
    o[1] = make_float2(v.z, v.w);
}
template <> __device__ __forceinline__ void lds_in4<__nv_bfloat16>(Quad& o, unsigned p) {
    unsigned u, v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(u), "=r"(v) : "r"(p) : "memory");
    o[0] = bf2_pair(u);
    o[1] = bf2_pair(v);
}
__device__ __forceinline__ float4 quad_f4(const Quad& q) { return make_float4(q[0].x, q[0].y, q[1].x, q[1].y); }
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 ex2_pair(float2 v) { return make_float2(ex2(v.x), ex2(v.y)); }
__device__ __forceinline__ float2 keep(bool on, float2 v) { return on ? v : make_float2(0.f, 0.f); }
__device__ __forceinline__ void clear(Quad (&s)[2]) { s[0][0] = s[0][1] = s[1][0] = s[1][1] = make_float2(0.f, 0.f); }

// Exchange between lanes that differ in bit `mask` of their number: this lane's pair plus the other one's `v`.
__device__ __forceinline__ float2 add_other(float2 own, float2 v, int mask) {
    return __fadd2_rn(own, make_float2(__shfl_xor_sync(0xffffffffu, v.x, mask), __shfl_xor_sync(0xffffffffu, v.y, mask)));
}
__device__ __forceinline__ float2 choose(bool c, float2 v, float2 w) { return make_float2(c ? v.x : w.x, c ? v.y : w.y); }
// Sums over the 8 cq lanes of a warp.  Lanes of its upper half have what they keep in `own`, as the lower ones have, and
// what the lower ones keep in `other`.  This lane is left with state 2*hi2 + hi1 of the four.
__device__ __forceinline__ float reduce_channels(const Quad& own, const Quad& other, bool hi2, bool hi1) {
    const float2 a = add_other(own[0], other[0], 16), b = add_other(own[1], other[1], 16);
    const float2 k = add_other(choose(hi2, b, a), choose(hi2, a, b), 8);
    return (hi1 ? k.y : k.x) + __shfl_xor_sync(0xffffffffu, hi1 ? k.x : k.y, 4);
}
// Sums over the 4 nq lanes of two channels of rows A and B.  This lane is left with channel nq & 1 of row (nq & 2 ? B : A).
__device__ __forceinline__ float reduce_rows(float2 vA, float2 vB, int nq) {
    const bool hi = (nq & 2) != 0, lo = (nq & 1) != 0;
    const float2 k = add_other(choose(hi, vB, vA), choose(hi, vA, vB), 2);
    return (lo ? k.y : k.x) + __shfl_xor_sync(0xffffffffu, lo ? k.x : k.y, 1);
}

// A lane's part of a block of states in the record: 16 bytes per channel (fp32), or 16 bytes in all (bf16).
template <typename rec_t> __device__ __forceinline__ void write_record(float4* p, const Quad (&s)[2]) {
    __stcs(p, quad_f4(s[0]));
    __stcs(p + 32, quad_f4(s[1]));
}
template <> __device__ __forceinline__ void write_record<__nv_bfloat16>(float4* p, const Quad (&s)[2]) {
    __stcs(p, make_float4(__uint_as_float(pack_bf16x2(s[0][0].x, s[0][0].y)), __uint_as_float(pack_bf16x2(s[0][1].x, s[0][1].y)),
                          __uint_as_float(pack_bf16x2(s[1][0].x, s[1][0].y)), __uint_as_float(pack_bf16x2(s[1][1].x, s[1][1].y))));
}
template <typename rec_t> __device__ __forceinline__ void lds_record(Quad& o, unsigned p, int c) {
    lds_in4<rec_t>(o, sizeof(rec_t) == 2 ? p + c * 8 : p + c * 512);
}
template <typename rec_t> __device__ __forceinline__ void request_record(unsigned smem, const float4* gmem) {
    if (sizeof(rec_t) == 2) cp_async16(smem, gmem);
    else cp_async_block(smem, gmem);
}

// Staging of a step's two cells, every distinct 16-byte piece (four elements) by exactly one lane: two copies per lane,
// the lower half of the warp for row A, the upper one for row B.  Pieces beyond E or N are never copied: they stay zero.
template <typename io_t, bool VEC>
struct PairCopy {
    const char *cbase, *bbase;
    int bpitch;              // bytes per pixel
    int cv, bv;              // valid elements of this lane's two pieces
    __device__ __forceinline__ void init(const ScanArgs& a, int g, int lane, bool with_gy) {
        const int k = lane & 15, t = k >> 2, piece = k & 3;
        const void* cp = t == 0 ? a.x : (t == 1 ? a.dT : (t == 2 ? a.dL : a.gy));
        const int ch = g * kGroup + piece * 4, n = piece * 4;
        cv = (t < 3 || with_gy) ? min(4, max(0, a.E - ch)) : 0;
        cbase = static_cast<const char*>(cp) + (size_t)ch * sizeof(io_t);
        const void* bp = t == 0 ? a.BT : (t == 1 ? a.BL : a.C);
        bpitch = (int)(t == 0 ? a.pBT : (t == 1 ? a.pBL : a.pC)) * (int)sizeof(io_t);
        bv = t < 3 ? min(4, max(0, a.N - n)) : 0;
        bbase = static_cast<const char*>(bp) + (size_t)n * sizeof(io_t);
    }
    // where this lane's first piece goes, from the start of a T buffer; the second one is 16 slots behind
    static __device__ __forceinline__ unsigned slot(int lane) { return ((lane >> 4) * kCellSlots + (lane & 15)) * 16; }
    __device__ __forceinline__ void issue(unsigned dst, bool on, int pix, int E) const {
        const char *sc = cbase + (long long)pix * (E * (int)sizeof(io_t)), *sb = bbase + (long long)pix * bpitch;
        if (VEC) {
            if (sizeof(io_t) == 4) {
                if (on && cv > 0) cp_async16(dst, sc);
                if (on && bv > 0) cp_async16(dst + 256, sb);
            } else {
                if (on && cv > 0) cp_async8(dst, sc);
                if (on && bv > 0) cp_async8(dst + 256, sb);
            }
        } else if (on) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k < cv) st_element(dst + k * (int)sizeof(io_t), reinterpret_cast<const io_t*>(sc) + k);
                if (k < bv) st_element(dst + 256 + k * (int)sizeof(io_t), reinterpret_cast<const io_t*>(sb) + k);
            }
        }
    }
    static __device__ __forceinline__ void st_element(unsigned p, const io_t* v) {
        if constexpr (sizeof(io_t) == 4) asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(__ldg(reinterpret_cast<const float*>(v))) : "memory");
        else asm volatile("st.shared.u16 [%0], %1;" ::"r"(p), "h"(__ldg(reinterpret_cast<const unsigned short*>(v))) : "memory");
    }
};

// One staged cell as a lane sees it.
struct CellIn { float2 x, dT, dL, gy; Quad bT, bL, c; };
// px, pn: this lane's first channel and first state of the cell (cell_x, cell_n: from the start of a T buffer, row A).
template <typename io_t> __device__ __forceinline__ unsigned cell_x(int cq) { return (cq >> 1) * 16 + (cq & 1) * 2 * (int)sizeof(io_t); }
__device__ __forceinline__ unsigned cell_n(int nq) { return (16 + nq) * 16; }
// x of the channel and row whose sums over states this lane is left with (reduce_rows)
template <typename io_t> __device__ __forceinline__ unsigned cell_out(int cq, int nq) {
    return cell_x<io_t>(cq) + (nq & 1) * (int)sizeof(io_t) + (nq >> 1) * kCellSlots * 16;
}
template <typename io_t, bool GY, bool READ_C>
__device__ __forceinline__ void read_cell(CellIn& v, unsigned px, unsigned pn) {
    v.x = lds_in2<io_t>(px);
    v.dT = lds_in2<io_t>(px + 64);
    v.dL = lds_in2<io_t>(px + 128);
    if (GY) v.gy = lds_in2<io_t>(px + 192);
    lds_in4<io_t>(v.bT, pn);
    lds_in4<io_t>(v.bL, pn + 64);
    if (READ_C) lds_in4<io_t>(v.c, pn + 128);
}
// ---- bands in several CTAs (CHAIN) ---------------------------------------------------------------------------------
// Where there are few images the bands of one go to `chain` CTAs, CTA c taking the bands c, c + chain, ...; a boundary row in
// global memory then takes the place of the ring.  As in the wave kernels it is zeroed before the launch and holds states
// with their bits inverted, so that a block that is not there yet shows: no arithmetic returns the NaN that would read as
// zero.  A block is requested two steps ahead like everything else; where it was not there, the warp that needs it polls,
// and the CTA falls behind the one above until its requests find what they ask for.
__device__ __forceinline__ uint4 invert_bits(const float4& v) {
    return make_uint4(~__float_as_uint(v.x), ~__float_as_uint(v.y), ~__float_as_uint(v.z), ~__float_as_uint(v.w));
}
__device__ __forceinline__ bool arrived(const float4& v) {
    return __float_as_uint(v.x) != 0 && __float_as_uint(v.y) != 0 && __float_as_uint(v.z) != 0 && __float_as_uint(v.w) != 0;
}
// Makes sure that the block in S buffer `smem` is the one at `src`.  Every poll is bounded; a warp that has given up once
// waits no more (what it reads then are NaNs).  (Waiting for a block two, four or six columns on as well, so that later
// requests come back in time, costs half a microsecond per band and column and gains nothing: 716, 744 and 786 us against
// 697 in the adjoint sweep at 2x200x336x64.)
__device__ __forceinline__ void wait_for_block(const ScanArgs& a, unsigned smem, const float4* src, bool& given_up) {
    if (__all_sync(0xffffffffu, arrived(lds4(smem)) && arrived(lds4(smem + 512)))) return;
#pragma unroll 1
    for (int polls = 0;; ++polls) {
        float4 v[2];
#pragma unroll
        for (int c = 0; c < 2; ++c)
            asm volatile("ld.volatile.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[c].x), "=f"(v[c].y), "=f"(v[c].z), "=f"(v[c].w) : "l"(src + c * 32) : "memory");
        if (polls > a.wait_limit || *reinterpret_cast<volatile int*>(a.status) != 0) {
            if (!given_up) {
                atomicExch(a.status, 1);
                if (a.host_flag) *reinterpret_cast<volatile int*>(a.host_flag) = 1;
            }
            given_up = true;
        }
        given_up = __any_sync(0xffffffffu, given_up);
        if (__all_sync(0xffffffffu, arrived(v[0]) && arrived(v[1])) || given_up) {
            sts4(smem, v[0]);
            sts4(smem + 512, v[1]);
            return;
        }
    }
}
__device__ __forceinline__ float2 flip_bits(float2 v, unsigned mask) {
    return make_float2(__uint_as_float(__float_as_uint(v.x) ^ mask), __uint_as_float(__float_as_uint(v.y) ^ mask));
}
template <bool CHAIN> __device__ __forceinline__ void push_block(float4* dst, const Quad& s0, const Quad& s1) {
    if (CHAIN) {
        __stcg(reinterpret_cast<uint4*>(dst), invert_bits(quad_f4(s0)));
        __stcg(reinterpret_cast<uint4*>(dst + 32), invert_bits(quad_f4(s1)));
    } else {
        __stcg(dst, quad_f4(s0));
        __stcg(dst + 32, quad_f4(s1));
    }
}

// What a CTA walks: the images blockIdx.y, blockIdx.y + gridDim.y, ... of channel group blockIdx.x with all their bands, or
// (CHAIN) every chain-th band of one image.  (The groups of an image have neighbouring blocks, run at the same time and find
// each other's lines of B, C and their gradients in L2.)
template <bool CHAIN>
struct PairWork {
    int img0, img_stride, nb, q0, dq, items;
    __device__ __forceinline__ PairWork(const ScanArgs& a) {
        if (CHAIN) {
            img0 = blockIdx.y / a.chain; img_stride = 0; nb = 1;
            q0 = blockIdx.y % a.chain; dq = a.chain;
            items = (a.nbands - q0 + dq - 1) / dq;
        } else {
            img0 = blockIdx.y; img_stride = gridDim.y; nb = (a.B - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;
            q0 = 0; dq = 1;
            items = nb * a.nbands;
        }
    }
};

// The rotation of the three buffers, as byte offsets.
struct Rotation {
    unsigned rd = kRot, wr = 0, ho = 2 * kRot;
    __device__ __forceinline__ void end_step() {
        cp_async_commit();
        cp_async_wait_prev();
        __syncthreads();
        const unsigned t = ho;
        ho = wr;
        wr = rd;
        rd = t;
    }
};

// Start of a kernel: shared memory zeroed, and behind its `bytes` the parameters, whose address is returned.
template <typename io_t>
__device__ __forceinline__ unsigned begin_pairs(const ScanArgs& a, float4* smem, size_t bytes, const PairLane& ln) {
    for (int k = threadIdx.x; k < (int)(bytes / sizeof(float4)); k += blockDim.x) smem[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    float4* const params = smem + bytes / sizeof(float4);
    if (threadIdx.x < 32) stage_params<io_t>(params, a.AT, a.AL, a.N, ln.ch0, ln.chv, ln.n0, ln.nv, ln.lane, a.a_log);
    __syncthreads();
    return smem_u32(params + ln.lane);
}

// How a step is compiled.  kInside: both cells exist and lie inside the map, where the weights are constants.  kTop: the
// same with A in row 0, which has no direction T.  kBorder: both exist, one of them in column 0; weights and zeros for
// missing neighbours are chosen without a branch, so that the two cells overlap as they do inside.  kPartial: one cell is
// missing, at the ends of the sweep and under an odd last row.
enum StepKind { kInside, kTop, kBorder, kPartial };
template <int K> struct StepTag { static constexpr int value = K; };

// RECORD (the backward's recompute sweep): every fresh state block goes to the state record a.hs, of type rec_t, and d_C is
// accumulated, and nothing is written to y.  D_lane: D of the channel whose y this lane stores.
//
// ACT: gelu(y) goes out instead of y.  It is worked out and stored in the warp's next step: behind the sum over states, at
// the end of its own, its chain of fifteen dependent instructions lies open in every step.
template <typename io_t, typename rec_t, bool VEC, bool RECORD, bool ACT, bool CHAIN>
__device__ __forceinline__ void forward_pairs(const ScanArgs& a, unsigned smem, unsigned params, float D_lane) {
    constexpr int HB = HsBlock<rec_t>::f4;
    const PairLane ln(a);
    const int lane = ln.lane, r = ln.r, cq = ln.cq, nq = ln.nq, g = ln.g;
    const int W = a.W, H = a.H, E = a.E, Rb = a.Rb, nbands = a.nbands;
    const PairWork<CHAIN> work(a);
    // the ring, or the boundary rows of this image and group
    float4* const ring = CHAIN ? a.bnd + ((size_t)(work.img0 * gridDim.x + g) * nbands * W) * kSlotF4 + lane
                               : a.ring + ((size_t)(blockIdx.y * gridDim.x + blockIdx.x) * W) * kSlotF4 + lane;
    const unsigned blk = smem + r * kFwdBlock + lane * 16;                // S of the row above; + kFwdBlock: of the row below
    const unsigned stage = smem + r * kFwdBlock + 3 * kRot;
    const unsigned stage_x = stage + cell_x<io_t>(cq), stage_n = stage + cell_n(nq), stage_o = stage + cell_out<io_t>(cq, nq), stage_w = stage + PairCopy<io_t, VEC>::slot(lane);
    const float ninf = __int_as_float(0xff800000);
    const int dir = a.dir;
    const bool upper = lane >= 16;
    const bool y_rowB = (nq & 2) != 0;
    const int y_ch = ln.ch0 + (nq & 1);
    const bool y_ok = y_ch < E;
    const int dc_n = ln.n0 + ((cq & 2) ? 2 : 0) + ((cq & 1) ? 1 : 0);
    const bool dc_ok = dc_n < a.N;
    float4* const hs_img = RECORD ? a.hs + (size_t)g * a.B * H * W * HB + lane : nullptr;   // + memory pixel * HB

    PairCopy<io_t, VEC> copy;
    copy.init(a, g, lane, RECORD);
    Quad aT[2], aL[2], hA[2], hB[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        lds_in4<float>(aT[c], params + c * 512);
        lds_in4<float>(aL[c], params + 1024 + c * 512);
    }
    clear(hA);
    clear(hB);
    Rotation rot;

    struct Rows { bool hasA, hasB, row0, pull, pushA, pushB; int pix, edge; };   // pix: memory pixel of column 0 of row A; edge: CHAIN, block 0 of this band's boundary row
    auto make_rows = [&](int bi, int q) {
        Rows w;
        const int i = q * Rb + 2 * r;
        w.hasA = bi < work.nb && 2 * r < Rb && i < H;
        w.hasB = w.hasA && 2 * r + 1 < Rb && i + 1 < H;
        w.row0 = (i == 0);
        w.pull = w.hasA && (r == 0) && (q > 0);
        const bool push = q < nbands - 1 && !(CHAIN && a.withhold && work.img0 == 0 && q == 0);
        w.pushA = w.hasA && (2 * r == Rb - 1) && push;
        w.pushB = w.hasB && (2 * r + 1 == Rb - 1) && push;
        w.pix = scan_pixel(a, work.img0 + bi * work.img_stride, i, 0);
        w.edge = CHAIN ? q * W : 0;
        return w;
    };
    // What is requested next: cell (A, s_col) by the lower half of the warp, cell (B, s_col - 1) by the upper one, each at its s_pix.
    bool s_on = false, s_pull = false;
    int s_pix = 0, s_col = 0, s_edge = 0;         // s_edge: the row above's boundary blocks
    auto request = [&](bool on) {
        copy.issue(stage_w + rot.wr, on, s_pix, E);
        if (s_pull) cp_async_block(blk + rot.wr, ring + (s_edge + s_col) * kSlotF4);
        s_pix += dir;
        ++s_col;
    };
    auto next_A = [&](const Rows& w) {
        if (!upper) { s_on = w.hasA; s_pix = w.pix; }
        s_pull = w.pull;
        s_col = 0;
        s_edge = CHAIN ? w.edge - W : 0;
    };
    auto next_B = [&](const Rows& w) {
        if (upper) { s_on = w.hasB; s_pix = w.pix + dir * W; }
    };

    float y_held = 0.f;                          // ACT: y of the warp's last cells and where its activation goes
    int y_to = -1;
    auto store_held = [&]() {
        if (ACT && y_to >= 0) store1(static_cast<io_t*>(a.y), y_to, gelu_erf(y_held));
        y_to = -1;
    };

    // one step: cell (A, colA) and cell (B, colB)
    bool hasA = false, hasB = false, row0 = false, pushA = false, pushB = false, given_up = false;
    int pixA = 0, pixB = 0, edgeA = 0, edgeB = 0;
    auto step = [&](auto tag, const int colA, const int colB) {
        constexpr int KIND = decltype(tag)::value;
        constexpr bool FAST = KIND <= kTop, ALL = KIND != kPartial;
        if (ACT) store_held();
        const bool pulled = CHAIN && r == 0 && KIND != kTop && hasA && !row0;
        if (CHAIN && pulled) wait_for_block(a, blk + rot.rd, ring + (edgeA - W + colA) * kSlotF4, given_up);
        const unsigned flip = pulled ? 0xffffffffu : 0u;
        Quad dC[2];
        float2 yv[2];
        // B first: what is above it is A's state of the last step, still in place (A first, with a copy of it, 320 us against 312 at
        // 128x56x56x64 fp32, 55 against 52 at 7x7x512; both cells read before either is computed, 315 and 54)
#pragma unroll
        for (int w = 1; w >= 0; --w) {
            Quad (&h)[2] = w ? hB : hA;
            const bool NO_T = KIND == kTop && w == 0;         // (a constant: the loop is unrolled)
            yv[w] = dC[w][0] = dC[w][1] = make_float2(0.f, 0.f);
            if (!ALL && !(w ? hasB : hasA)) continue;
            CellIn v;
            read_cell<io_t, RECORD, !RECORD>(v, stage_x + rot.rd + w * kCellSlots * 16, stage_n + rot.rd + w * kCellSlots * 16);
            float wT = 0.5f, wL = 0.5f, oT = -1.f, oL = -1.f;
            bool first = false, top_row = false;
            if (!FAST) {
                // (a missing neighbour's state is taken as zero)
                first = (w ? colB : colA) == 0;
                top_row = w == 0 && row0;
                wT = top_row ? 0.f : (first ? 1.f : 0.5f);
                wL = first ? (top_row ? 1.f : 0.f) : (top_row ? 1.f : 0.5f);
                oT = top_row ? ninf : (first ? 0.f : -1.f);
                oL = first ? ninf : (top_row ? 0.f : -1.f);
            }
            const float2 xT = __fmul2_rn(v.x, both(wT)), xL = NO_T ? v.x : FAST ? xT : __fmul2_rn(v.x, both(wL));
            const float2 vT = __fmul2_rn(v.dT, xT), vL = __fmul2_rn(v.dL, xL);
            const float dTs[2] = {v.dT.x, v.dT.y}, dLs[2] = {v.dL.x, v.dL.y}, gys[2] = {v.gy.x, v.gy.y};
            const float dtx[2] = {vT.x, vT.y}, dlx[2] = {vL.x, vL.y};
            float ysum[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                Quad top;
                if (w) { top[0] = hA[c][0]; top[1] = hA[c][1]; }
                else if (!NO_T) {
                    lds_in4<float>(top, blk + rot.rd + c * 512);
                    if (CHAIN) { top[0] = flip_bits(top[0], flip); top[1] = flip_bits(top[1], flip); }
                    if (!FAST) { top[0] = keep(!row0, top[0]); top[1] = keep(!row0, top[1]); }
                }
                float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float2 l = FAST ? h[c][k] : keep(!first, h[c][k]);
                    const float2 gL = ex2_pair(NO_T ? __fmul2_rn(both(dLs[c]), aL[c][k]) : __ffma2_rn(both(dLs[c]), aL[c][k], both(oL)));
                    float2 in = __fmul2_rn(both(dlx[c]), v.bL[k]);
                    if (!NO_T) {
                        const float2 gT = ex2_pair(__ffma2_rn(both(dTs[c]), aT[c][k], both(oT)));
                        in = __ffma2_rn(gT, top[k], __ffma2_rn(both(dtx[c]), v.bT[k], in));
                    }
                    h[c][k] = __ffma2_rn(gL, l, in);
                    if (RECORD) dC[w][k] = __ffma2_rn(both(gys[c]), h[c][k], dC[w][k]);
                    else acc = __ffma2_rn(h[c][k], v.c[k], acc);
                }
                ysum[c] = acc.x + acc.y;
            }
            yv[w] = make_float2(ysum[0], ysum[1]);
        }
        sts4(blk + kFwdBlock + rot.ho, quad_f4(hB[0]));
        sts4(blk + kFwdBlock + rot.ho + 512, quad_f4(hB[1]));
        if (pushB) push_block<CHAIN>(ring + (edgeB + colB) * kSlotF4, hB[0], hB[1]);
        if (!ALL && pushA) push_block<CHAIN>(ring + (edgeA + colA) * kSlotF4, hA[0], hA[1]);
        if (RECORD) {
            if (ALL || hasA) write_record<rec_t>(hs_img + (ptrdiff_t)pixA * HB, hA);
            if (ALL || hasB) write_record<rec_t>(hs_img + (ptrdiff_t)pixB * HB, hB);
            // d_C[pixel][n] = sum over channels of gy*h: 8 values (two rows, four states) over the 8 cq lanes
            const Quad own = {choose(upper, dC[1][0], dC[0][0]), choose(upper, dC[1][1], dC[0][1])};
            const Quad other = {choose(upper, dC[0][0], dC[1][0]), choose(upper, dC[0][1], dC[1][1])};
            const float v = reduce_channels(own, other, (cq & 2) != 0, (cq & 1) != 0);
            const int pix = upper ? pixB : pixA;
            if (dc_ok && (ALL || (upper ? hasB : hasA))) atomicAdd(a.accC + ((long long)pix * a.acc_pitch + dc_n), v);
        } else {
            const float y = fmaf(lds_in1<io_t>(stage_o + rot.rd), D_lane, reduce_rows(yv[0], yv[1], nq));
            const int pix = y_rowB ? pixB : pixA;
            if (y_ok && (ALL || (y_rowB ? hasB : hasA))) {
                const int to = pix * E + y_ch;
                if (ACT) { y_held = y; y_to = to; }
                else store1(static_cast<io_t*>(a.y), to, y);
            }
        }
    };

    // ---- the warp's sequence ---------------------------------------------------------------------
    // 2r idle steps, two steps that only request, W steps per (image, band) item, one for the last cell of row B, and
    // idle steps until the last warp is done
    for (int k = 0; k < 2 * r; ++k) rot.end_step();
    int bi = 0, q = work.q0;
    Rows cur = make_rows(bi, q);
    next_A(cur);
    request(s_on);
    rot.end_step();
    next_B(cur);
    request(s_on);
    rot.end_step();
    const int items = work.items;
    for (int m = 0; m <= items; ++m) {
        hasA = cur.hasA;
        row0 = cur.row0;
        pushA = cur.pushA;
        pixA = cur.pix;
        if (CHAIN) edgeA = cur.edge;
        if ((q += work.dq) >= nbands) { q = work.q0; ++bi; }
        Rows nxt = cur;
        const bool fast = cur.hasA && cur.hasB;
        const int cols = m < items ? W : 1;
        int col = 0;
        // requests at the end of a row are for the next one (nothing exists past the last item)
        auto request_ahead = [&]() {
            if (col + 2 == W) {
                nxt = make_rows(bi, q);
                next_A(nxt);
            } else if (col + 2 == W + 1) {
                next_B(nxt);
            }
            request(s_on);
        };
        for (; col < (fast ? 2 : cols); ++col) {
            request_ahead();
            if (col == 1) {
                hasB = cur.hasB;
                pushB = cur.pushB;
                if (CHAIN) edgeB = cur.edge;
                pixB = cur.pix + dir * W;
            }
            if (hasA && hasB) step(StepTag<kBorder>{}, col, col == 0 ? W - 1 : col - 1);
            else if (hasA || hasB) step(StepTag<kPartial>{}, col, col == 0 ? W - 1 : col - 1);
            pixA += dir;
            pixB += dir;
            rot.end_step();
        }
        for (; col < cols; ++col) {
            if (col + 2 < W) request(true);
            else request_ahead();
            if (row0) step(StepTag<kTop>{}, col, col - 1);
            else step(StepTag<kInside>{}, col, col - 1);
            pixA += dir;
            pixB += dir;
            rot.end_step();
        }
        cur = nxt;
    }
    if (ACT) store_held();
    for (int k = 0; k < 2 * (ln.nwarps - 1 - r); ++k) rot.end_step();
    cp_async_wait_all();                                      // (only empty groups can be pending here)
}

// Adjoint sweep of one CTA over its images.  Bands are visited last to first, the bottom row of a band leads, columns run
// right to left: in step j a warp computes cell (B, j) and cell (A, j+1); at j = W-1 that is column 0 of A in the band
// before.  Warp r runs two steps behind warp r+1.
template <typename io_t, typename rec_t, bool VEC, bool CHAIN>
__device__ __forceinline__ void reverse_pairs(const ScanArgs& a, unsigned smem, unsigned params, float D_lane,
                                              Quad (&dAT)[2], Quad (&dAL)[2], float& dD) {
    constexpr int HB = HsBlock<rec_t>::f4;     // float4 units per state-record block
    const PairLane ln(a);
    const int lane = ln.lane, r = ln.r, cq = ln.cq, nq = ln.nq, g = ln.g, nwarps = ln.nwarps;
    const int W = a.W, H = a.H, E = a.E, Rb = a.Rb, nbands = a.nbands;
    const int rr = nwarps - 1 - r;             // rank in the reverse sweep
    const int dir = a.dir;
    const PairWork<CHAIN> work(a);
    float4* const ring = CHAIN ? a.bnd_up + ((size_t)(work.img0 * gridDim.x + g) * nbands * W) * kSlotF4 + lane
                               : a.ring + ((size_t)(blockIdx.y * gridDim.x + blockIdx.x) * W) * kSlotF4 + lane;
    const unsigned blk = smem + 3 * kRot + r * kBwdBlock + lane * 16;     // S: pT of row A; + kBwdBlock: of the row below B
    const unsigned stage = smem + 6 * kRot + r * kBwdBlock;
    const unsigned stage_x = stage + cell_x<io_t>(cq), stage_n = stage + cell_n(nq), stage_o = stage + cell_out<io_t>(cq, nq), stage_w = stage + PairCopy<io_t, VEC>::slot(lane);
    constexpr int kHA = 6 * kRot, kHB = 9 * kRot, kUp = 9 * kRot - kBwdBlock;     // from blk: h[A][j], h[B][j-1], and h[A-1][j+1] of the warp above
    const float4* const hs_img = a.hs + (size_t)g * a.B * H * W * HB + lane;     // + memory pixel * HB
    const bool upper = lane >= 16;
    const bool o_rowB = (nq & 2) != 0;
    const int o_ch = ln.ch0 + (nq & 1);
    const bool o_ok = o_ch < E;
    const bool feeds_below = r + 1 < nwarps;
    const bool hi2 = (cq & 2) != 0, hi1 = (cq & 1) != 0;
    const int db_n = ln.n0 + (hi2 ? 2 : 0) + (hi1 ? 1 : 0);
    float* const db_acc = (upper ? a.accBL : a.accBT) + db_n;
    const bool db_ok = db_n < a.N;
    const float ninf = __int_as_float(0xff800000);

    PairCopy<io_t, VEC> copy;
    copy.init(a, g, lane, true);
    Quad pLA[2], pLB[2], carry[2];             // pL of the two rows; pT of B's last cell, for A's next one
    clear(pLA);
    clear(pLB);
    clear(carry);
    Rotation rot;

    struct Rows { bool hasA, hasB, row0, pullA, pullB, push, top, bottom; int pix, edge; };   // pix: memory pixel of column W-1 of row A; edge: CHAIN, block 0 of the boundary row below
    auto make_rows = [&](int bi, int q) {
        Rows w;
        const int i = q * Rb + 2 * r;
        w.hasA = bi < work.nb && 2 * r < Rb && i < H;
        w.hasB = w.hasA && 2 * r + 1 < Rb && i + 1 < H;
        w.row0 = (i == 0);
        w.pullA = w.hasA && (2 * r == Rb - 1) && i + 1 < H;       // pT of the row below comes through the ring
        w.pullB = w.hasB && (2 * r + 1 == Rb - 1) && i + 2 < H;
        w.push = w.hasA && (r == 0) && (q > 0) && !(CHAIN && q == a.mute_up);       // pT of row A goes to the band above through the ring
        w.top = w.hasA && (r == 0) && (i > 0);        // h of the row above is not requested by a warp of this band
        w.bottom = i + 2 >= H;                        // nothing below row B
        w.pix = scan_pixel(a, work.img0 + bi * work.img_stride, i, W - 1);
        w.edge = CHAIN ? q * W : 0;
        return w;
    };
    const int down = dir * W;                         // from a pixel to the one below it
    // request h[B][W-1] for the warp below (nobody's left neighbour, so no cell's request covers it)
    auto request_row_end = [&](const Rows& w) {
        if (feeds_below && w.hasB) request_record<rec_t>(blk + kHB + rot.wr, hs_img + (ptrdiff_t)(w.pix + down) * HB);
    };
    // What is requested next: cell (B, s_j), below pixel s_pixL of row A, by the upper half of the warp, cell (A, s_j + 1), at
    // s_pixA, by the lower one, each at its s_pix.
    bool s_on = false, s_hasA, s_hasB, s_pullB, t_pullA = false, t_top = false;
    int s_pix = 0, s_pixL, s_pixA = 0, s_j = W - 1, s_edge = 0, t_edge = 0;
    auto request = [&](auto tag) {
        constexpr bool FAST = decltype(tag)::value;       // both rows exist, and s_j > 0
        copy.issue(stage_w + rot.wr, FAST || s_on, s_pix, E);
        const float4* const ph = hs_img + (ptrdiff_t)s_pixL * HB;
        if (FAST || s_hasA) request_record<rec_t>(blk + kHA + rot.wr, ph);
        if (FAST || (s_hasB && s_j > 0)) request_record<rec_t>(blk + kHB + rot.wr, ph + (ptrdiff_t)(down - dir) * HB);
        if (t_top) request_record<rec_t>(blk + kUp + rot.wr, hs_img + (ptrdiff_t)(s_pixA - down) * HB);
        if (s_pullB) cp_async_block(blk + kBwdBlock + rot.wr, ring + (s_edge + s_j) * kSlotF4);
        if (!FAST && t_pullA) cp_async_block(blk + kBwdBlock + rot.wr, ring + (t_edge + (s_j == W - 1 ? 0 : s_j + 1)) * kSlotF4);
        s_pix -= dir;
        s_pixL -= dir;
        s_pixA -= dir;
        --s_j;
    };
    auto lead = [&](const Rows& w) {
        s_hasA = w.hasA; s_hasB = w.hasB; s_pullB = w.pullB; s_pixL = w.pix; s_j = W - 1;
        if (CHAIN) s_edge = w.edge;
        if (upper) { s_on = w.hasB; s_pix = w.pix + down; }
    };
    auto trail = [&](const Rows& w) {
        t_pullA = w.pullA; t_top = w.top; s_pixA = w.pix;
        if (CHAIN) t_edge = w.edge;
        if (!upper) { s_on = w.hasA; s_pix = w.pix; }
    };

    bool hasA = false, hasB = false, row0 = false, pullA = false, pullB = false, push = false, given_up = false;
    int pixA = 0, pixB = 0, edgeA = 0, edgeB = 0;
    auto step = [&](auto tag, const int j, const int jA) {
        constexpr int KIND = decltype(tag)::value;
        constexpr bool FAST = KIND <= kTop, ALL = KIND != kPartial;
        if (CHAIN && (pullB || (!ALL && pullA)))
            wait_for_block(a, blk + kBwdBlock + rot.rd, ring + (pullB ? edgeB + j : edgeA + jA) * kSlotF4, given_up);
        const unsigned flip = CHAIN && pullB ? 0xffffffffu : 0u;
        float2 o_dT[2], o_dL[2], o_dx[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            Quad (&pL)[2] = w ? pLB : pLA;
            const bool NO_T = KIND == kTop && w == 0, here = w ? hasB : hasA;
            o_dT[w] = o_dL[w] = o_dx[w] = make_float2(0.f, 0.f);
            if (!ALL && !here) {
                if (w) clear(carry);
                continue;
            }
            CellIn v;
            read_cell<io_t, true, true>(v, stage_x + rot.rd + w * kCellSlots * 16, stage_n + rot.rd + w * kCellSlots * 16);
            // cells inside the map have constant weights; kap = cfac * the adjoint of h
            float cfac = 0.5f, mT = 1.f, mL = 1.f, oT = 0.f, oL = 0.f;
            bool first = false, top_row = false;
            if (!FAST) {
                first = (w ? j : jA) == 0;
                top_row = w == 0 && row0;
                cfac = (top_row || first) ? 1.f : 0.5f;
                mT = top_row ? 0.f : 1.f;
                mL = (first && !top_row) ? 0.f : 1.f;
                oT = top_row ? ninf : 0.f;
                oL = first ? ninf : 0.f;
            }
            if (NO_T) cfac = 1.f;
            Quad dB, dB_other;                 // upper lanes keep d_BL, the others d_BT
            dB[0] = dB[1] = dB_other[0] = dB_other[1] = make_float2(0.f, 0.f);
            const float2 zero = make_float2(0.f, 0.f);
            const float2 xT = NO_T ? zero : FAST ? v.x : __fmul2_rn(v.x, both(mT)), xL = FAST ? v.x : __fmul2_rn(v.x, both(mL));
            const float2 wT = NO_T ? zero : __fmul2_rn(v.dT, xT), wL = __fmul2_rn(v.dL, xL);
            const float2 tT = FAST ? v.dT : __fmul2_rn(v.dT, both(mT)), tL = FAST ? v.dL : __fmul2_rn(v.dL, both(mL));
            const float2 gyc = __fmul2_rn(v.gy, both(cfac));
            const float dTs[2] = {v.dT.x, v.dT.y}, dLs[2] = {v.dL.x, v.dL.y}, gys[2] = {gyc.x, gyc.y};
            const float2 w_own = choose(upper, wL, wT), w_other = choose(upper, wT, wL);
            const float wo[2] = {w_own.x, w_own.y}, wx[2] = {w_other.x, w_other.y};
            float qTs[2], qLs[2], sTs[2], sLs[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                Quad aT, aL, ht, hl, pd;
                if (!NO_T) lds_in4<float>(aT, params + c * 512);
                lds_in4<float>(aL, params + 1024 + c * 512);
                if (!NO_T) lds_record<rec_t>(ht, blk + rot.rd + (w ? kHA : kUp), c);
                lds_record<rec_t>(hl, blk + rot.rd + (w ? kHB : kHA), c);
                if (w) {
                    lds_in4<float>(pd, blk + kBwdBlock + rot.rd + c * 512);
                    if (CHAIN) { pd[0] = flip_bits(pd[0], flip); pd[1] = flip_bits(pd[1], flip); }
                } else { pd[0] = carry[c][0]; pd[1] = carry[c][1]; }
                if (!ALL && w == 0 && pullA) {
                    lds_in4<float>(pd, blk + kBwdBlock + rot.rd + c * 512);
                    if (CHAIN) { pd[0] = flip_bits(pd[0], 0xffffffffu); pd[1] = flip_bits(pd[1], 0xffffffffu); }
                }
                if (!FAST) {
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        if (w == 0) ht[k] = keep(!top_row, ht[k]);
                        hl[k] = keep(!first, hl[k]);
                    }
                }
                float2 qT = make_float2(0.f, 0.f), qL = qT, sT = qT, sL = qT;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float2 gL = ex2_pair(FAST ? __fmul2_rn(both(dLs[c]), aL[k]) : __ffma2_rn(both(dLs[c]), aL[k], both(oL)));
                    const float2 kap = __ffma2_rn(both(gys[c]), v.c[k], __fmul2_rn(both(cfac), __fadd2_rn(pL[c][k], pd[k])));
                    pL[c][k] = __fmul2_rn(gL, kap);
                    const float2 zL = __fmul2_rn(pL[c][k], hl[k]);
                    dAL[c][k] = __ffma2_rn(zL, both(dLs[c]), dAL[c][k]);
                    qL = __ffma2_rn(zL, aL[k], qL);
                    sL = __ffma2_rn(kap, v.bL[k], sL);
                    if (!NO_T) {
                        const float2 gT = ex2_pair(FAST ? __fmul2_rn(both(dTs[c]), aT[k]) : __ffma2_rn(both(dTs[c]), aT[k], both(oT)));
                        pd[k] = __fmul2_rn(gT, kap);
                        const float2 zT = __fmul2_rn(pd[k], ht[k]);
                        dAT[c][k] = __ffma2_rn(zT, both(dTs[c]), dAT[c][k]);
                        qT = __ffma2_rn(zT, aT[k], qT);
                        sT = __ffma2_rn(kap, v.bT[k], sT);
                    }
                    dB[k] = __ffma2_rn(kap, both(wo[c]), dB[k]);
                    dB_other[k] = __ffma2_rn(kap, both(wx[c]), dB_other[k]);
                }
                if (w) { carry[c][0] = pd[0]; carry[c][1] = pd[1]; }
                else if (!NO_T) {
                    // pT of row A goes to the row above: through its slot, and the ring when that row is in another band
                    sts4(blk + rot.ho + c * 512, quad_f4(pd));
                    if (push) {
                        float4* const up = ring + (edgeA - (CHAIN ? W : 0) + jA) * kSlotF4 + c * 32;
                        if (CHAIN) __stcg(reinterpret_cast<uint4*>(up), invert_bits(quad_f4(pd)));
                        else __stcg(up, quad_f4(pd));
                    }
                }
                sTs[c] = sT.x + sT.y; sLs[c] = sL.x + sL.y;
                qTs[c] = qT.x + qT.y; qLs[c] = qL.x + qL.y;
            }
            const float2 sT = make_float2(sTs[0], sTs[1]), sL = make_float2(sLs[0], sLs[1]);
            if (!NO_T) o_dT[w] = __ffma2_rn(make_float2(qTs[0], qTs[1]), both(kLn2), __fmul2_rn(xT, sT));
            o_dL[w] = __ffma2_rn(make_float2(qLs[0], qLs[1]), both(kLn2), __fmul2_rn(xL, sL));
            o_dx[w] = NO_T ? __fmul2_rn(tL, sL) : __ffma2_rn(tT, sT, __fmul2_rn(tL, sL));
            const float s = reduce_channels(dB, dB_other, hi2, hi1);
            if (db_ok) atomicAdd(db_acc + (long long)(w ? pixB : pixA) * a.acc_pitch, s);
        }
        // sums over states: 2-step exchange over the nq lanes, both rows together
        const float r_dT = reduce_rows(o_dT[0], o_dT[1], nq), r_dL = reduce_rows(o_dL[0], o_dL[1], nq), r_dx = reduce_rows(o_dx[0], o_dx[1], nq);
        const int pix = o_rowB ? pixB : pixA;
        if (o_ok && (ALL || (o_rowB ? hasB : hasA))) {
            const int eo = pix * E + o_ch;
            const float gy = lds_in1<io_t>(stage_o + rot.rd + 192);
            dD = fmaf(gy, lds_in1<io_t>(stage_o + rot.rd), dD);
            store1(static_cast<io_t*>(a.d_dT), eo, r_dT);
            store1(static_cast<io_t*>(a.d_dL), eo, r_dL);
            store1(static_cast<io_t*>(a.d_x), eo, fmaf(gy, D_lane, r_dx));
        }
    };

    // ---- the warp's sequence ---------------------------------------------------------------------
    // 2rr idle steps (in the last of them the right-most state block of row B is requested for the warp below), two steps
    // that only request, W steps per band, one for the last cell of row A, and idle steps until the last warp is done
    const int items = work.items, q_last = CHAIN ? work.q0 + (items - 1) * work.dq : nbands - 1;
    int bi = 0, q = q_last;
    Rows cur = make_rows(bi, q);
    for (int k = 0; k < 2 * rr; ++k) {
        if (k == 2 * rr - 1) request_row_end(cur);
        rot.end_step();
    }
    lead(cur);
    request(std::false_type{});
    rot.end_step();
    trail(cur);
    request(std::false_type{});
    rot.end_step();
    for (int m = 0; m <= items; ++m) {
        if ((q -= work.dq) < 0) { q = q_last; ++bi; }         // (bi, q): the next item; nothing exists past the last one
        hasB = cur.hasB;
        pullB = cur.pullB;
        if (CHAIN) edgeB = cur.edge;
        if (cur.bottom && cur.hasB)                           // nothing arrives from below: B's cells read zeros from S
#pragma unroll
            for (int k = 0; k < 6; ++k) sts4(blk + kBwdBlock + k * 512, make_float4(0.f, 0.f, 0.f, 0.f));
        pixB = cur.pix + down;
        clear(pLB);                                           // a row starts from no right neighbour
        Rows nxt = cur;
        int j = W - 1;
        auto request_ahead = [&]() {
            if (j == 1) {
                nxt = make_rows(bi, q);
                lead(nxt);
            } else if (j == 0) {
                trail(nxt);
            }
            request(std::false_type{});
            // cell (B, 0) has no left block: its buffer is free for the right-most block of the next row
            if (j == 2) request_row_end(make_rows(bi, q));
        };
        const bool inside = cur.hasA && cur.hasB;
        while (j >= 0) {
            if (inside && j < W - 1 && j >= 1) {
                for (; j >= 1; --j) {
                    if (j >= 3) request(std::true_type{});
                    else request_ahead();
                    if (row0) step(StepTag<kTop>{}, j, j + 1);
                    else step(StepTag<kInside>{}, j, j + 1);
                    pixA -= dir;
                    pixB -= dir;
                    rot.end_step();
                }
            }
            request_ahead();
            if (hasA && hasB) step(StepTag<kBorder>{}, j, j == W - 1 ? 0 : j + 1);
            else if (hasA || hasB) step(StepTag<kPartial>{}, j, j == W - 1 ? 0 : j + 1);
            pixA -= dir;
            pixB -= dir;
            rot.end_step();
            if (j == W - 1) {                                 // row A of the band before is done
                if (m == items) break;
                hasA = cur.hasA;
                row0 = cur.row0;
                pullA = cur.pullA;
                if (CHAIN) edgeA = cur.edge;
                push = cur.push;
                pixA = cur.pix;
                clear(pLA);
            }
            --j;
        }
        cur = nxt;
    }
    for (int k = 0; k < 2 * (nwarps - 1 - rr); ++k) rot.end_step();
    cp_async_wait_all();                                      // (only empty groups can be pending here)
}

}  // namespace m2d
