// Forward wave sweep over one band after another: discretisation + two-neighbour recurrence + readout.
// Math per cell as in sweep_fwd.cuh; work split: see wave.cuh.
#pragma once

#include "wave.cuh"

namespace m2d {

// Shared memory: the input stages | hand-off slots per warp | boundary columns per warp (three chunks to
// read, one to write) | one block of zeros.
constexpr int kEdgeCols = 4 * kChunk;
template <typename io_t, int C>
__host__ __device__ inline size_t wave_fwd_smem() {
    return StageLayout<io_t, C, false>::kBytes + kWaveWarps * kSlotBytes<C> + (kWaveWarps * kEdgeCols + 1) * kEdgeFloats<C> * sizeof(float);
}

// The boundary row above a band, chunk by chunk: requested one chunk ahead, checked and parked in shared
// memory when the chunk begins.
template <int C>
struct EdgeReader {
    static constexpr int EF = kEdgeFloats<C>;
    static constexpr int kLoads = kChunk * EF / 4 / 32;
    uint4 v[kLoads];
    bool given_up = false;
    __device__ __forceinline__ bool mine(int k, int c0, int W, int lane) const { return c0 + (lane + 32 * k) / (EF / 4) < W; }
    __device__ __forceinline__ void request(const float* row, int c0, int W, int lane) {
#pragma unroll
        for (int k = 0; k < kLoads; ++k)
            if (mine(k, c0, W, lane)) v[k] = load_shared_line(row + (size_t)c0 * EF + (lane + 32 * k) * 4);
    }
    __device__ __forceinline__ void settle(const ScanArgs& a, const float* row, int c0, int W, int lane, unsigned dst) {
        int polls = 0;
        for (;;) {
            bool ok = true;
#pragma unroll
            for (int k = 0; k < kLoads; ++k) ok = ok && (!mine(k, c0, W, lane) || is_set(v[k]));
            if (__all_sync(0xffffffffu, ok) || given_up) break;
            if (++polls > a.wait_limit || *reinterpret_cast<volatile int*>(a.status) != 0) {
                atomicExch(a.status, 1);
                if (a.host_flag) *reinterpret_cast<volatile int*>(a.host_flag) = 1;
                given_up = true;
            }
            given_up = __any_sync(0xffffffffu, given_up);
            request(row, c0, W, lane);
        }
#pragma unroll
        for (int k = 0; k < kLoads; ++k)
            if (mine(k, c0, W, lane))
                asm volatile("st.shared.v4.u32 [%4], {%0, %1, %2, %3};" ::"r"(~v[k].x), "r"(~v[k].y), "r"(~v[k].z), "r"(~v[k].w), "r"(dst + (lane + 32 * k) * 16) : "memory");
        __syncwarp();
    }
};

template <typename io_t, int C, bool VEC, bool ACT>
__device__ __forceinline__ void wave_forward(const ScanArgs& a, char* smem) {
    typedef StageLayout<io_t, C, false> L;
    constexpr int EF = kEdgeFloats<C>, EB = EF * 4;
    const int lane = threadIdx.x & 31, r = lane >> 2, nq = lane & 3, w = threadIdx.x >> 5;
    const int cgroups = (a.E + C - 1) / C, cg = blockIdx.y * kWaveWarps + w;
    const int ch0 = cg * C, n0 = nq * 4;
    const int chv = min(C, a.E - ch0), nv = min(4, max(0, a.N - n0));
    const int W = a.W, H = a.H, T = W + kWaveRows - 1;

    for (int k = threadIdx.x * 16; k < (int)wave_fwd_smem<io_t, C>(); k += blockDim.x * 16)
        *reinterpret_cast<float4*>(smem + k) = make_float4(0.f, 0.f, 0.f, 0.f);

    float2 aT[4][C / 2], aL[4][C / 2], h[4][C / 2], Dm[C / 2];
#pragma unroll
    for (int c = 0; c < C; ++c) {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const bool ok = c < chv && n < nv;
            const long long idx = (long long)(ch0 + c) * a.N + n0 + n;
            const float t = ok ? load_A<io_t>(a.AT, idx, a.a_log) * kLog2e : 0.f, u = ok ? load_A<io_t>(a.AL, idx, a.a_log) * kLog2e : 0.f;
            if (c & 1) { aT[n][c / 2].y = t; aL[n][c / 2].y = u; } else { aT[n][c / 2].x = t; aL[n][c / 2].x = u; }
            h[n][c / 2] = dup(0.f);
        }
        // x*D enters the readout sum through lane nq == 0
        const float d = nq == 0 && c < chv ? load_D<io_t>(a, ch0 + c) : 0.f;
        if (c & 1) Dm[c / 2].y = d; else Dm[c / 2].x = d;
    }
    const int y_ch = C == 4 ? nq : nq >> 1;                  // the channel whose y this lane stores
    const bool y_lane = y_ch < chv && (C == 4 || (nq & 1) == 0);

    const unsigned stage0 = smem_u32(smem);
    const unsigned lane_x = stage0 + r * L::kCellBytes + w * C * (int)sizeof(io_t);
    const unsigned lane_b = stage0 + r * L::kCellBytes + (L::kTensors * L::kCh + n0) * (int)sizeof(io_t);
    // hand-off inside the warp: lane row r reads slot r and writes slot r + 1 (rows 5/4 of a block apart, so
    // that two neighbouring rows fall into different banks); lane row 0 reads the boundary row and lane row
    // 7 writes it, through the same instructions
    char* const slots = smem + L::kBytes + w * kSlotBytes<C>;
    char* const edge = smem + L::kBytes + kWaveWarps * kSlotBytes<C> + (size_t)w * kEdgeCols * EB;
    const unsigned edge_lane = smem_u32(edge) + nq * C * 4;
    const unsigned slot_in = smem_u32(slots) + r * (EB + EB / 4) + nq * C * 4, slot_out = slot_in + (EB + EB / 4);
    const unsigned zero_lane = smem_u32(smem + L::kBytes) + kWaveWarps * (kSlotBytes<C> + kEdgeCols * EB) + nq * C * 4;

    Stager<io_t, C, false, VEC> stager;
    stager.init(a, blockIdx.y * L::kCh, lane);
    __syncthreads();

    const int chains = (int)gridDim.x / a.chain, chain_id = (int)blockIdx.x / a.chain, cpos = (int)blockIdx.x % a.chain;
    for (int b = chain_id; b < a.B; b += chains)
        for (int band = cpos; band < a.nbands; band += a.chain) {
            const int q0 = band * kWaveRows;
            const size_t id = ((size_t)b * cgroups + cg) * a.nbands + band;
            const float* pull = band > 0 && chv > 0 ? reinterpret_cast<const float*>(a.bnd) + (id - 1) * W * EF : nullptr;
            float* push = band + 1 < a.nbands && chv > 0 && !(a.withhold && b == 0 && band == 0) ? reinterpret_cast<float*>(a.bnd) + id * W * EF : nullptr;
            const bool lrow = q0 + w < H, crow = q0 + r < H, row0 = q0 + r == 0;
            const int lpix = lrow ? scan_pixel(a, b, q0 + w, 0) : 0, cpix = crow ? scan_pixel(a, b, q0 + r, 0) : 0;

            // the gates of cell t ...
            float wT = 0.f, wL = 0.f, oT = 0.f, oL = 0.f;
            // ... and the state of cell t - 1
            float2 gT[4][C / 2], gL[4][C / 2], u[4][C / 2], y[C / 2], yr[C / 2];    // yr: readout of cell t - 2
            float cc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < C / 2; ++e) {
                y[e] = yr[e] = dup(0.f);
#pragma unroll
                for (int k = 0; k < 4; ++k) gT[k][e] = gL[k][e] = u[k][e] = dup(0.f);
            }
            bool y_on = false, yr_on = false, first = false;
            const int ystep = a.dir * a.E;
            io_t* yp = static_cast<io_t*>(a.y) + (cpix * a.E + ch0 + y_ch) - (r + 3) * ystep;    // stepped on before each use
            unsigned in_addr = zero_lane;
            EdgeReader<C> reader;

            auto stage_chunk = [&](int buf, int t0) {
                const int off = buf * kChunk * L::kStepBytes + w * L::kCellBytes, col = t0 - w;
                if (!lrow) return;
                if (VEC && col >= 0 && col + kChunk <= W) {
                    stager.copy_run(stage0 + off, lpix + a.dir * col, a.dir);
                } else {
#pragma unroll 1
                    for (int s = 0; s < kChunk; ++s)
                        if (col + s >= 0 && col + s < W) stager.copy(stage0 + off + s * L::kStepBytes, smem + off + s * L::kStepBytes, lpix + a.dir * (col + s));
                }
            };

            __syncthreads();                                 // every warp is done with the stages of the last band
#pragma unroll
            for (int k = 0; k < kStages - 1; ++k) {
                if (k * kChunk < T) stage_chunk(k, k * kChunk);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            if (pull) reader.request(pull, 0, W, lane);
            int eb = 2;                                      // boundary buffer (of three) of this chunk
#pragma unroll 1
            for (int t0 = 0, buf = 0; t0 < T + 2; t0 += kChunk, buf = (buf + 1) % kStages) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
                __syncthreads();
                if (t0 + (kStages - 1) * kChunk < T) stage_chunk((buf + kStages - 1) % kStages, t0 + (kStages - 1) * kChunk);
                asm volatile("cp.async.commit_group;" ::: "memory");
                eb = eb == 2 ? 0 : eb + 1;
                const unsigned ebase = edge_lane + eb * kChunk * EB;
                if (pull && t0 < W) {
                    reader.settle(a, pull, t0, W, lane, smem_u32(edge) + eb * kChunk * EB);
                    if (t0 + kChunk < W) reader.request(pull, t0 + kChunk, W, lane);
                }
                const unsigned out0 = r < kWaveRows - 1 ? slot_out : edge_lane + 3 * kChunk * EB;
                const int out_step = r < kWaveRows - 1 ? 0 : EB;

                // One step: the gates and input terms of cell t, the recurrence and readout of cell t - 1, and the
                // lane sums and the store of cell t - 2.  They have nothing to do with each other, which is the point: the exponentials of the
                // one fill the latencies of the others.
                auto step = [&](auto tag, const int s) {
                    constexpr bool HEAD = decltype(tag)::value;  // some lane starts, or ends, its row or has just done so
                    const unsigned so = (buf * kChunk + s) * L::kStepBytes;
                    float2 top[4][C / 2];
#pragma unroll
                    for (int k = 0; k < 4; ++k) lds_vec(in_addr + k * 16 * C, top[k]);
                    float2 x[C / 2], dT[C / 2], dL[C / 2], bT[2], bL[2], cN[2];
                    read_staged<io_t, C>(lane_x + so, x);
                    read_staged<io_t, C>(lane_x + so + L::kCh * sizeof(io_t), dT);
                    read_staged<io_t, C>(lane_x + so + 2 * L::kCh * sizeof(io_t), dL);
                    read_staged<io_t, 4>(lane_b + so, bT);
                    read_staged<io_t, 4>(lane_b + so + 16 * sizeof(io_t), bL);
                    read_staged<io_t, 4>(lane_b + so + 32 * sizeof(io_t), cN);
                    float yv = wave_reduce(yr, nq);
                    if (ACT) yv = 0.5f * yv * (1.f + erff(yv * 0.70710678118654752f));
                    yp += ystep;
                    store_if(yr_on, yp, yv);
                    bool y_onN = y_on, firstN = false;
                    if (HEAD) {
                        const int col = t0 + s - r;
                        firstN = col == 0;
                        y_onN = crow && col >= 0 && col < W && y_lane;
                        wT = row0 ? 0.f : (firstN ? 1.f : 0.5f);
                        wL = row0 ? 1.f : (firstN ? 0.f : 0.5f);
                        oT = firstN ? 0.f : -1.f;
                        oL = row0 ? 0.f : -1.f;
                        if (first) {                             // a row starts without a left state
#pragma unroll
                            for (int k = 0; k < 4; ++k)
#pragma unroll
                                for (int e = 0; e < C / 2; ++e) h[k][e] = dup(0.f);
                        }
                    }
                    float2 gTn[4][C / 2], gLn[4][C / 2], un[4][C / 2], yn[C / 2];
#pragma unroll
                    for (int e = 0; e < C / 2; ++e) {
                        const float2 vT = __fmul2_rn(__fmul2_rn(dT[e], x[e]), dup(wT)), vL = __fmul2_rn(__fmul2_rn(dL[e], x[e]), dup(wL));
                        yn[e] = __fmul2_rn(x[e], Dm[e]);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float2 qT = __ffma2_rn(dT[e], aT[k][e], dup(oT)), qL = __ffma2_rn(dL[e], aL[k][e], dup(oL));
                            gTn[k][e] = make_float2(ex2(qT.x), ex2(qT.y));
                            gLn[k][e] = make_float2(ex2(qL.x), ex2(qL.y));
                            const float bt = lane_of(bT, k), bl = lane_of(bL, k);
                            un[k][e] = make_float2(fmaf(vL.x, bl, vT.x * bt), fmaf(vL.y, bl, vT.y * bt));
                            h[k][e] = __ffma2_rn(gL[k][e], h[k][e], __ffma2_rn(gT[k][e], top[k][e], u[k][e]));
                            y[e].x = fmaf(h[k][e].x, cc[k], y[e].x);
                            y[e].y = fmaf(h[k][e].y, cc[k], y[e].y);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) sts_vec(out0 + s * out_step + k * 16 * C, h[k]);
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < C / 2; ++e) {
                        yr[e] = y[e];
                        y[e] = yn[e];
#pragma unroll
                        for (int k = 0; k < 4; ++k) { gT[k][e] = gTn[k][e]; gL[k][e] = gLn[k][e]; u[k][e] = un[k][e]; }
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) cc[k] = lane_of(cN, k);
                    yr_on = y_on;
                    y_on = y_onN;
                    first = firstN;
                    in_addr = row0 ? zero_lane : (r > 0 ? slot_in : (band > 0 ? ebase + s * EB : zero_lane));
                };
                if (t0 > kWaveRows && t0 + kChunk <= W) {
#pragma unroll
                    for (int s = 0; s < kChunk; ++s) step(std::false_type{}, s);
                } else {
#pragma unroll
                    for (int s = 0; s < kChunk; ++s) step(std::true_type{}, s);
                }
                if (push) {                                  // lane row 7's columns of this chunk go out
#pragma unroll
                    for (int k = 0; k < kChunk * EF / 4 / 32; ++k) {
                        const int p = lane + 32 * k, col = t0 + p / (EF / 4) - kWaveRows;
                        if (col >= 0 && col < W)
                            __stcg(reinterpret_cast<uint4*>(push + (size_t)col * EF) + p % (EF / 4), inverted(*reinterpret_cast<const uint4*>(edge + 3 * kChunk * EB + p * 16)));
                    }
                    __syncwarp();
                }
            }
        }
}

}  // namespace m2d
