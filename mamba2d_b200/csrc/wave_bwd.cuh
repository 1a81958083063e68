// Adjoint wave sweep over one band: the recurrence of the gradients, run against the forward's direction,
// and everything that is computed from it.  Work split: see wave.cuh.
//
// With lam = dLoss/dh of a cell (before its own gates):
//     lam = gy*C + pL[i,j+1] + pT[i+1,j],     pT = gT*lam  (to the row above),  pL = gL*lam  (to the left)
//     dA += (pT*h_top)*dT,  (pL*h_left)*dL     d_dT = sum_n pT*h_top*A + x*wT*sum_n lam*BT,  d_dL alike
//     d_x = sum over both directions of w*delta*sum_n lam*B, + gy*D      dB = sum_e lam*w*delta*x    dC = sum_e gy*h
// The sweep walks the forward's anti-diagonals backwards: the cells of step t are the ones whose states the
// recompute sweep wrote as record block t, so block t - 1 holds a lane's left state, and its neighbour
// lane's part of the same block is the state above.
#pragma once

#include "wave_fwd.cuh"

namespace m2d {

// Sums a lane keeps over all its cells.
template <int C>
struct WaveSums {
    float2 dAT[4][C / 2], dAL[4][C / 2], dD[C / 2];
};

template <typename io_t, int C, bool VEC>
__device__ __forceinline__ void wave_adjoint_band(const ScanArgs& a, char* smem, const WaveLane<io_t, C, VEC, true>& ln, WaveSums<C>& sum, int b,
                                                  int slot, int band, const float4* rec) {
    typedef WaveSmem<io_t, C, true> S;
    typedef typename S::Stage L;
    typedef RecordBlock<C> Rec;
    constexpr int EF = kEdgeFloats<C>, EB = EF * 4;
    const int lane = ln.lane, r = ln.r, nq = ln.nq, w = ln.w, chv = ln.chv;
    const float2 (&aT)[4][C / 2] = ln.aT;
    const float2 (&aL)[4][C / 2] = ln.aL;
    const int W = a.W, H = a.H, T = W + kWaveRows - 1;
    const int rr = kWaveRows - 1 - r;                        // distance from the leading lane row (the bottom one)
    const int o_ch = C == 4 ? nq : nq >> 1;                  // the channel whose d_x, d_dT, d_dL this lane stores
    const bool o_lane = o_ch < chv && (C == 4 || (nq & 1) == 0);

    char* const edge = smem + S::kEdge + w * kEdgeCols * EB;
    char* const above = smem + S::kAbove + w * S::kChunks * kChunk * EB;
    const unsigned edge_lane = smem_u32(edge) + nq * C * 4, above_lane = smem_u32(above) + nq * C * 4;
    const unsigned slot0 = smem_u32(smem + S::kSlots + w * kSlotBytes<C>) + nq * C * 4;
    const unsigned slot_in = slot0 + (r + 1) * (EB + EB / 4), slot_out = slot0 + r * (EB + EB / 4);
    const unsigned zero_lane = smem_u32(smem + S::kZeros) + nq * C * 4;
    const unsigned stage0 = smem_u32(smem);
    float* const part = reinterpret_cast<float*>(smem + S::kPart);
    const unsigned part_lane = smem_u32(part) + w * S::kPartBytes + lane * 16;

    const int q0 = band * kWaveRows;
    const size_t id = ((size_t)slot * ln.cgroups + ln.cg) * a.nbands + band;
    float* pull = band + 1 < a.nbands && chv > 0 ? reinterpret_cast<float*>(a.bnd_up) + id * W * EF : nullptr;
    float* push = band > 0 && band != a.mute_up && chv > 0 ? reinterpret_cast<float*>(a.bnd_up) + (id - 1) * W * EF : nullptr;
    const float* top_row = band > 0 && chv > 0 ? reinterpret_cast<const float*>(a.bnd) + (id - 1) * W * EF : nullptr;   // as the recompute sweep left it
    const bool lrow = q0 + w < H, crow = q0 + r < H, row0 = q0 + r == 0;
    const int lpix = lrow ? scan_pixel(a, b, q0 + w, W - 1) : 0, cpix = crow ? scan_pixel(a, b, q0 + r, W - 1) : 0;

    float2 pL[4][C / 2], hl[4][C / 2];                       // hl: left state of the last cell = own state of the next
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < C / 2; ++e) pL[k][e] = dup(0.f);
    Rec next[2];                                             // the record is requested two steps ahead (T >= 9)
    next[0].load(rec + (size_t)(T - 1) * (Rec::kVecs * 32), lane);
    next[0].unpack(hl);
    next[0].load(rec + (size_t)(T - 2) * (Rec::kVecs * 32), lane);
    next[1].load(rec + (size_t)(T - 3) * (Rec::kVecs * 32), lane);
    // neighbour weights; lane row 0 of the image has no row above
    float wT = row0 ? 0.f : 0.5f, wL = row0 ? 1.f : 0.5f, oT = -1.f;
    const float oL = row0 ? 0.f : -1.f;
    bool live = false;
    const int ostep = a.dir * a.E;
    int ooff = cpix * a.E + ln.ch0 + o_ch + rr * ostep;      // at column W - 1 - (tau - rr)
    const bool pull_here = pull && r == kWaveRows - 1;
    const unsigned in_fixed = crow && q0 + r + 1 < H && r < kWaveRows - 1 ? slot_in : zero_lane;
    unsigned in_addr = zero_lane;
    EdgeReader<C> reader;

    // tau counts steps from the end: lane row r is at column W - 1 - (tau - rr)
    auto stage_chunk = [&](int buf, int tau0) {
        const int off = buf * kChunk * L::kStepBytes + w * L::kCellBytes, col = tau0 - (kWaveRows - 1 - w);    // mirrored column
        if (lrow) {
            if (VEC && col >= 0 && col + kChunk <= W) {
                ln.stager.template copy_run<false>(stage0 + off, lpix - a.dir * col, -a.dir);
            } else {
#pragma unroll 1
                for (int s = 0; s < kChunk; ++s)
                    if (col + s >= 0 && col + s < W) ln.stager.template copy<false>(stage0 + off + s * L::kStepBytes, smem + off + s * L::kStepBytes, lpix - a.dir * (col + s));
            }
        }
        if (top_row) {                                       // the states above lane row 0's cells
#pragma unroll
            for (int k = 0; k < kChunk * EF / 4 / 32; ++k) {
                const int p = lane + 32 * k, c = W + kWaveRows - 2 - tau0 - p / (EF / 4);
                if (c >= 0 && c < W) cp_async16(smem_u32(above + buf * kChunk * EB + p * 16), top_row + (size_t)c * EF + p % (EF / 4) * 4);
            }
        }
    };

    __syncthreads();                                         // every warp is done with the stages of the last sweep
    if (!lrow)                                               // rows below the image read as zeros
        for (int k = lane * 16; k < L::kCellBytes; k += 512)
            for (int c = 0; c < S::kChunks * kChunk; ++c) *reinterpret_cast<float4*>(smem + c * L::kStepBytes + w * L::kCellBytes + k) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < S::kChunks - 1; ++k) {
        if (k * kChunk < T) stage_chunk(k, k * kChunk);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (pull) reader.request(pull, 0, W, lane);
    int eb = 2;
#pragma unroll 1
    for (int tau0 = 0, buf = 0; tau0 < T; tau0 += kChunk, buf = (buf + 1) % S::kChunks) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::kChunks - 2) : "memory");
        __syncthreads();
        if (tau0 + (S::kChunks - 1) * kChunk < T) stage_chunk((buf + S::kChunks - 1) % S::kChunks, tau0 + (S::kChunks - 1) * kChunk);
        asm volatile("cp.async.commit_group;" ::: "memory");
        eb = eb == 2 ? 0 : eb + 1;
        if (pull && tau0 < W) {
            reader.template settle<false>(a, pull, tau0, W, lane, smem_u32(edge) + eb * kChunk * EB);
            if (tau0 + kChunk < W) reader.request(pull, tau0 + kChunk, W, lane);
        }

        auto step = [&](auto tag, const int s) {
            constexpr bool HEAD = decltype(tag)::value;
            const unsigned so = (buf * kChunk + s) * L::kStepBytes;
            const int t = T - 1 - tau0 - s;                  // the record block of these cells
            in_addr = pull_here ? edge_lane + (eb * kChunk + s) * EB : in_fixed;
            float2 lam[4][C / 2], ht[4][C / 2], h[4][C / 2];
#pragma unroll
            for (int k = 0; k < 4; ++k) lds_vec(in_addr + k * 16 * C, lam[k]);               // pT of the row below
            float2 x[C / 2], dT[C / 2], dL[C / 2], gy[C / 2], bT[2], bL[2], cc[2];
            read_staged<io_t, C>(ln.lane_x + so, x);
            read_staged<io_t, C>(ln.lane_x + so + L::kCh * sizeof(io_t), dT);
            read_staged<io_t, C>(ln.lane_x + so + 2 * L::kCh * sizeof(io_t), dL);
            read_staged<io_t, C>(ln.lane_x + so + 3 * L::kCh * sizeof(io_t), gy);
            read_staged<io_t, 4>(ln.lane_b + so, bT);
            read_staged<io_t, 4>(ln.lane_b + so + 16 * sizeof(io_t), bL);
            read_staged<io_t, 4>(ln.lane_b + so + 32 * sizeof(io_t), cc);
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int e = 0; e < C / 2; ++e) h[k][e] = hl[k][e];
            next[0].unpack(hl);
            next[0] = next[1];
            if (!HEAD || t >= 3) next[1].load(rec + (size_t)(t - 3) * (Rec::kVecs * 32), lane);
            else next[1].clear();
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int e = 0; e < C / 2; ++e) {
                    ht[k][e].x = __shfl_up_sync(0xffffffffu, hl[k][e].x, 4);
                    ht[k][e].y = __shfl_up_sync(0xffffffffu, hl[k][e].y, 4);
                }
            lds_block_if(r == 0, top_row ? above_lane + (buf * kChunk + s) * EB : zero_lane, ht);
            if (HEAD) {
                const int cm = tau0 + s - rr;                // mirrored column
                const bool first = cm == W - 1;              // column 0
                live = crow && cm >= 0 && cm < W;
                wT = row0 ? 0.f : (first ? 1.f : 0.5f);
                wL = row0 ? 1.f : (first ? 0.f : 0.5f);
                oT = first ? 0.f : -1.f;
                if (cm <= 0 || cm >= W) {                    // nothing comes from beyond the last column, and outside the image lam = 0
                                                             // (hl stays: it may be the state of the next, real, cell)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int e = 0; e < C / 2; ++e) {
                            pL[k][e] = dup(0.f);
                            if (cm != 0) lam[k][e] = dup(0.f);
                        }
                    if (cm != 0) {
#pragma unroll
                        for (int e = 0; e < C / 2; ++e) x[e] = dT[e] = dL[e] = gy[e] = dup(0.f);
                    }
                }
            }
            float2 oX[C / 2], oDT[C / 2], oDL[C / 2], pB[4], pBL[4], pC[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) pB[k] = pBL[k] = pC[k] = dup(0.f);
            const unsigned out = r > 0 ? slot_out : edge_lane + (3 * kChunk + s) * EB;
#pragma unroll
            for (int e = 0; e < C / 2; ++e) {
                const float2 xT = __fmul2_rn(x[e], dup(wT)), xL = __fmul2_rn(x[e], dup(wL));
                const float2 vT = __fmul2_rn(dT[e], xT), vL = __fmul2_rn(dL[e], xL);
                float2 qT = dup(0.f), qL = dup(0.f), sT = dup(0.f), sL = dup(0.f);
                sum.dD[e] = __ffma2_rn(gy[e], x[e], sum.dD[e]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 eT = __ffma2_rn(dT[e], aT[k][e], dup(oT)), eL = __ffma2_rn(dL[e], aL[k][e], dup(oL));
                    const float2 gT = make_float2(ex2(eT.x), ex2(eT.y)), gL = make_float2(ex2(eL.x), ex2(eL.y));
                    const float bt = lane_of(bT, k), bl = lane_of(bL, k), cv = lane_of(cc, k);
                    float2 l = __fadd2_rn(lam[k][e], pL[k][e]);
                    l.x = fmaf(gy[e].x, cv, l.x);
                    l.y = fmaf(gy[e].y, cv, l.y);
                    lam[k][e] = __fmul2_rn(gT, l);           // pT of this cell, on its way up
                    pL[k][e] = __fmul2_rn(gL, l);
                    const float2 zT = __fmul2_rn(lam[k][e], ht[k][e]), zL = __fmul2_rn(pL[k][e], hl[k][e]);
                    sum.dAT[k][e] = __ffma2_rn(zT, dT[e], sum.dAT[k][e]);
                    sum.dAL[k][e] = __ffma2_rn(zL, dL[e], sum.dAL[k][e]);
                    qT = __ffma2_rn(zT, aT[k][e], qT);
                    qL = __ffma2_rn(zL, aL[k][e], qL);
                    sT.x = fmaf(l.x, bt, sT.x); sT.y = fmaf(l.y, bt, sT.y);
                    sL.x = fmaf(l.x, bl, sL.x); sL.y = fmaf(l.y, bl, sL.y);
                    pB[k] = __ffma2_rn(l, vT, pB[k]);
                    pBL[k] = __ffma2_rn(l, vL, pBL[k]);
                    pC[k] = __ffma2_rn(gy[e], h[k][e], pC[k]);
                }
                // (A is kept times log2(e))
                oDT[e] = __ffma2_rn(xT, sT, __fmul2_rn(qT, dup(kLn2)));
                oDL[e] = __ffma2_rn(xL, sL, __fmul2_rn(qL, dup(kLn2)));
                oX[e] = __ffma2_rn(__fmul2_rn(dT[e], dup(wT)), sT, __ffma2_rn(__fmul2_rn(dL[e], dup(wL)), sL, __fmul2_rn(gy[e], ln.Dm[e])));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) sts_vec(out + k * 16 * C, lam[k]);
            __syncwarp();
            {
                const float2 fT[2] = {make_float2(pB[0].x + pB[0].y, pB[1].x + pB[1].y), make_float2(pB[2].x + pB[2].y, pB[3].x + pB[3].y)};
                const float2 fL[2] = {make_float2(pBL[0].x + pBL[0].y, pBL[1].x + pBL[1].y), make_float2(pBL[2].x + pBL[2].y, pBL[3].x + pBL[3].y)};
                const float2 fC[2] = {make_float2(pC[0].x + pC[0].y, pC[1].x + pC[1].y), make_float2(pC[2].x + pC[2].y, pC[3].x + pC[3].y)};
                sts_vec(part_lane + (s * 3) * 512, fT);
                sts_vec(part_lane + (s * 3 + 1) * 512, fL);
                sts_vec(part_lane + (s * 3 + 2) * 512, fC);
            }
            const bool on = live && o_lane;
            const float rx = wave_reduce(oX, nq), rT = wave_reduce(oDT, nq), rL = wave_reduce(oDL, nq);
            store3_if(on, static_cast<io_t*>(a.d_x) + ooff, static_cast<io_t*>(a.d_dT) + ooff, static_cast<io_t*>(a.d_dL) + ooff, rx, rT, rL);
            ooff -= ostep;
        };
        if (tau0 >= kWaveRows && tau0 + kChunk < W) {
#pragma unroll
            for (int s = 0; s < kChunk; ++s) step(std::false_type{}, s);
        } else {
#pragma unroll
            for (int s = 0; s < kChunk; ++s)
                if (tau0 + s < T) step(std::true_type{}, s);
        }
        if (push) {                                          // lane row 0's pT of this chunk goes out
#pragma unroll
            for (int k = 0; k < kChunk * EF / 4 / 32; ++k) {
                const int p = lane + 32 * k, cm = tau0 + p / (EF / 4) - (kWaveRows - 1);
                if (cm >= 0 && cm < W)
                    __stcg(reinterpret_cast<uint4*>(push + (size_t)cm * EF) + p % (EF / 4), inverted(*reinterpret_cast<const uint4*>(edge + 3 * kChunk * EB + p * 16)));
            }
        }
        // the warps' shares of dBT, dBL, dC of the chunk's cells
        __syncthreads();
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            const int it = threadIdx.x + h2 * kWaveWarps * 32;
            if (it >= kChunk * 3 * kWaveRows * 4) break;
            const int s = it / 96, q = it % 96 / 32, pr = it % 32 / 4, n = it % 4 * 4;
            const int cm = tau0 + s - (kWaveRows - 1 - pr);
            if (q0 + pr < H && cm >= 0 && cm < W && n < a.N) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int k = 0; k < kWaveWarps; ++k) {
                    const float4 u = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(part) + k * S::kPartBytes + it * 16);
                    v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
                }
                float* dst = (q == 0 ? a.accBT : (q == 1 ? a.accBL : a.accC)) + (long long)scan_pixel(a, b, q0 + pr, W - 1 - cm) * a.acc_pitch + n;
                if (a.acc_vec) {
                    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
                } else {
                    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (n + k < a.N) atomicAdd(dst + k, e[k]);
                }
            }
        }
    }
}

template <typename io_t, int C, bool VEC>
__device__ __forceinline__ void wave_backward(const ScanArgs& a, char* smem) {
    typedef RecordBlock<C> Rec;
    WaveLane<io_t, C, VEC, true> ln;
    ln.init(a, smem);
    WaveSums<C> sum;
#pragma unroll
    for (int e = 0; e < C / 2; ++e) {
        sum.dD[e] = dup(0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) sum.dAT[k][e] = sum.dAL[k][e] = dup(0.f);
    }
    const int chains = (int)gridDim.x / a.chain, chain_id = (int)blockIdx.x / a.chain, cpos = (int)blockIdx.x % a.chain;
    const size_t band_rec = (size_t)(a.W + kWaveRows - 1) * Rec::kVecs * 32;
    for (int b = chain_id; b < a.B; b += chains) {
        // (channel groups beyond E write their record, and nothing else, into the padding of the last group)
        float4* const rec = a.hs + ((size_t)chain_id * gridDim.y * kWaveWarps + ln.cg) * a.nbands * band_rec;
        int band = cpos;
        for (; band < a.nbands; band += a.chain) wave_forward_band<io_t, C, VEC, kRecord, true>(a, smem, ln, b, chain_id, band, rec + band * band_rec);
        for (band -= a.chain; band >= 0; band -= a.chain) wave_adjoint_band<io_t, C, VEC>(a, smem, ln, sum, b, chain_id, band, rec + band * band_rec);
    }
    // ---- per-(channel, state) sums over the eight lane rows, then one atomic per value --------------------
#pragma unroll
    for (int c = 0; c < C; ++c) {
        auto rows = [](float v) {
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            return v + __shfl_xor_sync(0xffffffffu, v, 16);
        };
        const float dD = rows(c & 1 ? sum.dD[c / 2].y : sum.dD[c / 2].x);
        if (ln.lane == 0 && c < ln.chv) atomicAdd(a.accD + ln.ch0 + c, dD);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float t = rows(c & 1 ? sum.dAT[k][c / 2].y : sum.dAT[k][c / 2].x), l = rows(c & 1 ? sum.dAL[k][c / 2].y : sum.dAL[k][c / 2].x);
            if (ln.r == 0 && c < ln.chv && k < ln.nv) {
                // with A given as A_log the gradient asked for is d_A_log = d_A * A (A = -exp(A_log),
                // models/kernels/wavefront_cuda.py:72-73); the product is linear, so every CTA scales its share
                const long long idx = (long long)(ln.ch0 + c) * a.N + ln.n0 + k;
                atomicAdd(a.accAT + idx, t * (a.a_log ? load_A<io_t>(a.AT, idx, 1, true) : 1.f));
                atomicAdd(a.accAL + idx, l * (a.a_log ? load_A<io_t>(a.AL, idx, 1, true) : 1.f));
            }
        }
    }
}

}  // namespace m2d
