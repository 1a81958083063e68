// Forward wave sweep over one band after another: discretisation + two-neighbour recurrence + readout.
// Math per cell: scan_args.cuh; work split: wave.cuh.
#pragma once

#include "wave.cuh"

namespace m2d {

// The boundary row above a band, COLS columns at a time: requested one such piece ahead, checked and parked in shared
// memory before the first step that needs it.
template <int C, int COLS = kChunk>
struct EdgeReader {
    static constexpr int EF = kEdgeFloats<C>;
    static constexpr int kLoads = COLS * EF / 4 / 32;
    static_assert(COLS * EF % 128 == 0, "whole loads of a warp");
    uint4 v[kLoads];
    bool given_up = false;
    __device__ __forceinline__ bool mine(int k, int c0, int W, int lane) const { return c0 + (lane + 32 * k) / (EF / 4) < W; }
    __device__ __forceinline__ void request(const float* row, int c0, int W, int lane) {
#pragma unroll
        for (int k = 0; k < kLoads; ++k)
            if (mine(k, c0, W, lane)) v[k] = load_shared_line(row + (size_t)c0 * EF + (lane + 32 * k) * 4);
    }
    // KEEP: also put the values back where they came from, as plain floats (this warp is their only reader).
    template <bool KEEP>
    __device__ __forceinline__ void settle(const ScanArgs& a, float* row, int c0, int W, int lane, unsigned dst) {
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
            if (mine(k, c0, W, lane)) {
                const uint4 f = inverted(v[k]);
                asm volatile("st.shared.v4.u32 [%4], {%0, %1, %2, %3};" ::"r"(f.x), "r"(f.y), "r"(f.z), "r"(f.w), "r"(dst + (lane + 32 * k) * 16) : "memory");
                if (KEEP) __stcg(reinterpret_cast<uint4*>(row + (size_t)c0 * EF) + lane + 32 * k, f);
            }
        __syncwarp();
    }
};

// What the sweep is for.
enum WaveKind { kReadout, kReadoutGelu, kRecord };

// One band of image b (the `slot`-th image or list the launch has boundary rows for), top to bottom of the
// image's dependences: lane row 0 leads, columns ascending.  kRecord writes
// every state to `rec` ([t][m][lane], zeros for lanes outside the image) instead of the readout.
//
// COLS: boundary columns handed over at a time, a whole chunk of four or pairs: edge_pairs (plan.cuh).  Pairs are also taken
// as late as they can be, before the step that reads the first of them.
template <typename io_t, int C, bool VEC, WaveKind KIND, bool BWD, int COLS = kChunk>
__device__ __forceinline__ void wave_forward_band(const ScanArgs& a, char* smem, const WaveLane<io_t, C, VEC, BWD>& ln, int b, int slot, int band, float4* rec) {
    typedef WaveSmem<io_t, C, BWD> S;
    typedef typename S::Stage L;
    constexpr int EF = kEdgeFloats<C>, EB = EF * 4;
    const int lane = ln.lane, r = ln.r, nq = ln.nq, w = ln.w, chv = ln.chv;
    const float2 (&aT)[4][C / 2] = ln.aT;
    const float2 (&aL)[4][C / 2] = ln.aL;
    const float2 (&Dm)[C / 2] = ln.Dm;
    const int W = a.W, H = a.H, T = W + kWaveRows - 1;
    const int y_ch = C == 4 ? nq : nq >> 1;                  // the channel whose y this lane stores
    const bool y_lane = y_ch < chv && (C == 4 || (nq & 1) == 0);
    // hand-off inside the warp: lane row r reads slot r and writes slot r + 1; lane row 0 reads the boundary
    // row and lane row 7 writes it, through the same instructions
    char* const edge = smem + S::kEdge + w * kEdgeCols * EB;
    const unsigned edge_lane = smem_u32(edge) + nq * C * 4;
    const unsigned slot_in = smem_u32(smem + S::kSlots + w * kSlotBytes<C>) + r * (EB + EB / 4) + nq * C * 4, slot_out = slot_in + (EB + EB / 4);
    const unsigned zero_lane = smem_u32(smem + S::kZeros) + nq * C * 4;
    const unsigned stage0 = smem_u32(smem);

    const int q0 = band * kWaveRows;
    float* const rows = reinterpret_cast<float*>(a.bnd) + ((size_t)slot * ln.cgroups + ln.cg) * a.bnd_rows * W * EF;
    float* pull = band > 0 && chv > 0 ? rows + (size_t)((band - 1) % a.bnd_rows) * W * EF : nullptr;
    float* push = band + 1 < a.nbands && chv > 0 && !(a.withhold && b == 0 && band == 0) ? rows + (size_t)(band % a.bnd_rows) * W * EF : nullptr;
    const bool lrow = q0 + w < H, crow = q0 + r < H, row0 = q0 + r == 0;
    const int lpix = lrow ? scan_pixel(a, b, q0 + w, 0) : 0, cpix = crow ? scan_pixel(a, b, q0 + r, 0) : 0;

    float2 h[4][C / 2];
    // the gates of cell t ...
    float wT = 0.f, wL = 0.f, oT = 0.f, oL = 0.f;
    // ... and the state of cell t - 1
    float2 gT[4][C / 2], gL[4][C / 2], u[4][C / 2], y[C / 2], yr[C / 2];    // yr: readout of cell t - 2
    float cc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < C / 2; ++e) {
        y[e] = yr[e] = dup(0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) gT[k][e] = gL[k][e] = u[k][e] = h[k][e] = dup(0.f);
    }
    bool y_on = false, yr_on = false, first = false;
    const int ystep = a.dir * a.E;
    io_t* yp = static_cast<io_t*>(a.y) + (cpix * a.E + ln.ch0 + y_ch) - (r + 3) * ystep;    // stepped on before each use
    unsigned in_addr = zero_lane;
    EdgeReader<C, COLS> reader;
    typedef RecordBlock<C> Rec;
    // Where the chunk's columns are sent from: from the steps, or, with bf16 I/O and four channels per lane, from one place
    // behind them (512x512x192 bf16 1020 us from the steps, 1000 from behind; fp32 1004 and 1009; 512x512x64 fp32, two
    // channels per lane, 608 and 638).
    constexpr bool kGiveAfter = C == 4 && COLS == kChunk && sizeof(io_t) == 2;

    auto stage_chunk = [&](int buf, int t0) {
        const int off = buf * kChunk * L::kStepBytes + w * L::kCellBytes, col = t0 - w;
        if (!lrow) return;
        if (VEC && col >= 0 && col + kChunk <= W) {
            ln.stager.template copy_run<KIND == kRecord>(stage0 + off, lpix + a.dir * col, a.dir);
        } else {
#pragma unroll 1
            for (int s = 0; s < kChunk; ++s)
                if (col + s >= 0 && col + s < W) ln.stager.template copy<KIND == kRecord>(stage0 + off + s * L::kStepBytes, smem + off + s * L::kStepBytes, lpix + a.dir * (col + s));
        }
    };

    __syncthreads();                                 // every warp is done with the stages of the last band
    if (KIND == kRecord && !lrow)                    // rows below the image read as zeros
        for (int k = lane * 16; k < L::kCellBytes; k += 512)
            for (int c = 0; c < S::kChunks * kChunk; ++c) *reinterpret_cast<float4*>(smem + c * L::kStepBytes + w * L::kCellBytes + k) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < S::kChunks - 1; ++k) {
        if (k * kChunk < T) stage_chunk(k, k * kChunk);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (pull) reader.request(pull, 0, W, lane);
    int eb = 2;                                      // boundary buffer (of three) of this chunk
#pragma unroll 1
    for (int t0 = 0, buf = 0; t0 < T + 2; t0 += kChunk, buf = (buf + 1) % S::kChunks) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::kChunks - 2) : "memory");
        __syncthreads();
        if (t0 + (S::kChunks - 1) * kChunk < T) stage_chunk((buf + S::kChunks - 1) % S::kChunks, t0 + (S::kChunks - 1) * kChunk);
        asm volatile("cp.async.commit_group;" ::: "memory");
        eb = eb == 2 ? 0 : eb + 1;
        const unsigned ebase = edge_lane + eb * kChunk * EB;
        auto take_edge = [&](const int s) {                              // columns t0 + s ... of the row above
            if (s % COLS == 0 && pull && t0 + s < W) {
                reader.template settle<KIND == kRecord>(a, pull, t0 + s, W, lane, smem_u32(edge) + (eb * kChunk + s) * EB);
                if (t0 + s + COLS < W) reader.request(pull, t0 + s + COLS, W, lane);
            }
        };
        auto give_edge = [&](const int s) {                              // lane row 7's columns of the steps up to s go out
            if (s % COLS != COLS - 1 || !push) return;
#pragma unroll
            for (int k = 0; k < COLS * EF / 4 / 32; ++k) {
                const int p = lane + 32 * k, from = s + 1 - COLS, col = t0 + from + p / (EF / 4) - kWaveRows;
                if (col >= 0 && col < W)
                    __stcg(reinterpret_cast<uint4*>(push + (size_t)col * EF) + p % (EF / 4),
                           inverted(*reinterpret_cast<const uint4*>(edge + (3 * kChunk + from) * EB + p * 16)));
            }
            __syncwarp();
        };
        if (COLS == kChunk) take_edge(0);
        const unsigned out0 = r < kWaveRows - 1 ? slot_out : edge_lane + 3 * kChunk * EB;
        const int out_step = r < kWaveRows - 1 ? 0 : EB;

        // One step: the gates and input terms of cell t, the recurrence and readout of cell t - 1, and the
        // lane sums and the store of cell t - 2.  They have nothing to do with each other, which is the point:
        // the exponentials of the one fill the latencies of the others.
        auto step = [&](auto tag, const int s) {
            constexpr bool HEAD = decltype(tag)::value;  // some lane starts, or ends, its row or has just done so
            const unsigned so = (buf * kChunk + s) * L::kStepBytes;
            float2 top[4][C / 2];
#pragma unroll
            for (int k = 0; k < 4; ++k) lds_vec(in_addr + k * 16 * C, top[k]);
            float2 x[C / 2], dT[C / 2], dL[C / 2], bT[2], bL[2], cN[2] = {dup(0.f), dup(0.f)};
            read_staged<io_t, C>(ln.lane_x + so, x);
            read_staged<io_t, C>(ln.lane_x + so + L::kCh * sizeof(io_t), dT);
            read_staged<io_t, C>(ln.lane_x + so + 2 * L::kCh * sizeof(io_t), dL);
            read_staged<io_t, 4>(ln.lane_b + so, bT);
            read_staged<io_t, 4>(ln.lane_b + so + 16 * sizeof(io_t), bL);
            if (KIND != kRecord) read_staged<io_t, 4>(ln.lane_b + so + 32 * sizeof(io_t), cN);
            if (KIND != kRecord) {
                float yv = wave_reduce(yr, nq);
                if (KIND == kReadoutGelu) yv = gelu_erf(yv);
                yp += ystep;
                store_if(yr_on, yp, yv);
            }
            bool y_onN = y_on, firstN = false;
            if (HEAD) {
                const int col = t0 + s - r;
                firstN = col == 0;
                y_onN = crow && col >= 0 && col < W && (KIND == kRecord || y_lane);
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
            if (KIND == kRecord) {
                const int t = t0 + s - 1;
                Rec out;
                out.pack(h);
                if (HEAD && !y_on) out.clear();
                if (!HEAD || (t >= 0 && t < T)) out.store(rec + (size_t)t * (Rec::kVecs * 32), lane);
            }
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
        // (the boundary column of step s is read in step s + 1, where the recurrence of its cells is)
        auto steps = [&](auto tag) {
#pragma unroll
            for (int s = 0; s < kChunk; ++s) {
                if (COLS < kChunk && s > 0) take_edge(s - 1);
                step(tag, s);
                if (!kGiveAfter) give_edge(s);
            }
        };
        if (t0 > kWaveRows && t0 + kChunk <= W) steps(std::false_type{});
        else steps(std::true_type{});
        if (kGiveAfter) give_edge(kChunk - 1);
    }
}

template <typename io_t, int C, bool VEC, WaveKind KIND, int COLS = kChunk>
__device__ __forceinline__ void wave_forward(const ScanArgs& a, char* smem) {
    WaveLane<io_t, C, VEC, false> ln;
    ln.init(a, smem);
    const int chains = (int)gridDim.x / a.chain, chain_id = (int)blockIdx.x / a.chain, cpos = (int)blockIdx.x % a.chain;
    for (int b = chain_id; b < a.B; b += chains)
        for (int band = cpos; band < a.nbands; band += a.chain) wave_forward_band<io_t, C, VEC, KIND, false, COLS>(a, smem, ln, b, chain_id, band, nullptr);
}

}  // namespace m2d
