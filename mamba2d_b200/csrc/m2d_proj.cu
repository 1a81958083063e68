// Fused parameter projections around the wavefront scan (C ABI in m2d_proj.h).
//
//   dtproj_fwd   delta = softplus(r @ W^T + b) for both directions, one pass over (P,E)
//   dtproj_bwd   softplus', weight / bias gradients and the gradient of r, one pass over (P,E)
//   xproj_wgrad  d_Wx = d_proj^T @ x, a reduction over all pixels split across the GPU
//
// The reference does this in PyTorch (proj_params, models/kernels/wavefront_cuda.py:63-95, and
// its autograd backward).  All three kernels are HBM-streaming: a thread owns one channel, lanes of
// a warp own consecutive channels of one pixel (coalesced rows), the per-pixel rank-R vectors sit
// in shared memory, and the big reductions over pixels stay in registers until the end of the
// kernel, when each CTA writes one partial result that a small second kernel sums.
#include <type_traits>
#include "m2d_proj.h"

#include "common.cuh"
#include "launch.cuh"
#include "plan.cuh"
#include "proj_mma.cuh"
#include "wgrad_tc.cuh"

namespace m2d {

constexpr int kProjIters = 8;          // pixels per thread per tile

struct ProjPlan {
    int EB, PS, threads, TP, RB, gx;
    int ntiles;
    // x-projection weight gradient
    int tilesK, tilesE, slabs, rows_per_slab, K;
    size_t dt_partials, wg_partials;   // bytes
};

struct ProjArgs {
    Clear clear;
    int P, pitch, ntiles;              // every element index fits 31 bits (checked on the host)
    int E, R, EB, PS, TP;
    int params_f32;                    // weights and biases are fp32, rounded to io_t when read
    int wide16;                        // bf16 backward: rows and pointers allow 16-byte copies
    const void *proj, *WT, *WL, *bT, *bL;
    void *dT, *dL;
    const void *g_dT, *g_dL;
    void* d_proj;
    float* partials;                   // [dir][cta][RB+1][EB]
};

struct WgArgs {
    int P, pitch;
    int E, K, rows_per_slab;
    const void *x, *d_proj;
    float* partials;                   // [slab][K][E]
};

static int check_proj(const m2d_proj_desc* d) {
    if (!d) return M2D_ERR_NULL;
    if (d->struct_bytes != sizeof(m2d_proj_desc)) return M2D_ERR_ABI;
    if (d->dtype != M2D_F32 && d->dtype != M2D_BF16) return M2D_ERR_DTYPE;
    if (d->flags & ~M2D_PROJ_PARAMS_F32) return M2D_ERR_FLAGS;
    if (d->P < 1 || d->E < 1 || d->R < 1 || d->N < 1) return M2D_ERR_SHAPE;
    if (d->E > M2D_PROJ_MAX_E || d->R > M2D_PROJ_MAX_R) return M2D_ERR_TOO_LARGE;
    if (d->proj_pitch < 2ll * d->R + 3ll * d->N) return M2D_ERR_PITCH;
    {
        // the kernels stage 8 pixels x RB ranks per EB channels with two values per thread at most
        const int EB = (d->E + 31) / 32 * 32;
        const int RB = d->R <= 4 ? 4 : d->R <= 8 ? 8 : d->R <= 16 ? 16 : d->R <= 32 ? 32 : 64;
        if (4 * RB > EB) return M2D_ERR_SHAPE;
    }
    const long long widest = d->proj_pitch > d->E ? d->proj_pitch : d->E;
    // the kernels use 31-bit element indices, as the scan does (with room for the look-ahead of one grid of tiles)
    if (d->P * widest >= (1ll << 31) - (1ll << 26)) return M2D_ERR_TOO_LARGE;
    return M2D_OK;
}

static ProjPlan plan_proj(const m2d_proj_desc* d) {
    ProjPlan p;
    const int sms = sm_count();
    p.EB = (d->E + 31) / 32 * 32;
    p.PS = p.EB >= 256 ? 1 : 256 / p.EB;
    p.threads = p.EB * p.PS;
    p.TP = kProjIters * p.PS;
    p.RB = d->R <= 4 ? 4 : d->R <= 8 ? 8 : d->R <= 16 ? 16 : d->R <= 32 ? 32 : 64;
    p.ntiles = (int)((d->P + p.TP - 1) / p.TP);
    p.gx = p.ntiles < 2 * sms ? p.ntiles : 2 * sms;
    p.dt_partials = align256((size_t)2 * p.gx * (p.RB + 1) * p.EB * sizeof(float));
    p.K = 2 * d->R + 3 * d->N;
    p.tilesK = (p.K + 63) / 64;
    p.tilesE = (d->E + 63) / 64;
    const int tiles = p.tilesK * p.tilesE;
    long long slabs = (4ll * sms + tiles - 1) / tiles;
    const long long max_slabs = (d->P + 63) / 64;
    if (slabs > max_slabs) slabs = max_slabs;
    if (slabs < 1) slabs = 1;
    p.rows_per_slab = (int)(((d->P + slabs - 1) / slabs + 31) / 32 * 32);
    p.slabs = (int)((d->P + p.rows_per_slab - 1) / p.rows_per_slab);
    p.wg_partials = align256((size_t)p.slabs * p.K * d->E * sizeof(float));
    return p;
}

// ------------------------------------------------------------------------------------------------
// delta = softplus(r @ W^T + b).  grid (ctas, 2 directions); block = EB channels x PS pixels.
// ------------------------------------------------------------------------------------------------
template <typename io_t, int RB, int MAXT>
__global__ void __launch_bounds__(MAXT) dtproj_fwd_kernel(const ProjArgs a) {
    extern __shared__ float sm[];                  // rs[TP][RB]: this tile's rank-R rows, zero padded
    const int dir = blockIdx.y;
    const int te = threadIdx.x % a.EB, ps = threadIdx.x / a.EB;
    const bool e_ok = te < a.E;
    const void* W = dir ? a.WL : a.WT;
    const void* bias = dir ? a.bL : a.bT;
    const io_t* proj = static_cast<const io_t*>(a.proj);
    io_t* out = static_cast<io_t*>(dir ? a.dL : a.dT);
    const int col0 = dir * a.R;
    a.clear.run();

    float w[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) w[r] = (e_ok && r < a.R) ? load_param<io_t>(W, te * a.R + r, a.params_f32) : 0.f;
    const float b = e_ok ? load_param<io_t>(bias, te, a.params_f32) : 0.f;

    // The rank-R rows of the next tile are fetched into registers while this tile is computed
    // (TP*RB <= 2*blockDim is guaranteed by the host: two values per thread at most).
    const int tile_elems = a.TP * RB;
    auto fetch_rows = [&](int tile, float (&v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int idx = threadIdx.x + h * blockDim.x;
            const int pp = idx / RB, r = idx % RB;
            const int p = tile * a.TP + pp;
            v[h] = (idx < tile_elems && r < a.R && p < a.P && tile < a.ntiles) ? load1(proj, p * a.pitch + col0 + r) : 0.f;
        }
    };
    float nxt[2];
    fetch_rows(blockIdx.x, nxt);
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
        const int p0 = tile * a.TP;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int idx = threadIdx.x + h * blockDim.x;
            if (idx < tile_elems) sm[idx] = nxt[h];
        }
        __syncthreads();
        fetch_rows(tile + gridDim.x, nxt);
        io_t* dst = out + (p0 + ps) * a.E + te;
        const int row_step = a.PS * a.E;
#pragma unroll
        for (int k = 0; k < kProjIters; ++k) {
            const int pp = k * a.PS + ps;
            const float4* rr = reinterpret_cast<const float4*>(sm + pp * RB);
            float z = b;
#pragma unroll
            for (int r4 = 0; r4 < RB / 4; ++r4) {
                const float4 v = rr[r4];
                z = fmaf(v.x, w[4 * r4], z);
                z = fmaf(v.y, w[4 * r4 + 1], z);
                z = fmaf(v.z, w[4 * r4 + 2], z);
                z = fmaf(v.w, w[4 * r4 + 3], z);
            }
            if (e_ok && p0 + pp < a.P) store1(dst, k * row_step, softplus_f(z));
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// Backward of the dt projections.  A thread owns channel te of the pixels k*PS + ps (k = 0..7) of
// each tile: it forms s = g * softplus', keeps d_b and its row of d_W in registers, and parks s in a
// per-warp [8 pixels][32 channels] slab of shared memory.  The warp then re-reads the slab with the
// roles turned round -- a lane owns rank r (and a subset of the 8 pixels), holds W[e][r] of the
// warp's 32 channels in registers and sums over them -- which yields the warp's share of
// d_r = s @ W without any shuffle; the shares of the CTA's warps meet in shared memory: by adds, or from 32
// ranks on, where 12 to 20 warps would meet in each, as a copy per warp (P = 784, E = 384: 20.7 -> 17.4 us,
// P = 6272, E = 512: 57 -> 54; but 131 -> 150 at P = 401408, E = 64, where two warps meet).
// Shared memory: rs[TP][RB], drs[1 or EB/32][TP][RB], slab[warps][8][36] and two buffers of the tile's g and
// delta rows; the end-of-kernel reduction accS[RB+1][EB] reuses the same bytes.
// ------------------------------------------------------------------------------------------------
template <int RB> constexpr bool kShares = RB >= 32;
constexpr int kSlabStride = 36;        // 32 channels + 4: rows of a slab start in different banks
__device__ __forceinline__ float smem_value(const float* p) { return *p; }
__device__ __forceinline__ float smem_value(const __nv_bfloat16* p) { return bf16_bits_to_float(*reinterpret_cast<const unsigned short*>(p)); }

template <typename io_t, int RB, int MAXT>
__global__ void __launch_bounds__(MAXT) dtproj_bwd_kernel(const ProjArgs a) {
    extern __shared__ float sm[];
    float* accS = sm;                              // used after the tile loop only: overlays everything else
    float* rs = sm;
    const int slices = kShares<RB> ? a.EB >> 5 : 1;          // copies of drs
    float* drs = rs + a.TP * RB;
    float* slab = drs + slices * a.TP * RB + (threadIdx.x >> 5) * (kProjIters * kSlabStride);
    io_t* tiles = reinterpret_cast<io_t*>(drs + slices * a.TP * RB + (blockDim.x >> 5) * (kProjIters * kSlabStride));   // [2 buffers][g | delta][TP*E]
    const int dir = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int te = threadIdx.x % a.EB, ps = threadIdx.x / a.EB;
    const bool e_ok = te < a.E;
    const void* W = dir ? a.WL : a.WT;
    const io_t* proj = static_cast<const io_t*>(a.proj);
    const io_t* delta = static_cast<const io_t*>(dir ? a.dL : a.dT);
    const io_t* g = static_cast<const io_t*>(dir ? a.g_dL : a.g_dT);
    io_t* d_proj = static_cast<io_t*>(a.d_proj);
    const int col0 = dir * a.R;

    // roles of the second phase: lane = (pl, rl): ranks rl + 32*h, pixels pl + PL*kk of the warp's 8
    constexpr int RL = RB > 32 ? 32 : RB;          // ranks handled side by side
    constexpr int PL = 32 / RL;                    // pixels handled side by side
    constexpr int KPL = kProjIters / PL;           // pixels per lane
    constexpr int NH = RB / RL;                    // rank halves per lane
    const int rl = lane % RL, pl = lane / RL;
    const int e_slice = te - lane;                 // first channel of this warp
    float wreg[NH][32];
#pragma unroll
    for (int h = 0; h < NH; ++h)
#pragma unroll
        for (int e = 0; e < 32; ++e) {
            const int r = h * RL + rl, ch = e_slice + e;
            wreg[h][e] = (ch < a.E && r < a.R) ? load_param<io_t>(W, ch * a.R + r, a.params_f32) : 0.f;
        }

    float acc[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) acc[r] = 0.f;
    float accb = 0.f;

    const int tile_elems = a.TP * RB;
    auto fetch_rows = [&](int tile, float (&v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int idx = threadIdx.x + h * blockDim.x;
            const int pp = idx / RB, r = idx % RB;
            const int p = tile * a.TP + pp;
            v[h] = (idx < tile_elems && r < a.R && p < a.P && tile < a.ntiles) ? load1(proj, p * a.pitch + col0 + r) : 0.f;
        }
    };
    // The tile's g and delta rows (TP consecutive pixels = one contiguous chunk of each tensor) are
    // copied to shared memory with cp.async, one tile ahead, in pieces of 4 elements.
    const int tile_chunk = a.TP * a.E;                       // elements per tensor per tile
    auto issue_inputs = [&](int tile, int buf) {
        io_t* dst_g = tiles + (size_t)(buf * 2) * tile_chunk;
        io_t* dst_d = dst_g + tile_chunk;
        const int base = tile * a.TP * a.E;
        // 16-byte pieces (4 fp32 or 8 bf16 elements, L2-only copies) where rows allow it and both
        // tensors are 16-byte aligned; 8-byte pieces for bf16 rows that are only a multiple of 4
        const bool wide = sizeof(io_t) == 4 || a.wide16;
        const int pe = wide ? 16 / (int)sizeof(io_t) : 4;
        for (int piece = threadIdx.x; piece * pe < tile_chunk; piece += blockDim.x) {
            const int off = piece * pe;
            const bool ok = tile < a.ntiles && tile * a.TP + off / a.E < a.P;
            if (wide) {
                cp_async16_if(ok, smem_u32(dst_g + off), g + base + off);
                cp_async16_if(ok, smem_u32(dst_d + off), delta + base + off);
                if (!ok) {
                    *reinterpret_cast<float4*>(dst_g + off) = make_float4(0.f, 0.f, 0.f, 0.f);
                    *reinterpret_cast<float4*>(dst_d + off) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            } else {
                cp_async8_if(ok, smem_u32(dst_g + off), g + base + off);
                cp_async8_if(ok, smem_u32(dst_d + off), delta + base + off);
                if (!ok) {
                    *reinterpret_cast<uint2*>(dst_g + off) = make_uint2(0u, 0u);
                    *reinterpret_cast<uint2*>(dst_d + off) = make_uint2(0u, 0u);
                }
            }
        }
    };
    float nxt[2];
    fetch_rows(blockIdx.x, nxt);
    issue_inputs(blockIdx.x, 0);
    int buf = 0;
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, buf ^= 1) {
        const int p0 = tile * a.TP;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int idx = threadIdx.x + h * blockDim.x;
            if (idx < tile_elems) {
                rs[idx] = nxt[h];
                if (!kShares<RB>) drs[idx] = 0.f;
            }
        }
        cp_async_wait_all();
        __syncthreads();
        fetch_rows(tile + gridDim.x, nxt);
        issue_inputs(tile + gridDim.x, buf ^ 1);      // next tile's copies fly while this one is reduced
        const io_t* cur_g = tiles + (size_t)(buf * 2) * tile_chunk + ps * a.E + te;
        const io_t* cur_d = cur_g + tile_chunk;
        float sv[kProjIters];
#pragma unroll
        for (int k = 0; k < kProjIters; ++k) {
            const float gk = e_ok ? smem_value(cur_g + k * a.PS * a.E) : 0.f;
            const float d = e_ok ? smem_value(cur_d + k * a.PS * a.E) : 0.f;
            // softplus'(z) = sigmoid(z) = 1 - exp(-softplus(z)); a short series where 1 - exp cancels
            const float series = d * (1.f - d * (0.5f - d * (1.f / 6.f - d * (1.f / 24.f - d * (1.f / 120.f)))));
            sv[k] = gk * (d < 0.1f ? series : 1.f - __expf(-d));
            slab[k * kSlabStride + lane] = sv[k];
            accb += sv[k];
        }
        __syncwarp();
        // d_W row of this channel: acc[r] += s * r_row[r]
#pragma unroll
        for (int k = 0; k < kProjIters; ++k) {
            const float4* rr = reinterpret_cast<const float4*>(rs + (k * a.PS + ps) * RB);
#pragma unroll
            for (int r4 = 0; r4 < RB / 4; ++r4) {
                const float4 q = rr[r4];
                acc[4 * r4] = fmaf(sv[k], q.x, acc[4 * r4]);
                acc[4 * r4 + 1] = fmaf(sv[k], q.y, acc[4 * r4 + 1]);
                acc[4 * r4 + 2] = fmaf(sv[k], q.z, acc[4 * r4 + 2]);
                acc[4 * r4 + 3] = fmaf(sv[k], q.w, acc[4 * r4 + 3]);
            }
        }
        // d_r of the warp's pixels over the warp's 32 channels
#pragma unroll
        for (int kk = 0; kk < KPL; ++kk) {
            const int k = pl + kk * PL;
            const float4* row = reinterpret_cast<const float4*>(slab + k * kSlabStride);
            float sum[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) sum[h] = 0.f;
#pragma unroll
            for (int e4 = 0; e4 < 8; ++e4) {
                const float4 q = row[e4];
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    sum[h] = fmaf(q.x, wreg[h][4 * e4], sum[h]);
                    sum[h] = fmaf(q.y, wreg[h][4 * e4 + 1], sum[h]);
                    sum[h] = fmaf(q.z, wreg[h][4 * e4 + 2], sum[h]);
                    sum[h] = fmaf(q.w, wreg[h][4 * e4 + 3], sum[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const int at = (k * a.PS + ps) * RB + h * RL + rl;
                if (kShares<RB>) drs[(e_slice >> 5) * tile_elems + at] = sum[h];
                else atomicAdd(&drs[at], sum[h]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int idx = threadIdx.x + h * blockDim.x;
            const int pp = idx / RB, r = idx % RB;
            if (idx < tile_elems && r < a.R && p0 + pp < a.P) {
                float sum = 0.f;
                for (int k = 0; k < slices; ++k) sum += drs[k * tile_elems + idx];
                store1(d_proj, (p0 + pp) * a.pitch + col0 + r, sum);
            }
        }
        __syncthreads();
    }

    // one partial per CTA: the sum over the PS pixel rows of the block, a row at a time
    float* part = a.partials + ((size_t)dir * gridDim.x + blockIdx.x) * (RB + 1) * a.EB;
    if (a.PS == 1) {
#pragma unroll
        for (int r = 0; r < RB; ++r) part[r * a.EB + te] = acc[r];
        part[RB * a.EB + te] = accb;
        return;
    }
    cp_async_wait_all();
    for (int row = 0; row < a.PS; ++row) {
        __syncthreads();
        if (ps == row) {
#pragma unroll
            for (int r = 0; r < RB; ++r) accS[r * a.EB + te] = row ? accS[r * a.EB + te] + acc[r] : acc[r];
            accS[RB * a.EB + te] = row ? accS[RB * a.EB + te] + accb : accb;
        }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < (RB + 1) * a.EB; idx += blockDim.x) part[idx] = accS[idx];
}

// ------------------------------------------------------------------------------------------------
// d_Wx[k][e] = sum_p d_proj[p][k] * x[p][e].  grid (slabs, tilesE, tilesK); a CTA of 256 threads
// computes a 64x64 tile of the result over its slab of pixels, 32 pixels per shared-memory stage,
// each thread a 4x4 block.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float4 load4g(const __nv_bfloat16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                       __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}

__global__ void __launch_bounds__(256) xproj_wgrad_kernel(const WgArgs a) {      // bf16
    typedef __nv_bfloat16 io_t;
    __shared__ float4 As[2][32][16];
    __shared__ float4 Bs[2][32][16];
    const io_t* A = static_cast<const io_t*>(a.d_proj);
    const io_t* B = static_cast<const io_t*>(a.x);
    const int tid = threadIdx.x, te = tid & 15, tk = tid >> 4;
    const int e0 = blockIdx.y * 64, k0 = blockIdx.z * 64;
    const int row0 = blockIdx.x * a.rows_per_slab;
    int row_end = row0 + a.rows_per_slab;
    if (row_end > a.P) row_end = a.P;
    const int chunks = (int)((row_end - row0 + 31) / 32);

    // each thread stages two float4 of A and two of B per chunk: rows lr and lr + 16, column quad lc
    const int lr = tid >> 4, lc = tid & 15;
    auto fetch = [&](int chunk, float4 (&ra)[2], float4 (&rb)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = row0 + chunk * 32 + lr + 16 * h;
            const bool row_ok = p < row_end;
            const int ka = k0 + lc * 4, eb = e0 + lc * 4;
            ra[h] = make_float4(0.f, 0.f, 0.f, 0.f);
            rb[h] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row_ok && ka + 4 <= a.K) {
                ra[h] = load4g(A + p * a.pitch + ka);
            } else if (row_ok && ka < a.K) {       // ragged last quad of the K columns
                float t[4] = {0.f, 0.f, 0.f, 0.f};
                for (int i = 0; i < 4 && ka + i < a.K; ++i) t[i] = load1(A, p * a.pitch + ka + i);
                ra[h] = make_float4(t[0], t[1], t[2], t[3]);
            }
            if (row_ok && eb < a.E) rb[h] = load4g(B + p * a.E + eb);
        }
    };

    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    float4 ra[2], rb[2];
    if (chunks > 0) {
        fetch(0, ra, rb);
        As[0][lr][lc] = ra[0]; As[0][lr + 16][lc] = ra[1];
        Bs[0][lr][lc] = rb[0]; Bs[0][lr + 16][lc] = rb[1];
    }
    __syncthreads();
    for (int c = 0; c < chunks; ++c) {
        const int buf = c & 1;
        const bool more = c + 1 < chunks;
        if (more) fetch(c + 1, ra, rb);
#pragma unroll 8
        for (int p = 0; p < 32; ++p) {
            const float4 av = As[buf][p][tk], bv = Bs[buf][p][te];
            const float aa[4] = {av.x, av.y, av.z, av.w}, bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(aa[i], bb[j], acc[i][j]);
        }
        if (more) {
            As[buf ^ 1][lr][lc] = ra[0]; As[buf ^ 1][lr + 16][lc] = ra[1];
            Bs[buf ^ 1][lr][lc] = rb[0]; Bs[buf ^ 1][lr + 16][lc] = rb[1];
        }
        __syncthreads();
    }
    float* part = a.partials + (size_t)blockIdx.x * a.K * a.E;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = k0 + tk * 4 + i, e = e0 + te * 4;
        if (k < a.K && e < a.E)
            *reinterpret_cast<float4*>(part + (size_t)k * a.E + e) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// The same for fp32: a CTA of 128 threads, the even pixels of a stage for the first two warps, the odd ones for the
// others, each thread an 8x8 block, the stages filled by asynchronous copies.  Bound by the loads from shared memory at a 4x4
// block (two for 16 multiply-adds, that pipe 83 % busy, 93 us at P = 401408, E = 64); with four for 64, and no registers
// for the next stage, 72 us (27 -> 22.6 at 6272 x 512).  (On the CUDA cores: TF32 would not hold the tolerance.)
constexpr int kWgThreads = 128;

__global__ void __launch_bounds__(kWgThreads, 4) xproj_wgrad_f32_kernel(const WgArgs a) {
    __shared__ float4 tiles[2][2][32][16];         // [d_proj, x][buffer][pixel][quad]
    const float* A = static_cast<const float*>(a.d_proj);
    const float* B = static_cast<const float*>(a.x);
    const int tid = threadIdx.x, half = tid >> 6, te = tid >> 2 & 7, tk = (tid & 3) + (tid >> 5 & 1) * 4;
    const int e0 = blockIdx.y * 64, k0 = blockIdx.z * 64;
    const int row0 = blockIdx.x * a.rows_per_slab, row_end = min(row0 + a.rows_per_slab, a.P);
    const int chunks = (row_end - row0 + 31) / 32;

    // each thread copies four quads of either per stage: rows lr, lr + 8, ..., column quad lc; zeros beyond the last row and column
    const int lr = tid >> 4, lc = tid & 15, ka = k0 + lc * 4, eb = e0 + lc * 4;
    const int a_bytes = 4 * max(0, min(4, a.K - ka)), b_bytes = eb < a.E ? 16 : 0;
    const float* ap = A + (long long)(row0 + lr) * a.pitch + ka;
    const float* bp = B + (long long)(row0 + lr) * a.E + eb;
    const unsigned dst = smem_u32(&tiles[0][0][lr][lc]);
    auto fetch = [&](int chunk) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const bool on = row0 + chunk * 32 + lr + 8 * h < row_end;
            const unsigned d = dst + (chunk & 1) * 8192 + h * 2048;
            const float* const as = on && a_bytes ? ap + (long long)h * 8 * a.pitch : A;
            const float* const bs = on && b_bytes ? bp + (long long)h * 8 * a.E : B;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(as), "r"(on ? a_bytes : 0) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + 16384), "l"(bs), "r"(on ? b_bytes : 0) : "memory");
        }
        ap += (long long)32 * a.pitch;
        bp += (long long)32 * a.E;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    fetch(0);
    for (int c = 0; c < chunks; ++c) {
        cp_async_wait_all();
        __syncthreads();                           // the stage is there, and the other buffer is free
        if (c + 1 < chunks) fetch(c + 1);
        const float4 (&As)[32][16] = tiles[0][c & 1];
        const float4 (&Bs)[32][16] = tiles[1][c & 1];
#pragma unroll 2
        for (int p = half; p < 32; p += 2) {
            const float4 a0 = As[p][tk], a1 = As[p][tk + 8], b0 = Bs[p][te], b1 = Bs[p][te + 8];
            const float aa[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(aa[i], bb[j], acc[i][j]);
        }
    }
    // the odd pixels' share joins the even ones'
    cp_async_wait_all();
    __syncthreads();
    float4* const meet = &tiles[0][0][0][0] + (tid & 63);
    if (half) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) meet[(i * 2 + j) * 64] = make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
    }
    __syncthreads();
    if (half) return;
    float* part = a.partials + (size_t)blockIdx.x * a.K * a.E;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int k = k0 + tk * 4 + (i & 3) + (i >> 2) * 32, e = e0 + te * 4 + j * 32;
            const float4 o = meet[(i * 2 + j) * 64];
            if (k < a.K && e < a.E)
                *reinterpret_cast<float4*>(part + (size_t)k * a.E + e) =
                    make_float4(acc[i][4 * j] + o.x, acc[i][4 * j + 1] + o.y, acc[i][4 * j + 2] + o.z, acc[i][4 * j + 3] + o.w);
        }
}

// ------------------------------------------------------------------------------------------------
// The parameters' gradients from the partial results, d_W[e][r] (r < R), d_b[e] (r == RB) and d_Wx: block (32, ROWS), 32
// neighbouring results, the partial results dealt round-robin to the rows of the block.  One launch for the
// sums of both kernels (a launch costs a small call as much as the sums).  Bound by the latency of its loads where the
// results are few and the partial results many (571 of them at P = 401408, E = 64: eight rows make a thread add 70,
// 19 us for 5 MB; 32 rows 6.4), by the number of its warps where the results are many.
// ------------------------------------------------------------------------------------------------
struct DtSums {
    const float* partials;             // [dir][cta][RB+1][EB]
    int ctas, RB, EB, E, R;
    void *d_WT, *d_WL, *d_bT, *d_bL;
    __host__ __device__ int blocks() const { return partials ? (2 * (RB + 1) * EB + 31) / 32 : 0; }
};
struct WgSums {
    const float* partials;             // [slab][K*E]
    int slabs;
    long long ke;
    void* d_Wx;
    __host__ __device__ int blocks() const { return partials ? (int)((ke + 31) / 32) : 0; }
};

template <typename g_t, int ROWS>      // type of the parameters' gradients
__global__ void __launch_bounds__(32 * ROWS) proj_bwd_finalize(const DtSums dt, const WgSums wg) {
    __shared__ float red[ROWS][33];
    const bool is_dt = (int)blockIdx.x < dt.blocks();
    const long long idx = (long long)(is_dt ? blockIdx.x : blockIdx.x - dt.blocks()) * 32 + threadIdx.x;
    const long long step = is_dt ? (dt.RB + 1) * dt.EB : wg.ke, n = is_dt ? 2 * step : wg.ke;
    const int count = is_dt ? dt.ctas : wg.slabs;
    const int dir = is_dt && idx >= step ? 1 : 0, rem = (int)(idx - dir * step);
    float s = 0.f;
    if (idx < n) {
        const float* src = (is_dt ? dt.partials + dir * count * step : wg.partials) + rem;
#pragma unroll 8
        for (int c = threadIdx.y; c < count; c += ROWS) s += src[c * step];
    }
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0 || idx >= n) return;
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < ROWS; ++y) t += red[y][threadIdx.x];
    if (!is_dt) {
        store1(static_cast<g_t*>(wg.d_Wx), idx, t);
        return;
    }
    const int r = rem / dt.EB, e = rem % dt.EB;
    if (e >= dt.E) return;
    if (r == dt.RB) store1(static_cast<g_t*>(dir ? dt.d_bL : dt.d_bT), e, t);
    else if (r < dt.R) store1(static_cast<g_t*>(dir ? dt.d_WL : dt.d_WT), (long long)e * dt.R + r, t);
}

// ------------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------------
static Clear clear_of(const m2d_proj_desc* d) { return Clear{static_cast<uint4*>(d->clear), d->clear ? (long long)(d->clear_bytes / 16) : 0}; }

static ProjArgs proj_args(const m2d_proj_desc* d, const ProjPlan& p) {
    ProjArgs a;
    a.P = (int)d->P; a.pitch = (int)d->proj_pitch; a.ntiles = p.ntiles;
    a.E = d->E; a.R = d->R; a.EB = p.EB; a.PS = p.PS; a.TP = p.TP;
    a.proj = d->proj; a.WT = d->WT; a.WL = d->WL; a.bT = d->bT; a.bL = d->bL;
    a.dT = d->dT; a.dL = d->dL; a.g_dT = d->g_dT; a.g_dL = d->g_dL;
    a.d_proj = d->d_proj;
    a.params_f32 = (d->flags & M2D_PROJ_PARAMS_F32) ? 1 : 0;
    a.clear = clear_of(d);
    a.partials = static_cast<float*>(d->workspace);
    a.wide16 = d->E % 8 == 0 && aligned(d->g_dT, 16) && aligned(d->g_dL, 16) && aligned(d->dT, 16) && aligned(d->dL, 16);
    return a;
}

// CTAs per direction: the grid (gx, 2 directions) fills the resident CTA slots of the device exactly
// once, so that every SM gets the same number of CTAs and every CTA the same number of tiles (with the
// planned 2 x SMs per direction some SMs held five CTAs and others three: a quarter of the kernel was
// spent waiting for the fuller ones).  Never more than the plan's gx, which sized the workspace.
template <typename K>
static int balanced_gx(K kern, const ProjPlan& p, size_t smem) {
    const int per_sm = resident_ctas(reinterpret_cast<const void*>(kern), p.threads, smem);
    if (per_sm < 1) return p.gx;
    const int gx = per_sm * sm_count() / 2;
    return gx < 1 ? 1 : (gx < p.gx ? gx : p.gx);
}

template <typename io_t, int RB>
static int launch_dt_fwd(const ProjArgs& a, const ProjPlan& p, cudaStream_t st) {
    const size_t smem = (size_t)p.TP * RB * sizeof(float);
    auto kern = p.threads <= 256   ? dtproj_fwd_kernel<io_t, RB, 256>
                : p.threads <= 384 ? dtproj_fwd_kernel<io_t, RB, 384>
                : p.threads <= 512 ? dtproj_fwd_kernel<io_t, RB, 512>
                                   : dtproj_fwd_kernel<io_t, RB, M2D_PROJ_MAX_E>;
    kern<<<dim3(balanced_gx(kern, p, smem), 2), p.threads, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? M2D_OK : M2D_ERR_LAUNCH;
}

template <typename io_t>
static int launch_sums(const m2d_proj_desc* d, const DtSums& dt, const WgSums& wg, cudaStream_t st) {
    const int blocks = dt.blocks() + wg.blocks();
    // 32 rows while a block per SM is not enough to keep its loads in flight.  8 / 32 rows, us: 132 blocks 19 / 6.4
    // (P = 401408, E = 64), 328 blocks 9 / 6 (100352, 128); 1540 blocks 12 / 14 (25088, 320), 2848 blocks 8 / 19 (6272, 512).
    const bool few = blocks < 4 * sm_count();
    auto launch = [&](auto rows) {
        constexpr int ROWS = decltype(rows)::value;
        if (d->flags & M2D_PROJ_PARAMS_F32) proj_bwd_finalize<float, ROWS><<<blocks, dim3(32, ROWS), 0, st>>>(dt, wg);
        else proj_bwd_finalize<io_t, ROWS><<<blocks, dim3(32, ROWS), 0, st>>>(dt, wg);
    };
    if (few) launch(std::integral_constant<int, 32>{});
    else launch(std::integral_constant<int, 8>{});
    return cudaGetLastError() == cudaSuccess ? M2D_OK : M2D_ERR_LAUNCH;
}
static DtSums dt_sums(const m2d_proj_desc* d, const ProjPlan& p, int ctas) {
    return DtSums{static_cast<const float*>(d->workspace), ctas, p.RB, p.EB, d->E, d->R, d->d_WT, d->d_WL, d->d_bT, d->d_bL};
}

template <typename io_t, int RB>
static int launch_dt_bwd(const m2d_proj_desc* d, const ProjArgs& a, const ProjPlan& p, DtSums* sums, cudaStream_t st) {
    const size_t loop_bytes = ((size_t)(1 + (kShares<RB> ? p.EB / 32 : 1)) * p.TP * RB + (size_t)(p.threads / 32) * kProjIters * kSlabStride) * sizeof(float) +
                              (size_t)4 * p.TP * d->E * sizeof(io_t);
    const size_t tail_bytes = (size_t)(RB + 1) * p.EB * sizeof(float);
    const size_t smem = loop_bytes > tail_bytes ? loop_bytes : tail_bytes;
    // the launch bound follows the block size, so that small blocks keep their registers
    auto kern = p.threads <= 256   ? dtproj_bwd_kernel<io_t, RB, 256>
                : p.threads <= 384 ? dtproj_bwd_kernel<io_t, RB, 384>
                : p.threads <= 512 ? dtproj_bwd_kernel<io_t, RB, 512>
                                   : dtproj_bwd_kernel<io_t, RB, M2D_PROJ_MAX_E>;
    if (!allow_smem(reinterpret_cast<const void*>(kern), smem)) return M2D_ERR_LAUNCH;
    const int gx = balanced_gx(kern, p, smem);
    kern<<<dim3(gx, 2), p.threads, smem, st>>>(a);
    if (cudaGetLastError() != cudaSuccess) return M2D_ERR_LAUNCH;
    *sums = dt_sums(d, p, gx);
    return M2D_OK;
}

// Which kernels a call gets.  The tensor-core ones read and write rows of 16-byte pieces (E a multiple of 8,
// aligned tensors), and the backward's sums fit its registers up to 39 ranks.  Measured, CUDA cores / tensor cores in
// us (R = E / 16; CUDA events around one call with the L2 flushed, which adds about 5 to a kernel's own time):
//   forward, bf16: 92 / 56 (P = 401408, E = 64), 68 / 38 (25088, 320), 13 / 11 (784, 384): tensor cores always.
//   forward, fp32 (a product is six), by elements P * E:
//                E = 64      128       192       320       384       512       576
//       2 M     14 / 16   16 / 16   18 / 23   25 / 26   25 / 33   40 / 29   35 / 43
//       3.25 M  18 / 18   21 / 20   23 / 24   32 / 35   33 / 33   47 / 47   49 / 43
//       4 M     21 / 21   24 / 25   27 / 31   37 / 35   37 / 45   51 / 47   57 / 54
//       7 M     31 / 27   35 / 29   41 / 41   57 / 49   57 / 45   70 / 57   93 / 66
//     The line is at 3 M.  (The tensor-core times are steps: its CTAs take whole tiles of 128 pixels.)
//   backward, bf16:
//       P       E = 64      128       320       384       512
//       784     16 / 15   20 / 21   30 / 35   32 / 46   34 / 53
//       3136    19 / 15   26 / 22   44 / 38   47 / 48   50 / 54
//       4736    22 / 16   28 / 22   53 / 41   55 / 52   58 / 58
//       6272    23 / 17   29 / 24   62 / 44   66 / 69   70 / 74
//       12544   26 / 18   34 / 28  104 / 65  107 / 89  113 / 90
//     The line is where its tiles of 64 pixels, in two directions, give every SM one (P = 4736 on 148 SMs); below
//     it the wider stages lose.
//   backward, fp32: the tensor cores lose everywhere (131 / 149 at P = 401408, E = 64).
// The six products of an fp32 call need six times the rank in shared memory: from 49 ranks on 256 channels a CTA do
// not fit (R = 64: 298 KB), and the CUDA cores keep those calls.  (128 channels would fit; at P = 25088, R = 64 they
// take 99 us against 91 with E = 256, 193 against 201 with E = 640.)
static int mma_fwd_chunk(int E) {      // channels per CTA at most: up to 256, the chunks of a wider call alike
    const int n = (E + 255) / 256;
    return ((E + n - 1) / n + 31) / 32 * 32;
}
template <typename io_t> static bool mma_fwd_fits(const m2d_proj_desc* d) { return mma_fwd_smem(mma_fwd_chunk(d->E), mma_k<io_t>(d->R)) <= kMaxSmem; }
static bool mma_fwd_ok(const m2d_proj_desc* d) {
    if (d->E % 8 != 0 || !aligned(d->dT, 16) || !aligned(d->dL, 16)) return false;
    return d->dtype == M2D_BF16 ? mma_fwd_fits<__nv_bfloat16>(d) : d->P * d->E >= 3000000 && mma_fwd_fits<float>(d);
}
static bool mma_bwd_ok(const m2d_proj_desc* d) {
    return d->dtype == M2D_BF16 && d->E % 8 == 0 && d->R < 40 && d->P >= 32 * sm_count() && aligned(d->dT, 16) && aligned(d->dL, 16) &&
           aligned(d->g_dT, 16) && aligned(d->g_dL, 16);
}

template <typename io_t>
static int launch_mma_fwd(const m2d_proj_desc* d, cudaStream_t st) {
    MmaFwdArgs a;
    a.P = (int)d->P; a.pitch = (int)d->proj_pitch; a.E = d->E; a.R = d->R; a.nk = mma_k<io_t>(d->R);
    a.params_f32 = (d->flags & M2D_PROJ_PARAMS_F32) ? 1 : 0;
    a.proj = d->proj; a.WT = d->WT; a.WL = d->WL; a.bT = d->bT; a.bL = d->bL; a.dT = d->dT; a.dL = d->dL;
    // up to 256 channels per CTA (the tile of r is split and read once per chunk of channels); fewer while the
    // pixels alone do not give every SM a CTA.  Chunks of one size: with 256 + 64 channels at E = 320 half the CTAs had
    // a quarter of the work (fp32, us, before / now: P = 9375, 36 / 27; 21875, 57 / 49; 50000, 100 / 77; E = 384, P = 41666,
    // 94 / 82; E = 576, P = 6944, 65 / 54; bf16 E = 320, P = 12544, 25 / 22)
    const long long tiles = (d->P + 127) / 128;
    int chunk = mma_fwd_chunk(d->E);
    while (chunk > 32 && tiles * 2 * ((d->E + chunk - 1) / chunk) < sm_count()) chunk = (chunk / 2 + 31) / 32 * 32;
    a.chunk = chunk;
    const size_t smem = mma_fwd_smem(chunk, a.nk);
    auto kern = dtproj_fwd_mma_kernel<io_t>;
    if (!allow_smem(reinterpret_cast<const void*>(kern), smem)) return M2D_ERR_LAUNCH;
    a.clear = clear_of(d);
    const int chunks = (d->E + chunk - 1) / chunk, per_sm = resident_ctas(reinterpret_cast<const void*>(kern), 256, smem);
    long long gx = (long long)(per_sm > 0 ? per_sm : 1) * sm_count() / (2 * chunks);
    if (gx > tiles) gx = tiles;
    kern<<<dim3((unsigned)(gx < 1 ? 1 : gx), 2, chunks), 256, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? M2D_OK : M2D_ERR_LAUNCH;
}

template <int CH, int NCH, int NT>
static int launch_mma_bwd(const m2d_proj_desc* d, const ProjPlan& p, DtSums* sums, cudaStream_t st) {
    MmaBwdArgs a;
    a.P = (int)d->P; a.pitch = (int)d->proj_pitch; a.E = d->E; a.R = d->R; a.RB = p.RB; a.EB = p.EB;
    a.params_f32 = (d->flags & M2D_PROJ_PARAMS_F32) ? 1 : 0;
    a.proj = d->proj; a.WT = d->WT; a.WL = d->WL; a.dT = d->dT; a.dL = d->dL; a.g_dT = d->g_dT; a.g_dL = d->g_dL;
    a.d_proj = d->d_proj;
    a.partials = static_cast<float*>(d->workspace);
    const size_t smem = mma_bwd_smem<CH>(NCH, NT);
    auto kern = dtproj_bwd_mma_kernel<CH, NCH, NT>;
    if (!allow_smem(reinterpret_cast<const void*>(kern), smem)) return M2D_ERR_LAUNCH;
    const int per_sm = resident_ctas(reinterpret_cast<const void*>(kern), 256, smem);
    long long gx = (long long)(per_sm > 0 ? per_sm : 1) * sm_count() / 2;
    const long long tiles = (d->P + MmaTile<CH>::kPix - 1) / MmaTile<CH>::kPix;
    if (gx > tiles) gx = tiles;
    if (gx > p.gx) gx = p.gx;                      // the workspace holds that many partial results
    if (gx < 1) gx = 1;
    kern<<<dim3((unsigned)gx, 2), 256, smem, st>>>(a);
    if (cudaGetLastError() != cudaSuccess) return M2D_ERR_LAUNCH;
    *sums = dt_sums(d, p, (int)gx);
    return M2D_OK;
}

template <typename io_t>
static int dispatch_dt_fwd(const m2d_proj_desc* d, cudaStream_t st) {
    if (mma_fwd_ok(d)) return launch_mma_fwd<io_t>(d, st);
    const ProjPlan p = plan_proj(d);
    const ProjArgs a = proj_args(d, p);
    switch (p.RB) {
        case 4: return launch_dt_fwd<io_t, 4>(a, p, st);
        case 8: return launch_dt_fwd<io_t, 8>(a, p, st);
        case 16: return launch_dt_fwd<io_t, 16>(a, p, st);
        case 32: return launch_dt_fwd<io_t, 32>(a, p, st);
        default: return launch_dt_fwd<io_t, 64>(a, p, st);
    }
}

template <typename io_t>
static int dispatch_dt_bwd(const m2d_proj_desc* d, const ProjPlan& p, DtSums* sums, cudaStream_t st) {
    if constexpr (sizeof(io_t) == 2) if (mma_bwd_ok(d)) {
        // register blocks (chunks of channels, rank tiles) that cover the shipped widths (R = E / 16) closely and
        // everything else with some padding
        const int nch = (d->E + 127) / 128, nt = (d->R + 8) / 8;
        if (d->E <= 64 && nt <= 1) return launch_mma_bwd<64, 1, 1>(d, p, sums, st);
        if (d->E <= 192 && nt <= 2) return launch_mma_bwd<64, 3, 2>(d, p, sums, st);
        if (nch <= 3 && nt <= 3) return launch_mma_bwd<128, 3, 3>(d, p, sums, st);
        if (nch <= 3) return launch_mma_bwd<128, 3, 5>(d, p, sums, st);
        return launch_mma_bwd<128, 5, 5>(d, p, sums, st);
    }
    const ProjArgs a = proj_args(d, p);
    switch (p.RB) {
        case 4: return launch_dt_bwd<io_t, 4>(d, a, p, sums, st);
        case 8: return launch_dt_bwd<io_t, 8>(d, a, p, sums, st);
        case 16: return launch_dt_bwd<io_t, 16>(d, a, p, sums, st);
        case 32: return launch_dt_bwd<io_t, 32>(d, a, p, sums, st);
        default: return launch_dt_bwd<io_t, 64>(d, a, p, sums, st);
    }
}

// bf16 operands: the tensor-core kernel, when the problem meets its alignment rules (otherwise, and for
// fp32, whose 1e-4 bar rules out tf32 operands, the CUDA-core kernel below).  Returns -1 for "not taken".
static int launch_wgrad_tc(const m2d_proj_desc* d, const ProjPlan& p, float* partials, WgSums* sums, cudaStream_t st) {
    const TcPlan t = tc_plan(d->P, d->E, p.K, d->proj_pitch, d->x, d->d_proj, p.slabs);
    if (!t.ok) return -1;
    CUtensorMap map_a, map_b;
    if (!tc_make_map(&map_a, d->d_proj, d->P, p.K, d->proj_pitch) || !tc_make_map(&map_b, d->x, d->P, d->E, d->E)) return -1;
    TcArgs a;
    a.K = p.K; a.E = d->E; a.nbk = t.nbk; a.stages = t.stages; a.total_blocks = t.total_blocks; a.blocks_per_cta = t.blocks_per_cta;
    a.partials = partials;
    a.status = wait_failure_flag();      // host memory: a wait that gives up shows in m2d_take_wait_failure()
    if (!allow_smem(reinterpret_cast<const void*>(xproj_wgrad_tc_kernel), t.smem)) return M2D_ERR_LAUNCH;
    xproj_wgrad_tc_kernel<<<dim3(t.grid_x, t.ny), 128, t.smem, st>>>(map_a, map_b, a);
    if (cudaGetLastError() != cudaSuccess) return M2D_ERR_LAUNCH;
    *sums = WgSums{partials, t.grid_x, (long long)p.K * d->E, d->d_Wx};
    return M2D_OK;
}

template <typename io_t>
static int launch_wgrad(const m2d_proj_desc* d, const ProjPlan& p, float* partials, WgSums* sums, cudaStream_t st) {
    if constexpr (sizeof(io_t) == 2) {
        const int rc = launch_wgrad_tc(d, p, partials, sums, st);
        if (rc >= 0) return rc;
    }
    WgArgs a;
    a.P = (int)d->P; a.pitch = (int)d->proj_pitch; a.E = d->E; a.K = p.K; a.rows_per_slab = p.rows_per_slab;
    a.x = d->x; a.d_proj = d->d_proj;
    a.partials = partials;
    if constexpr (sizeof(io_t) == 4) xproj_wgrad_f32_kernel<<<dim3(p.slabs, p.tilesE, p.tilesK), kWgThreads, 0, st>>>(a);
    else xproj_wgrad_kernel<<<dim3(p.slabs, p.tilesE, p.tilesK), 256, 0, st>>>(a);
    if (cudaGetLastError() != cudaSuccess) return M2D_ERR_LAUNCH;
    *sums = WgSums{partials, p.slabs, (long long)p.K * d->E, d->d_Wx};
    return M2D_OK;
}

// Either half of the backward, or both with their sums in one launch; the partial results of the second lie behind
// those of the first.
template <typename io_t>
static int launch_bwd(const m2d_proj_desc* d, const ProjPlan& p, bool dt, bool wgrad, cudaStream_t st) {
    DtSums ds{};
    WgSums ws{};
    int rc = dt ? dispatch_dt_bwd<io_t>(d, p, &ds, st) : M2D_OK;
    if (rc == M2D_OK && wgrad) rc = launch_wgrad<io_t>(d, p, reinterpret_cast<float*>(static_cast<char*>(d->workspace) + (dt ? p.dt_partials : 0)), &ws, st);
    return rc == M2D_OK ? launch_sums<io_t>(d, ds, ws, st) : rc;
}

static bool workspace_ok(const m2d_proj_desc* d, size_t need) {
    return need == 0 || (d->workspace && d->workspace_bytes >= need && aligned(d->workspace, 256));
}

}  // namespace m2d

using namespace m2d;

extern "C" uint64_t m2d_proj_workspace(const m2d_proj_desc* d) {
    if (check_proj(d) != M2D_OK) return 0;
    const ProjPlan p = plan_proj(d);
    return p.dt_partials + p.wg_partials;
}

extern "C" int m2d_dtproj_fwd(const m2d_proj_desc* d, void* stream) {
    const int rc = check_proj(d);
    if (rc != M2D_OK) return rc;
    if (!d->proj || !d->WT || !d->WL || !d->bT || !d->bL || !d->dT || !d->dL) return M2D_ERR_NULL;
    if (d->clear && (!aligned(d->clear, 16) || d->clear_bytes % 16)) return M2D_ERR_PITCH;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return d->dtype == M2D_F32 ? dispatch_dt_fwd<float>(d, st) : dispatch_dt_fwd<__nv_bfloat16>(d, st);
}

static int check_dt_bwd(const m2d_proj_desc* d) {
    if (!d->proj || !d->WT || !d->WL || !d->dT || !d->dL || !d->g_dT || !d->g_dL || !d->d_proj || !d->d_WT || !d->d_WL ||
        !d->d_bT || !d->d_bL)
        return M2D_ERR_NULL;
    // the g / delta rows are copied in 4-element pieces
    const size_t al = d->dtype == M2D_F32 ? 16 : 8;
    if (d->E % 4 != 0 || !aligned(d->g_dT, al) || !aligned(d->g_dL, al) || !aligned(d->dT, al) || !aligned(d->dL, al)) return M2D_ERR_PITCH;
    return M2D_OK;
}
static int check_wgrad(const m2d_proj_desc* d) {
    if (!d->x || !d->d_proj || !d->d_Wx) return M2D_ERR_NULL;
    const size_t al = d->dtype == M2D_F32 ? 16 : 8;
    if (d->E % 4 != 0 || d->proj_pitch % 4 != 0 || !aligned(d->x, al) || !aligned(d->d_proj, al)) return M2D_ERR_PITCH;
    return M2D_OK;
}
static int proj_bwd(const m2d_proj_desc* d, bool dt, bool wgrad, void* stream) {
    int rc = check_proj(d);
    if (rc == M2D_OK && dt) rc = check_dt_bwd(d);
    if (rc == M2D_OK && wgrad) rc = check_wgrad(d);
    if (rc != M2D_OK) return rc;
    const ProjPlan p = plan_proj(d);
    if (!workspace_ok(d, (dt ? p.dt_partials : 0) + (wgrad ? p.wg_partials : 0))) return M2D_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return d->dtype == M2D_F32 ? launch_bwd<float>(d, p, dt, wgrad, st) : launch_bwd<__nv_bfloat16>(d, p, dt, wgrad, st);
}

extern "C" int m2d_dtproj_bwd(const m2d_proj_desc* d, void* stream) { return proj_bwd(d, true, false, stream); }
extern "C" int m2d_xproj_wgrad(const m2d_proj_desc* d, void* stream) { return proj_bwd(d, false, true, stream); }
extern "C" int m2d_proj_bwd(const m2d_proj_desc* d, void* stream) { return proj_bwd(d, true, true, stream); }

extern "C" int m2d_xproj_wgrad_on_tensor_cores(const m2d_proj_desc* d) {
    if (check_proj(d) != M2D_OK || d->dtype != M2D_BF16 || !d->x || !d->d_proj) return 0;
    const ProjPlan p = plan_proj(d);
    const TcPlan t = tc_plan(d->P, d->E, p.K, d->proj_pitch, d->x, d->d_proj, p.slabs);
    if (!t.ok) return 0;
    CUtensorMap map_a, map_b;
    return tc_make_map(&map_a, d->d_proj, d->P, p.K, d->proj_pitch) && tc_make_map(&map_b, d->x, d->P, d->E, d->E) ? 1 : 0;
}
