// The dt projections on the tensor cores (mma.sync m16n8k16, bf16 operands, fp32 accumulators).
//
// delta = softplus(r @ W^T + b) and its backward are contractions over a rank R of 4 ... 36 or over the
// pixels, next to one transcendental per element.  On the CUDA cores they cost R multiply-adds per
// element and were bound by issue slots (R = 20, E = 320: 60 us forward, 166 us backward for 16 M elements
// of bf16 whose traffic takes 5 and 10 us; 33 and 56 here, all in a graph).  The products are too small in K (forward) and N (backward)
// for tcgen05 to pay: a 128x256x16 tile would be nine tenths padding or wait on its own epilogue; mma.sync
// fragments are consumed where they are produced.
//
// fp32 precision from bf16 operands: a float is split into three bf16 parts, h + m + l, exact to 24 bits, and
// a product of two floats is the six products that reach above 2^-24 of it (hh, hm, mh, hl, mm, lh).
// With bf16 tensors r and W are exact already: the forward needs one product, and in the backward only
// s = g * softplus' is split, three products.
#pragma once

#include "common.cuh"

namespace m2d {

// Element of a weight or bias: of the I/O type, or fp32 rounded to it.
template <typename io_t>
__device__ __forceinline__ float load_param(const void* p, int off, int f32) {
    if (!f32) return load1(static_cast<const io_t*>(p), off);
    const float v = __ldg(static_cast<const float*>(p) + off);
    return sizeof(io_t) == 2 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x2_trans(unsigned& r0, unsigned& r1, unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}

// v = part 0 + part 1 + part 2 to 24 bits; parts as bf16.
__device__ __forceinline__ __nv_bfloat16 split_part(float v, int part) {
    __nv_bfloat16 p = __float2bfloat16_rn(v);
    for (int k = 0; k < part; ++k) {
        v -= __bfloat162float(p);
        p = __float2bfloat16_rn(v);
    }
    return p;
}
__device__ __forceinline__ float2 bf16x2_to_float2(unsigned u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// The six products of a three-way split, in the order of the K-extended operands: part of the left factor and
// part of the right one.
__device__ __forceinline__ int left_part(int g) { return g == 2 || g == 5 ? 1 : (g == 4 ? 2 : 0); }
__device__ __forceinline__ int right_part(int g) { return g == 1 || g == 5 ? 1 : (g == 3 ? 2 : 0); }

__device__ __forceinline__ float rcp_approx(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// The larger of two, NaN if either is (fmaxf would drop it).
__device__ __forceinline__ float max_nan(float a, float b) {
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}
// softplus with the reference's threshold of 20 (torch.nn.functional.softplus defaults)
// log1p(t) for t in (0, 1] as 2*atanh(t / (2 + t)): the argument stays below 1/3, where seven terms of
// the series are exact to fp32 rounding (next term 2 s^15 / 15 < 1e-8 of the result); half the
// instructions of log1pf, which was a third of the forward kernel.
__device__ __forceinline__ float log1p_unit(float t) {
    const float s = __fdividef(t, 2.f + t), s2 = s * s;
    float p = 1.f / 13.f;
    p = fmaf(p, s2, 1.f / 11.f);
    p = fmaf(p, s2, 1.f / 9.f);
    p = fmaf(p, s2, 1.f / 7.f);
    p = fmaf(p, s2, 1.f / 5.f);
    p = fmaf(p, s2, 1.f / 3.f);
    p = fmaf(p, s2, 1.f);
    return 2.f * s * p;
}
// softplus(z) = max(z, 0) + log1p(exp(-|z|)); past the reference's threshold of 20 the second term is
// below half an ulp of z, so the threshold of torch.nn.functional.softplus needs no branch
__device__ __forceinline__ float softplus_f(float z) {
    // exp(-|z|) = 2^(a + e): a is the rounded product with log2(e); e collects what that rounding and
    // the rounding of the constant lost (without it the error grows with |z|: 3e-6 at |z| = 60)
    const float m = max_nan(-fabsf(z), -200.f);      // (exp is zero there; an infinity would leave no remainder)
    const float a = m * kLog2e;
    const float e = fmaf(m, kLog2e, -a) + m * 1.92596299e-8f;
    const float t = ex2(a) * fmaf(e, kLn2, 1.f);
    return fmaxf(z, 0.f) + log1p_unit(t);
}
// softplus of two values: max(z, 0) + log1p(exp(-|z|)), the arithmetic of softplus_f on packed pairs.  (The
// divisor of the series' argument is 2 + t in (2, 3]: a plain reciprocal needs none of a division's scaling.)
// Without ANY a |z| whose product with log2(e) overflows, from 2.3e38 on, gives NaN.
template <bool ANY>
__device__ __forceinline__ float2 softplus2(float2 z) {
    const float2 m = ANY ? make_float2(max_nan(-fabsf(z.x), -200.f), max_nan(-fabsf(z.y), -200.f)) : make_float2(-fabsf(z.x), -fabsf(z.y));
    const float2 b = __fmul2_rn(m, dup2(-kLog2e));          // exp(-|z|) = 2^(-b + e), e what rounding b lost
    const float2 e = __ffma2_rn(m, dup2(1.92596299e-8f), __ffma2_rn(m, dup2(kLog2e), b));
    const float2 t = __fmul2_rn(make_float2(ex2(-b.x), ex2(-b.y)), __ffma2_rn(e, dup2(kLn2), dup2(1.f)));
    const float2 q = __fadd2_rn(t, dup2(2.f));
    const float2 s = __fmul2_rn(t, make_float2(rcp_approx(q.x), rcp_approx(q.y)));
    const float2 s2 = __fmul2_rn(s, s);
    // 2 atanh(s) / s on s^2 in (0, 1/9]: interpolated at Chebyshev nodes, within 4e-9 (a series needs seven terms)
    float2 p = dup2(0.28157778f);
    p = __ffma2_rn(p, s2, dup2(0.27965158f));
    p = __ffma2_rn(p, s2, dup2(0.40024595f));
    p = __ffma2_rn(p, s2, dup2(0.66666322f));
    p = __ffma2_rn(p, s2, dup2(2.f));
    return __ffma2_rn(s, p, make_float2(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f)));
}
// 1 - exp(-d) of two softplus outputs: softplus' through its own output; a short series where it cancels.
__device__ __forceinline__ float2 softplus_grad2(float2 d) {
    const float2 n = make_float2(-d.x, -d.y);
    float2 q = __ffma2_rn(n, dup2(1.f / 120.f), dup2(1.f / 24.f));
    q = __ffma2_rn(n, q, dup2(1.f / 6.f));
    q = __ffma2_rn(n, q, dup2(0.5f));
    q = __ffma2_rn(n, q, dup2(1.f));
    q = __fmul2_rn(d, q);
    const float2 e = make_float2(1.f - __expf(n.x), 1.f - __expf(n.y));
    return make_float2(d.x < 0.1f ? q.x : e.x, d.y < 0.1f ? q.y : e.y);
}

// ------------------------------------------------------------------------------------------------
// Forward.  grid (CTAs, 2 directions, channel chunks); a warp computes 16 pixels x the chunk's channels.  The
// rank is extended to K' = R (bf16) or 6R (fp32, the six products side by side) and padded to 16.  Columns of
// W are dealt to the fragments so that a lane's results over four n-tiles are 8 neighbouring channels:
// 16-byte stores.  What infinite and very large sums cost, us without / with: fp32 P = 401408, E = 64 80.5 / 80.7, 1048576, 64
// 180.4 / 181.3, 25088, 320 57.1 / 58.0; bf16 401408, 64 60.2 / 61.7, 25088, 320 42.5 / 43.2 (events around one call, L2 flushed);
// fp32 rows that are all NaN take up to three times as long.
// (The bounds are the CTAs an SM takes; left to itself the compiler spills fp32 into 48 registers for the sake of the call.)
// ------------------------------------------------------------------------------------------------
// Memory that a kernel zeroes before anything else, so that the stores drain while its weights and first rows
// arrive: a memset of its own is a launch.  Worth it for small pieces; the 537 MB of boundary rows of a 1024x1024
// map cost 95 us here, as a burst or next to each tile, against a memset's 87.
struct Clear {
    uint4* p;
    long long n;
    __device__ __forceinline__ void run() const {
        const long long cta = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x, ctas = (long long)gridDim.x * gridDim.y * gridDim.z;
        for (long long i = cta * blockDim.x + threadIdx.x; i < n; i += ctas * blockDim.x) p[i] = make_uint4(0u, 0u, 0u, 0u);
    }
};

struct MmaFwdArgs {
    Clear clear;
    int P, pitch, E, R, nk, chunk, params_f32;     // chunk: channels per CTA, a multiple of 32
    const void *proj, *WT, *WL, *bT, *bL;
    void *dT, *dL;
};

// 16 pixels with ordinary multiply-adds, a lane owns a channel: for fp32 tiles that hold an infinity, a float that rounds
// to one in bf16, or a sum beyond softplus2<false>'s range.  (The parts of the first two hold differences of infinities; all
// three show as a NaN.)  Kept out of the kernel's registers and schedule: a branch inside its loop cost up to a tenth of it.
template <typename io_t>
__device__ __noinline__ void dtproj_fwd_plain(const io_t* proj, int pitch, int pixels, const void* W, const void* bias, int e0, int params_f32, int R, int ec,
                                              io_t* out, int E) {
    for (int ch = threadIdx.x & 31; ch < ec; ch += 32)
        for (int i = 0; i < pixels; ++i) {
            float z = load_param<io_t>(bias, e0 + ch, params_f32);
            for (int r = 0; r < R && !isnan(z); ++r) z = fmaf(load1(proj, (long long)i * pitch + r), load_param<io_t>(W, (e0 + ch) * R + r, params_f32), z);
            store1(out, (long long)i * E + ch, softplus_f(z));
        }
}

template <typename io_t> __host__ __device__ inline int mma_k(int R) { return ((sizeof(io_t) == 4 ? 6 * R : R) + 15) / 16; }
__host__ __device__ inline size_t mma_fwd_smem(int chunk, int nk) {
    const int nt = chunk / 8;
    return (size_t)nt * nk * 256 + (size_t)nt * 8 * sizeof(float) + (size_t)8 * 16 * (nk * 16 + 8) * 2;
}

template <typename io_t>
__global__ void __launch_bounds__(256, sizeof(io_t) == 4 ? 3 : 4) dtproj_fwd_mma_kernel(const MmaFwdArgs a) {
    extern __shared__ __align__(16) char smem_mma[];
    const int dir = blockIdx.y, e0 = blockIdx.z * a.chunk, ec = min(a.chunk, a.E - e0);
    const int nt = a.chunk / 8, nk = a.nk, ks = nk * 16, R = a.R;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, q = lane & 3, row = lane >> 2;
    uint2* const Bf = reinterpret_cast<uint2*>(smem_mma);
    float* const bias = reinterpret_cast<float*>(smem_mma + (size_t)nt * nk * 256);
    const int lda = ks + 8;                        // 16 bytes of padding: rows of a fragment in different banks
    __nv_bfloat16* const At = reinterpret_cast<__nv_bfloat16*>(bias + nt * 8) + w * 16 * lda;
    const void* W = dir ? a.WL : a.WT;
    const void* bp = dir ? a.bL : a.bT;
    constexpr bool F32 = sizeof(io_t) == 4;
    a.clear.run();

    // W into B fragments: every element is read once, in order, and its parts go where the fragments want them
    for (int idx = threadIdx.x; idx < nt * nk * 32; idx += blockDim.x) Bf[idx] = make_uint2(0, 0);
    __syncthreads();
#pragma unroll 4
    for (int idx = threadIdx.x; idx < ec * R; idx += blockDim.x) {
        const int c = idx / R, r = idx - c * R;
        const float v = load_param<io_t>(W, e0 * R + idx, a.params_f32);
        const int t = c / 32 * 4 + c % 8 / 2, n = c % 32 / 8 * 2 + (c & 1);
        auto put = [&](int k, __nv_bfloat16 part) {
            const int kr = k % 16;
            reinterpret_cast<__nv_bfloat16*>(Bf + (t * nk + k / 16) * 32 + n * 4 + kr % 8 / 2)[kr / 8 * 2 + (k & 1)] = part;
        };
        if (F32) {
            const __nv_bfloat16 part[3] = {split_part(v, 0), split_part(v, 1), split_part(v, 2)};
#pragma unroll
            for (int g = 0; g < 6; ++g) put(g * R + r, part[right_part(g)]);
        } else {
            put(r, __float2bfloat16_rn(v));
        }
    }
    // (a bias of -inf is as good as -1e38: it must not send every tile the slow way)
    for (int k = threadIdx.x; k < nt * 8; k += blockDim.x) bias[k] = e0 + k < a.E ? max_nan(load_param<io_t>(bp, e0 + k, a.params_f32), F32 ? -1e38f : -INFINITY) : 0.f;
    for (int k = lane; k < 16 * lda; k += 32) At[k] = __nv_bfloat16(0.f);
    __syncthreads();

    const io_t* const proj = static_cast<const io_t*>(a.proj) + dir * R;
    io_t* const out = static_cast<io_t*>(dir ? a.dL : a.dT) + e0;
    const unsigned a_addr = smem_u32(At + (lane & 15) * lda + (lane >> 4) * 8);
    for (int p0 = (blockIdx.x * 8 + w) * 16; p0 < a.P; p0 += gridDim.x * 128) {
        __syncwarp();
        for (int idx = lane; idx < 16 * R; idx += 32) {
            const int i = idx / R, r = idx - i * R;
            const float v = p0 + i < a.P ? load1(proj, (long long)(p0 + i) * a.pitch + r) : 0.f;
            __nv_bfloat16* const d = At + i * lda + r;
            if (F32) {
                const __nv_bfloat16 part[3] = {split_part(v, 0), split_part(v, 1), split_part(v, 2)};
#pragma unroll
                for (int g = 0; g < 6; ++g) d[g * R] = part[left_part(g)];
            } else {
                d[0] = __float2bfloat16_rn(v);
            }
        }
        __syncwarp();
        const bool ok0 = p0 + row < a.P, ok1 = p0 + row + 8 < a.P;
        io_t* const o0 = out + (long long)(p0 + row) * a.E, *const o1 = o0 + (long long)8 * a.E;
        float2 sum = make_float2(0.f, 0.f);
        for (int g = 0; g < nt / 4; ++g) {
            float acc[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
            for (int kk = 0; kk < nk; ++kk) {
                unsigned af[4];
                ldmatrix_x4(af, a_addr + kk * 32);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint2 b = Bf[((g * 4 + j) * nk + kk) * 32 + lane];
                    mma_bf16(acc[j], af, b.x, b.y);
                }
            }
            const int ch = g * 32 + q * 8;
            if (ch < ec) {
                float2 v0[4], v1[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 b = *reinterpret_cast<const float2*>(bias + ch + 2 * j);
                    v0[j] = softplus2<!F32>(__fadd2_rn(make_float2(acc[j][0], acc[j][1]), b));
                    v1[j] = softplus2<!F32>(__fadd2_rn(make_float2(acc[j][2], acc[j][3]), b));
                }
                if (F32) {
                    float* f0 = reinterpret_cast<float*>(o0 + ch), *f1 = reinterpret_cast<float*>(o1 + ch);
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        if (ok0) *reinterpret_cast<float4*>(f0 + 2 * j) = make_float4(v0[j].x, v0[j].y, v0[j + 1].x, v0[j + 1].y);
                        if (ok1) *reinterpret_cast<float4*>(f1 + 2 * j) = make_float4(v1[j].x, v1[j].y, v1[j + 1].x, v1[j + 1].y);
                    }
                } else {
                    if (ok0) *reinterpret_cast<uint4*>(o0 + ch) = make_uint4(pack_bf16x2(v0[0].x, v0[0].y), pack_bf16x2(v0[1].x, v0[1].y), pack_bf16x2(v0[2].x, v0[2].y), pack_bf16x2(v0[3].x, v0[3].y));
                    if (ok1) *reinterpret_cast<uint4*>(o1 + ch) = make_uint4(pack_bf16x2(v1[0].x, v1[0].y), pack_bf16x2(v1[1].x, v1[1].y), pack_bf16x2(v1[2].x, v1[2].y), pack_bf16x2(v1[3].x, v1[3].y));
                }
                if (F32) {                         // (no result is below zero: a NaN among them is one of the sum)
#pragma unroll
                    for (int j = 0; j < 4; ++j) sum = __fadd2_rn(__fadd2_rn(v0[j], v1[j]), sum);
                }
            }
        }
        if (F32 && __any_sync(0xffffffffu, isnan(sum.x + sum.y)))
            dtproj_fwd_plain<io_t>(proj + (long long)p0 * a.pitch, a.pitch, min(16, a.P - p0), W, bp, e0, a.params_f32, R, ec, out + (long long)p0 * a.E, a.E);
    }
}

// ------------------------------------------------------------------------------------------------
// Backward.  With s = g * (1 - exp(-delta)) (P x E):
//     d_W[e][r] = sum_p s*r     d_b[e] = sum_p s (the column of ones beside r)     d_r[p][r] = sum_e s*W
// grid (CTAs, 2 directions); a CTA takes 8192 elements at a time, 64 pixels x 128 channels or, for narrow E,
// 128 pixels x 64 channels: s is formed once, split and parked in shared memory as bf16, from where ldmatrix
// reads it with the pixels as K (d_W: a warp owns 16 channels, and with 64 of them one half of the pixels, and
// keeps its sums in registers over all tiles) and with the channels as K (d_r: a warp owns 16 pixels, and with
// 64 of them one half of the channels).
// ------------------------------------------------------------------------------------------------
template <int CH> struct MmaTile {
    static constexpr int kPix = 8192 / CH, kLds = CH + 8;     // rows of s start in different banks
};

struct MmaBwdArgs {
    int P, pitch, E, R, RB, EB, params_f32;
    const void *proj, *WT, *WL, *dT, *dL, *g_dT, *g_dL;
    void* d_proj;
    float* partials;                   // [dir][cta][RB+1][EB]
};

template <int CH>
__host__ __device__ inline size_t mma_bwd_smem(int nch, int nt) {
    typedef MmaTile<CH> T;
    return (size_t)3 * T::kPix * T::kLds * 2 + (size_t)T::kPix * (nt | 1) * 8 * 2 +
           (size_t)nch * (CH / 16) * nt * 256 + (size_t)T::kPix * nt * 8 * sizeof(float);
}

template <int CH, int NCH, int NT>
__global__ void __launch_bounds__(256) dtproj_bwd_mma_kernel(const MmaBwdArgs a) {
    extern __shared__ __align__(16) char smem_mma[];
    typedef __nv_bfloat16 io_t;
    constexpr int RS = (NT | 1) * 8;      // RS: an odd number of 16-byte pieces per row of r
    constexpr int PIX = MmaTile<CH>::kPix, LDS = MmaTile<CH>::kLds, KS = CH / 16;
    constexpr bool WIDE = CH == 128;
    __nv_bfloat16* const S = reinterpret_cast<__nv_bfloat16*>(smem_mma);
    __nv_bfloat16* const Rt = S + 3 * PIX * LDS;
    uint2* const Wf = reinterpret_cast<uint2*>(Rt + PIX * RS);
    float* const dr = reinterpret_cast<float*>(Wf + NCH * KS * NT * 32);
    const int dir = blockIdx.y, R = a.R;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, q = lane & 3, row = lane >> 2;
    const void* W = dir ? a.WL : a.WT;
    const io_t* const proj = static_cast<const io_t*>(a.proj) + dir * R;
    const io_t* const delta = static_cast<const io_t*>(dir ? a.dL : a.dT);
    const io_t* const grad = static_cast<const io_t*>(dir ? a.g_dL : a.g_dT);
    io_t* const d_proj = static_cast<io_t*>(a.d_proj) + dir * R;

    // W as B fragments (K = channels, N = ranks): read once, in order
    for (int idx = threadIdx.x; idx < NCH * KS * NT * 32; idx += blockDim.x) Wf[idx] = make_uint2(0, 0);
    __syncthreads();
#pragma unroll 4
    for (int idx = threadIdx.x; idx < a.E * R; idx += blockDim.x) {
        const int ch = idx / R, r = idx - ch * R, kr = ch % 16;
        const float v = load_param<io_t>(W, idx, a.params_f32);
        __nv_bfloat16* const dst = reinterpret_cast<__nv_bfloat16*>(Wf + (ch / 16 * NT + r / 8) * 32 + r % 8 * 4 + kr % 8 / 2) + kr / 8 * 2 + (ch & 1);
        *dst = __float2bfloat16_rn(v);
    }
    float accW[NCH][NT][4];
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) accW[c][t][i] = 0.f;

    // ldmatrix row addresses: s with pixels as K (transposed), with channels as K, and r
    const unsigned s_base = smem_u32(S);
    const int wt = WIDE ? w : w & 3, wh = WIDE ? 0 : w >> 2;               // d_W: channel tile, half of the pixels
    const unsigned sT_addr = s_base + ((wh * 64 + (lane & 7) + (lane >> 4) * 8) * LDS + wt * 16 + ((lane >> 3) & 1) * 8) * 2;
    const int mt = WIDE ? w & 3 : w, kh = WIDE ? w >> 2 : 0;               // d_r: pixel tile, half of the channels
    const unsigned sN_addr = s_base + ((mt * 16 + (lane & 15)) * LDS + kh * 64 + (lane >> 4) * 8) * 2;
    const unsigned r_addr = smem_u32(Rt) + (wh * 64 + (lane & 15)) * RS * 2;
    constexpr int SP = PIX * LDS * 2;              // bytes between parts

    for (int p0 = blockIdx.x * PIX; p0 < a.P; p0 += gridDim.x * PIX) {
        __syncthreads();
        for (int idx = threadIdx.x; idx < PIX * NT * 8; idx += blockDim.x) {
            const int i = idx / (NT * 8), r = idx % (NT * 8);
            const float v = p0 + i < a.P && r < R ? load1(proj, (long long)(p0 + i) * a.pitch + r) : (r == R ? 1.f : 0.f);
            Rt[i * RS + r] = __float2bfloat16_rn(v);
        }
        float accR[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) accR[t][i] = 0.f;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            if (c * CH >= a.E) break;
            if (c > 0) __syncthreads();
            // s of the tile, eight channels per item
            constexpr int V = 8, ITEMS = PIX * CH / V / 256;
#pragma unroll
            for (int i0 = 0; i0 < ITEMS; i0 += 4) {
                uint4 gv[4], dv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int it = threadIdx.x + (i0 + i) * 256, px = it / (CH / V), ch = c * CH + it % (CH / V) * V;
                    gv[i] = dv[i] = make_uint4(0, 0, 0, 0);
                    if (p0 + px < a.P && ch < a.E) {
                        const long long off = (long long)(p0 + px) * a.E + ch;
                        gv[i] = __ldg(reinterpret_cast<const uint4*>(grad + off));
                        dv[i] = __ldg(reinterpret_cast<const uint4*>(delta + off));
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int it = threadIdx.x + (i0 + i) * 256, px = it / (CH / V), cl = it % (CH / V) * V;
                    const unsigned gu[4] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w}, du[4] = {dv[i].x, dv[i].y, dv[i].z, dv[i].w};
                    unsigned o[3][V / 2];
#pragma unroll
                    for (int j = 0; j < V / 2; ++j) {
                        const float2 g = bf16x2_to_float2(gu[j]);
                        const float2 d = bf16x2_to_float2(du[j]);
                        float2 s = __fmul2_rn(g, softplus_grad2(d));
#pragma unroll
                        for (int part = 0; part < 3; ++part) {
                            o[part][j] = pack_bf16x2(s.x, s.y);
                            const float2 b = bf16x2_to_float2(o[part][j]);
                            s = __fadd2_rn(s, make_float2(-b.x, -b.y));
                        }
                    }
                    __nv_bfloat16* const dst = S + px * LDS + cl;
#pragma unroll
                    for (int part = 0; part < 3; ++part) memcpy(__builtin_assume_aligned(dst + part * PIX * LDS, V * 2), o[part], V * 2);
                }
            }
            __syncthreads();
            if (c * CH + wt * 16 < a.E) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    unsigned af[3][4];
#pragma unroll
                    for (int part = 0; part < 3; ++part) ldmatrix_x4_trans(af[part], sT_addr + part * SP + k * 16 * LDS * 2);
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        unsigned b0, b1;
                        ldmatrix_x2_trans(b0, b1, r_addr + (k * 16 * RS + t * 8) * 2);
#pragma unroll
                        for (int part = 0; part < 3; ++part) mma_bf16(accW[c][t], af[part], b0, b1);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (c * CH + kh * 64 + k * 16 >= a.E) break;
                unsigned af[3][4];
#pragma unroll
                for (int part = 0; part < 3; ++part) ldmatrix_x4(af[part], sN_addr + part * SP + k * 32);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const uint2 b = Wf[((c * KS + kh * 4 + k) * NT + t) * 32 + lane];
#pragma unroll
                    for (int part = 0; part < 3; ++part) mma_bf16(accR[t], af[part], b.x, b.y);
                }
            }
        }
        if (kh == 1) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                *reinterpret_cast<float2*>(dr + (mt * 16 + row) * NT * 8 + t * 8 + 2 * q) = make_float2(accR[t][0], accR[t][1]);
                *reinterpret_cast<float2*>(dr + (mt * 16 + row + 8) * NT * 8 + t * 8 + 2 * q) = make_float2(accR[t][2], accR[t][3]);
            }
        }
        if (WIDE) __syncthreads();
        if (kh == 0) {
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int px = mt * 16 + row + (i >> 1) * 8, r = t * 8 + 2 * q + (i & 1);
                    if (p0 + px < a.P && r < R) store1(d_proj, (long long)(p0 + px) * a.pitch + r, accR[t][i] + (WIDE ? dr[px * NT * 8 + r] : 0.f));
                }
        }
    }
    float* const part = a.partials + ((size_t)dir * gridDim.x + blockIdx.x) * (a.RB + 1) * a.EB;
    if (!WIDE) {                                   // the two halves of the pixels
        __syncthreads();
        float* const sh = reinterpret_cast<float*>(smem_mma) + ((size_t)wt * 32 + lane) * NCH * NT * 4;
        if (wh == 1) {
#pragma unroll
            for (int k = 0; k < NCH * NT * 4; ++k) sh[k] = accW[k / (NT * 4)][k / 4 % NT][k % 4];
        }
        __syncthreads();
        if (wh == 1) return;
#pragma unroll
        for (int k = 0; k < NCH * NT * 4; ++k) accW[k / (NT * 4)][k / 4 % NT][k % 4] += sh[k];
    }
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = c * CH + wt * 16 + row + (i >> 1) * 8, r = t * 8 + 2 * q + (i & 1);
                if (e < a.E && r <= R) part[(r == R ? a.RB : r) * a.EB + e] = accW[c][t][i];
            }
}

}  // namespace m2d
