// fp32 products of pixel rows with a small matrix: the x projection (P, E) @ Wx^T and the part of d_x that comes
// back through it, d_x += d_proj @ Wx.  Both have 10^2 ... 10^6 rows and at most a few hundred columns.
//
// The GEMM library runs fp32 at full precision on the CUDA cores, in tiles of 64 or 128 columns where these
// products have 56 ... 156: 102 and 132 us at P = 401408, E = 64 (262 us at P = 1048576) for operands that
// stream in 30 and 46 us (78 us), and 7.7 us for the 196 rows of one 14x14 image; 55 and 74 (132), and 3.3 here.  (A
// kernel's own times, in a graph; events around one call with the L2 flushed show 5 us more.)
//
// Here a float is split into three bf16 parts, exact to 24 bits, and a product of floats is the six products of
// parts that reach above 2^-24 of it, on the tensor cores (mma.sync m16n8k16: fragments are split in registers, where
// tcgen05 would want the parts of every row staged in shared memory).  The six are summed
// smallest first in a fresh accumulator per 16 terms and that sum is added to the running one by an ordinary
// fp32 add: the tensor cores' own accumulation truncates, and over E / 16 steps that would show.
//
// Parts of an infinity, or of a float beyond 3.39e38 whose first part rounds to one, have differences of infinities in
// them.  Whatever holds such a part sums to something that is not finite (inf * 0 is a NaN), so where the sums of a
// lane are not all finite it computes its results again, from the floats.  (Below 2^-110 the last part of a float
// falls under bf16's smallest number, 2^-133.)
#include <algorithm>

#include "m2d_proj.h"

#include "common.cuh"
#include "plan.cuh"
#include "proj_mma.cuh"

namespace m2d {

struct GemmArgs {
    long long rows;
    int n, k, ksteps, transposed, accumulate;      // w: (n, k) if transposed, else (k, n)
    const float *a, *w;
    float* out;
};

// Two neighbouring floats as three pairs of bf16 parts.
__device__ __forceinline__ void split2(float x, float y, unsigned (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const unsigned*>(&b);
        const float2 f = bf16x2_to_float2(p[i]);
        x -= f.x;
        y -= f.y;
    }
}

// The terms k0 ... k0 + 15 of a product meet in any order as long as both factors take the same one: a lane (row or
// column lane / 4, t = lane % 4) holds the four neighbours k0 + 4t ..., one 16-byte load of a row.
struct AFrag {
    unsigned part[3][4];
    __device__ __forceinline__ void set(const float4& top, const float4& bottom) {      // rows g and g + 8
        unsigned p[3];
        split2(top.x, top.y, p);
        for (int i = 0; i < 3; ++i) part[i][0] = p[i];
        split2(bottom.x, bottom.y, p);
        for (int i = 0; i < 3; ++i) part[i][1] = p[i];
        split2(top.z, top.w, p);
        for (int i = 0; i < 3; ++i) part[i][2] = p[i];
        split2(bottom.z, bottom.w, p);
        for (int i = 0; i < 3; ++i) part[i][3] = p[i];
    }
};
struct BFrag {
    uint2 part[3];
    __device__ __forceinline__ void set(const float4& v) {
        unsigned p[3], q[3];
        split2(v.x, v.y, p);
        split2(v.z, v.w, q);
        for (int i = 0; i < 3; ++i) part[i] = make_uint2(p[i], q[i]);
    }
};
// G n-tiles: the six products in turn over all of them, so that the next one that a sum waits for is G instructions
// away.
template <int G>
__device__ __forceinline__ void mma_split(float (*acc)[4], const AFrag& a, const BFrag (&b)[G]) {
    float t[G][4];
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        constexpr int ap[6] = {0, 2, 1, 0, 1, 0}, bp[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
        for (int n = 0; n < G; ++n) {
            if (p == 0) t[n][0] = t[n][1] = t[n][2] = t[n][3] = 0.f;
            mma_bf16(t[n], a.part[ap[p]], b[n].part[bp[p]].x, b[n].part[bp[p]].y);
        }
    }
#pragma unroll
    for (int n = 0; n < G; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] += t[n][i];
}

__device__ __forceinline__ float4 load_w(const GemmArgs& a, int col, int k) {      // w[k ... k + 3] of a column; k and a.k multiples of 4
    if (col >= a.n || k >= a.k) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.transposed) return __ldg(reinterpret_cast<const float4*>(a.w + (size_t)col * a.k + k));
    const float* w = a.w + (size_t)k * a.n + col;
    return make_float4(__ldg(w), __ldg(w + a.n), __ldg(w + 2 * (size_t)a.n), __ldg(w + 3 * (size_t)a.n));
}
__device__ __forceinline__ float4 load_a(const GemmArgs& a, long long row, int k) {
    return row < a.rows && k < a.k ? __ldg(reinterpret_cast<const float4*>(a.a + row * a.k + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ float2 load2(const GemmArgs& a, long long row, int col) {       // n is even
    return row < a.rows && col < a.n ? *reinterpret_cast<const float2*>(a.out + row * a.n + col) : make_float2(0.f, 0.f);
}
__device__ __forceinline__ void put2(const GemmArgs& a, long long row, int col, const float2& v) {
    if (row < a.rows && col < a.n) *reinterpret_cast<float2*>(a.out + row * a.n + col) = v;
}

// Two neighbouring results as ordinary fp32 sums of products.  (A NaN stays one, whatever is added.)
__device__ __forceinline__ float2 plain_sums(const GemmArgs& a, long long row, int col) {
    float2 s = make_float2(0.f, 0.f);
    if (row >= a.rows || col >= a.n) return s;
    const float* x = a.a + row * a.k;
    const float* w = a.w + (a.transposed ? (size_t)col * a.k : col);
    const int next = a.transposed ? 1 : a.n, other = a.transposed ? a.k : 1;
#pragma unroll 1
    for (int k = 0; k < a.k && !(isnan(s.x) && isnan(s.y)); ++k, w += next) {
        const float v = __ldg(x + k);
        s.x = fmaf(v, __ldg(w), s.x);
        s.y = fmaf(v, __ldg(w + other), s.y);
    }
    return s;
}
__device__ __forceinline__ void put_result(const GemmArgs& a, long long row, int col, float2 v) {
    if (a.accumulate) {
        const float2 old = load2(a, row, col);
        v.x += old.x;
        v.y += old.y;
    }
    put2(a, row, col, v);
}

// Many rows.  grid (CTAs, chunks of NT * 8 columns); a warp computes 16 rows at a time against the chunk, whose
// fragments every CTA splits once into shared memory.  The rows come straight from global memory, two steps of 16
// terms ahead, the first of the next tile among them.  Bound by the rate of mma.sync (four cycles of an SM each).  Two
// 16-row tiles per warp, which halve the reads of the fragments, need twice the registers: 166 against 112 us for the
// product that accumulates at P = 401408, E = 64, and nothing gained for the other (events, L2 flushed).  The look at
// the sums costs nothing that shows (67.3 / 67.8 and 86.9 / 86.4 us there without / with); a branch for each pair of
// results, between their stores, was 75 and 92.
template <int NT>
__global__ void __launch_bounds__(256, NT == 2 ? 3 : 2) rows_gemm_kernel(const GemmArgs a) {
    extern __shared__ uint2 gemm_w[];              // [step][n-tile][part][lane]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int col0 = blockIdx.y * NT * 8;
    for (int idx = threadIdx.x; idx < a.ksteps * NT * 32; idx += blockDim.x) {
        const int l = idx & 31, tile = idx >> 5;
        BFrag b;
        b.set(load_w(a, col0 + tile % NT * 8 + (l >> 2), tile / NT * 16 + (l & 3) * 4));
#pragma unroll
        for (int i = 0; i < 3; ++i) gemm_w[(tile * 3 + i) * 32 + l] = b.part[i];
    }
    __syncthreads();

    const long long step = (long long)gridDim.x * 128;
    long long row0 = ((long long)blockIdx.x * 8 + warp) * 16;
    long long lrow = row0 + g;                     // the next load: row and step
    int lks = 0;
    auto load = [&](float4 (&v)[2]) {
        v[0] = load_a(a, lrow, lks * 16 + t * 4);
        v[1] = load_a(a, lrow + 8, lks * 16 + t * 4);
        if (++lks == a.ksteps) {
            lks = 0;
            lrow += step;
        }
    };
    float4 next[2][2];
    load(next[0]);
    load(next[1]);
    for (; row0 < a.rows; row0 += step) {
        float acc[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
        for (int ks = 0; ks < a.ksteps; ++ks) {
            AFrag af;
            af.set(next[0][0], next[0][1]);
            next[0][0] = next[1][0];
            next[0][1] = next[1][1];
            load(next[1]);
            const uint2* w = gemm_w + ks * NT * 96 + lane;
            // groups of four n-tiles (and what is left of NT)
            auto group = [&](int n0, auto& b) {
                constexpr int N = sizeof(b) / sizeof(b[0]);
#pragma unroll
                for (int n = 0; n < N; ++n)
#pragma unroll
                    for (int i = 0; i < 3; ++i) b[n].part[i] = w[((n0 + n) * 3 + i) * 32];
                mma_split(&acc[n0], af, b);
            };
#pragma unroll
            for (int n0 = 0; n0 + 4 <= NT; n0 += 4) {
                BFrag b[4];
                group(n0, b);
            }
            if constexpr (NT % 4 != 0) {
                BFrag b[NT % 4];
                group(NT - NT % 4, b);
            }
        }
        // What is there already: all of it on its way before the first sum is waited for and stored (one by one, each
        // behind the store before it, 103 us against 75 at P = 401408, E = 64, of 16 cycles per issue 9 waiting for
        // global memory; 2 now).
        float2 old[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                old[n][h] = a.accumulate ? load2(a, row0 + g + 8 * h, col0 + n * 8 + t * 2) : make_float2(0.f, 0.f);
        float size[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) size[i] += fabsf(acc[n][i]);
        if (size[0] + size[1] + (size[2] + size[3]) < INFINITY) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float2 v = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
                    if (a.accumulate) { v.x += old[n][h].x; v.y += old[n][h].y; }
                    put2(a, row0 + g + 8 * h, col0 + n * 8 + t * 2, v);
                }
        } else {
#pragma unroll 1
            for (int i = 0; i < 2 * NT; ++i) {
                const long long row = row0 + g + i % 2 * 8;
                const int col = col0 + i / 2 * 8 + t * 2;
                put_result(a, row, col, plain_sums(a, row, col));
            }
        }
    }
}

// Few rows.  grid (16-row tiles, pairs of n-tiles); the warps of a CTA share out the steps of the contraction, read
// both factors straight from global memory, and their sums meet in shared memory: one load's latency, three
// steps at most, one barrier.
__global__ void __launch_bounds__(256) rows_gemm_small_kernel(const GemmArgs a) {
    __shared__ float sums[8][2][4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const long long row0 = (long long)blockIdx.x * 16;
    const int col0 = blockIdx.y * 16;
    float acc[2][4] = {};
#pragma unroll 3
    for (int ks = warp; ks < a.ksteps; ks += 8) {
        const int k = ks * 16 + t * 4;
        const float4 top = load_a(a, row0 + g, k), bottom = load_a(a, row0 + g + 8, k);
        const float4 w0 = load_w(a, col0 + g, k), w1 = load_w(a, col0 + 8 + g, k);
        AFrag af;
        af.set(top, bottom);
        BFrag b[2];
        b[0].set(w0);
        b[1].set(w1);
        mma_split(acc, af, b);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sums[warp][n][i][lane] = acc[n][i];
    __syncthreads();
    const int n = threadIdx.x >> 6, h = threadIdx.x >> 5 & 1;       // the first four warps: (n-tile, upper or lower rows)
    if (n >= 2) return;
    float x = 0.f, y = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        x += sums[w][n][2 * h][lane];
        y += sums[w][n][2 * h + 1][lane];
    }
    const long long row = row0 + h * 8 + g;
    const int col = col0 + n * 8 + t * 2;
    put_result(a, row, col, fabsf(x) + fabsf(y) < INFINITY ? make_float2(x, y) : plain_sums(a, row, col));
}

template <int NT>
static int launch_rows_gemm(const GemmArgs& a, int chunks, cudaStream_t st) {
    const auto kern = rows_gemm_kernel<NT>;
    const size_t smem = (size_t)a.ksteps * NT * 768;
    if (!allow_smem(reinterpret_cast<const void*>(kern), smem)) return M2D_ERR_LAUNCH;
    const int per_sm = resident_ctas(reinterpret_cast<const void*>(kern), 256, smem);
    const long long tiles = (a.rows + 127) / 128;
    const long long fit = std::max(1ll, (long long)std::max(per_sm, 1) * sm_count() / chunks);
    const long long rounds = (tiles + fit - 1) / fit;      // every CTA the same number of tiles, or one less
    kern<<<dim3((unsigned)((tiles + rounds - 1) / rounds), chunks), 256, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? M2D_OK : M2D_ERR_LAUNCH;
}

}  // namespace m2d

extern "C" int m2d_rows_gemm_f32(int64_t rows, int32_t n, int32_t k, const float* a, const float* w, int32_t transposed, int32_t accumulate,
                                 float* out, void* stream) {
    using namespace m2d;
    if (!a || !w || !out) return M2D_ERR_NULL;
    if (rows < 1 || n < 1 || k < 1) return M2D_ERR_SHAPE;
    if (n > 4 * M2D_PROJ_MAX_E || k > 4 * M2D_PROJ_MAX_E || rows > (1ll << 31)) return M2D_ERR_TOO_LARGE;
    if (n % 4 || k % 4 || !aligned(a, 16) || !aligned(w, 16) || !aligned(out, 16)) return M2D_ERR_PITCH;
    GemmArgs g;
    g.rows = rows; g.n = n; g.k = k; g.ksteps = (k + 15) / 16;
    g.transposed = transposed; g.accumulate = accumulate;
    g.a = a; g.w = w; g.out = out;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int tiles_n = (n + 7) / 8, sms = sm_count();
    // Column chunks: as few as keep the accumulators (8 n-tiles) and two CTAs' fragments on an SM, more while the
    // 128-row tiles alone do not give every SM a CTA.  Where even chunks of two n-tiles do not, the contraction is
    // split instead.
    const long long tiles = (rows + 127) / 128;
    int chunks = (tiles_n + 7) / 8, nt;
    for (;; ++chunks) {
        nt = (tiles_n + chunks - 1) / chunks;
        if (nt <= 2 || ((size_t)g.ksteps * nt * 768 <= 100 * 1024 && tiles * chunks >= sms)) break;
    }
    nt = nt == 1 ? 2 : nt == 3 ? 4 : nt;           // (the instantiated widths)
    chunks = (tiles_n + nt - 1) / nt;
    if ((size_t)g.ksteps * nt * 768 > 200 * 1024) return M2D_ERR_TOO_LARGE;
    if (tiles * chunks < sms) {
        rows_gemm_small_kernel<<<dim3((unsigned)((rows + 15) / 16), (tiles_n + 1) / 2), 256, 0, st>>>(g);
        return cudaGetLastError() == cudaSuccess ? M2D_OK : M2D_ERR_LAUNCH;
    }
    switch (nt) {
        case 2: return launch_rows_gemm<2>(g, chunks, st);
        case 4: return launch_rows_gemm<4>(g, chunks, st);
        case 5: return launch_rows_gemm<5>(g, chunks, st);
        case 6: return launch_rows_gemm<6>(g, chunks, st);
        case 7: return launch_rows_gemm<7>(g, chunks, st);
        default: return launch_rows_gemm<8>(g, chunks, st);
    }
}
