// The eager entry points as native autograd nodes: wavefront_scan_cuda and wf_cuda_fn_pr of
// wavefront_cuda.py without the Python around the kernels.
//
// At the sizes of a single image or of the last stages the GPU work of a call is tens of microseconds
// while the Python formulation of it -- two autograd Functions, seven parameter casts, ctypes descriptors --
// takes hundreds.  Here a whole block call is ONE autograd node: the fp32 parameters go to the kernels as
// they are (no cast launches, and their gradients come back in fp32), the scan's backward writes the
// gradients of B and C straight into the columns of the projection's gradient, and the two parts of d_x meet
// in the GEMM that computes the second one.
//
// Every function returns None where it does not apply (shapes or dtypes outside the fused kernels' range,
// autocast to another type); the caller then takes the op-by-op path.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "m2d_proj.h"
#include "m2d_scan.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

void check(int rc, const char* fn) { TORCH_CHECK(rc == M2D_OK, fn, " failed: ", m2d_strerror(rc), " (status ", rc, ")"); }
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
int dtype_of(const Tensor& t) { return t.scalar_type() == at::kFloat ? M2D_F32 : M2D_BF16; }
bool supported(const Tensor& t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16; }
Tensor scratch(uint64_t bytes, const Tensor& like) { return at::empty({(int64_t)bytes}, like.options().dtype(at::kByte)); }

// A failed wait of an earlier launch (see m2d_take_wait_failure) surfaces here, like any other
// asynchronous error.
void check_waits() {
    TORCH_CHECK(!m2d_take_wait_failure(), "wavefront scan: a wait between CTAs of an earlier launch timed out; the results of that launch are invalid");
}

struct Dims {
    int64_t B, H, W, E, N, R, K;
};

struct ScanIn {      // what the scan reads; BT, BL, C with their pixel pitch
    Tensor x, dT, dL, AT, AL, BT, BL, C, D;
    int64_t pBT, pBL, pC;
};

m2d_scan_desc scan_desc(const Dims& s, const ScanIn& in, unsigned flags) {
    m2d_scan_desc d{};
    d.struct_bytes = sizeof(d);
    d.dtype = dtype_of(in.x);
    d.B = (int)s.B; d.H = (int)s.H; d.W = (int)s.W; d.E = (int)s.E; d.N = (int)s.N;
    d.flags = flags;
    d.x = in.x.data_ptr(); d.dT = in.dT.data_ptr(); d.dL = in.dL.data_ptr();
    d.AT = in.AT.data_ptr(); d.AL = in.AL.data_ptr();
    d.BT = in.BT.data_ptr(); d.BL = in.BL.data_ptr(); d.C = in.C.data_ptr();
    d.BT_pitch = in.pBT; d.BL_pitch = in.pBL; d.C_pitch = in.pC;
    d.D = in.D.data_ptr();
    return d;
}

Tensor scan_forward(const Dims& s, const ScanIn& in, unsigned flags) {
    m2d_scan_desc d = scan_desc(s, in, flags);
    Tensor y = at::empty({s.B, s.H, s.W, s.E}, in.x.options());
    d.y = y.data_ptr();
    d.workspace_bytes = m2d_scan_fwd_workspace(&d);
    const Tensor ws = scratch(d.workspace_bytes, in.x);
    d.workspace = ws.data_ptr();
    check(m2d_scan_fwd(&d, stream_of(in.x)), "m2d_scan_fwd");
    return y;
}

struct ScanGrads {
    Tensor x, dT, dL, AT, AL, D;
};

// `bt`, `bl`, `c`: where the gradients of B and C go, at `pitch` elements per pixel.
ScanGrads scan_backward(const Dims& s, const ScanIn& in, const Tensor& gy, void* bt, void* bl, void* c, int64_t pitch, unsigned flags) {
    m2d_scan_desc d = scan_desc(s, in, flags);
    const auto fp32 = in.x.options().dtype(at::kFloat);
    ScanGrads g;
    // the per-channel gradients are neighbours in the order the library zeroes them, where they share a type
    const auto aopt = (flags & M2D_SCAN_A_LOG) ? fp32 : in.x.options(), dopt = (flags & M2D_SCAN_D_F32) ? fp32 : in.x.options();
    if (aopt.dtype() == dopt.dtype()) {
        const Tensor small = at::empty({2 * s.E * s.N + s.E}, aopt);
        g.AT = small.narrow(0, 0, s.E * s.N).view({s.E, s.N});
        g.AL = small.narrow(0, s.E * s.N, s.E * s.N).view({s.E, s.N});
        g.D = small.narrow(0, 2 * s.E * s.N, s.E);
    } else {
        g.AT = at::empty({s.E, s.N}, aopt);
        g.AL = at::empty({s.E, s.N}, aopt);
        g.D = at::empty({s.E}, dopt);
    }
    g.x = at::empty({s.B, s.H, s.W, s.E}, in.x.options());
    g.dT = at::empty({s.B, s.H, s.W, s.E}, in.x.options());
    g.dL = at::empty({s.B, s.H, s.W, s.E}, in.x.options());
    d.gy = gy.data_ptr();
    d.d_x = g.x.data_ptr(); d.d_dT = g.dT.data_ptr(); d.d_dL = g.dL.data_ptr();
    d.d_AT = g.AT.data_ptr(); d.d_AL = g.AL.data_ptr(); d.d_D = g.D.data_ptr();
    d.d_BT = bt; d.d_BL = bl; d.d_C = c;
    d.d_BC_pitch = pitch;
    d.workspace_bytes = m2d_scan_bwd_workspace(&d);
    const Tensor ws = scratch(d.workspace_bytes, in.x);
    d.workspace = ws.data_ptr();
    check(m2d_scan_bwd(&d, stream_of(in.x)), "m2d_scan_bwd");
    return g;
}

// ---- the block call: projections + scan ---------------------------------------------------------

struct BlockParams {      // contiguous; Wx in x's type (a GEMM operand), the rest as they are
    Tensor AT_log, AL_log, Wx, WT, bT, WL, bL, D;
    bool f32;             // WT ... D are fp32 next to a bf16 x
};

m2d_proj_desc proj_desc(const Dims& s, const Tensor& x, const BlockParams& p) {
    m2d_proj_desc d{};
    d.struct_bytes = sizeof(d);
    d.dtype = dtype_of(x);
    d.P = s.B * s.H * s.W;
    d.E = (int)s.E; d.R = (int)s.R; d.N = (int)s.N;
    d.flags = p.f32 ? M2D_PROJ_PARAMS_F32 : 0;
    d.proj_pitch = s.K;
    d.WT = p.WT.data_ptr(); d.WL = p.WL.data_ptr();
    d.bT = p.bT.data_ptr(); d.bL = p.bL.data_ptr();
    return d;
}

struct Projected {
    Tensor proj, dT, dL;
};

Projected project(const Dims& s, const Tensor& x, const BlockParams& p) {
    const int64_t P = s.B * s.H * s.W;
    Projected o;
    o.proj = at::empty({P, s.K}, x.options());
    at::mm_out(o.proj, x.view({P, s.E}), p.Wx.t());
    o.dT = at::empty({s.B, s.H, s.W, s.E}, x.options());
    o.dL = at::empty({s.B, s.H, s.W, s.E}, x.options());
    m2d_proj_desc d = proj_desc(s, x, p);
    d.proj = o.proj.data_ptr();
    d.dT = o.dT.data_ptr(); d.dL = o.dL.data_ptr();
    check(m2d_dtproj_fwd(&d, stream_of(x)), "m2d_dtproj_fwd");
    return o;
}

ScanIn block_scan_in(const Dims& s, const Tensor& x, const BlockParams& p, const Projected& o) {
    ScanIn in;
    in.x = x; in.dT = o.dT; in.dL = o.dL;
    in.AT = p.AT_log; in.AL = p.AL_log; in.D = p.D;
    in.BT = o.proj.narrow(1, 2 * s.R, s.N);
    in.BL = o.proj.narrow(1, 2 * s.R + s.N, s.N);
    in.C = o.proj.narrow(1, 2 * s.R + 2 * s.N, s.N);
    in.pBT = in.pBL = in.pC = s.K;
    return in;
}

unsigned block_flags(const BlockParams& p, bool reverse) { return M2D_SCAN_A_LOG | (p.f32 ? M2D_SCAN_D_F32 : 0u) | (reverse ? M2D_SCAN_REVERSE : 0u); }

Dims block_dims(const Tensor& x, const Tensor& A_log, const Tensor& WT) {
    Dims s;
    s.B = x.size(0); s.H = x.size(1); s.W = x.size(2); s.E = x.size(3);
    s.N = A_log.size(1); s.R = WT.size(1); s.K = 2 * s.R + 3 * s.N;
    return s;
}

BlockParams block_params(const Tensor& x, const Tensor& AT_log, const Tensor& AL_log, const Tensor& Wx, const Tensor& WT, const Tensor& bT,
                         const Tensor& WL, const Tensor& bL, const Tensor& D) {
    BlockParams p;
    p.f32 = x.scalar_type() != at::kFloat && WT.scalar_type() == at::kFloat;
    p.AT_log = AT_log.to(at::kFloat).contiguous();
    p.AL_log = AL_log.to(at::kFloat).contiguous();
    p.Wx = Wx.to(x.scalar_type()).contiguous();
    p.WT = WT.contiguous(); p.bT = bT.contiguous(); p.WL = WL.contiguous(); p.bL = bL.contiguous(); p.D = D.contiguous();
    return p;
}

class BlockFn : public torch::autograd::Function<BlockFn> {
public:
    static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& AT_log, const Tensor& AL_log, const Tensor& Wx, const Tensor& WT,
                          const Tensor& bT, const Tensor& WL, const Tensor& bL, const Tensor& D, bool full, bool reverse) {
        const c10::cuda::CUDAGuard guard(x_.device());
        const Tensor x = x_.contiguous();
        const Dims s = block_dims(x, AT_log, WT);
        const BlockParams p = block_params(x, AT_log, AL_log, Wx, WT, bT, WL, bL, D);
        const Projected o = project(s, x, p);
        Tensor y = scan_forward(s, block_scan_in(s, x, p, o), block_flags(p, reverse));
        // "full" recomputation keeps x and the parameters only
        if (full) ctx->save_for_backward({x, AT_log, AL_log, Wx, WT, bT, WL, bL, D});
        else ctx->save_for_backward({x, AT_log, AL_log, Wx, WT, bT, WL, bL, D, o.proj, o.dT, o.dL});
        ctx->saved_data["reverse"] = reverse;
        return y;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const at::NoGradGuard no_grad;
        const variable_list v = ctx->get_saved_variables();
        const Tensor& x = v[0];
        const c10::cuda::CUDAGuard guard(x.device());
        const bool reverse = ctx->saved_data["reverse"].toBool();
        const Dims s = block_dims(x, v[1], v[4]);
        const BlockParams p = block_params(x, v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]);
        const int64_t P = s.B * s.H * s.W;
        Projected o;
        if (v.size() > 9) { o.proj = v[9]; o.dT = v[10]; o.dL = v[11]; }
        else o = project(s, x, p);
        const Tensor gy = grads[0].to(x.scalar_type()).contiguous();

        const bool f32 = x.scalar_type() == at::kFloat;      // the fp32 scan accumulates in place, the bf16 one in its workspace
        const Tensor d_proj = f32 ? at::zeros({P, s.K}, x.options()) : at::empty({P, s.K}, x.options());
        char* dp = static_cast<char*>(d_proj.data_ptr());
        const int64_t es = d_proj.element_size();
        const ScanGrads g = scan_backward(s, block_scan_in(s, x, p, o), gy, dp + 2 * s.R * es, dp + (2 * s.R + s.N) * es,
                                          dp + (2 * s.R + 2 * s.N) * es, s.K, block_flags(p, reverse) | (f32 ? M2D_SCAN_BC_ZEROED : 0u));

        const auto popt = p.f32 ? x.options().dtype(at::kFloat) : x.options();
        Tensor dWT = at::empty({s.E, s.R}, popt), dWL = at::empty({s.E, s.R}, popt), dbT = at::empty({s.E}, popt), dbL = at::empty({s.E}, popt);
        Tensor dWx = at::empty({s.K, s.E}, popt);
        m2d_proj_desc d = proj_desc(s, x, p);
        d.x = x.data_ptr(); d.proj = o.proj.data_ptr();
        d.dT = o.dT.data_ptr(); d.dL = o.dL.data_ptr();
        d.g_dT = g.dT.data_ptr(); d.g_dL = g.dL.data_ptr();
        d.d_proj = d_proj.data_ptr();
        d.d_WT = dWT.data_ptr(); d.d_WL = dWL.data_ptr(); d.d_bT = dbT.data_ptr(); d.d_bL = dbL.data_ptr();
        d.d_Wx = dWx.data_ptr();
        d.workspace_bytes = m2d_proj_workspace(&d);
        const Tensor ws = scratch(d.workspace_bytes, x);
        d.workspace = ws.data_ptr();
        check(m2d_dtproj_bwd(&d, stream_of(x)), "m2d_dtproj_bwd");
        check(m2d_xproj_wgrad(&d, stream_of(x)), "m2d_xproj_wgrad");
        // d_x = (scan's part) + d_proj @ Wx
        Tensor dx2 = g.x.view({P, s.E});
        at::addmm_out(dx2, dx2, d_proj, p.Wx);

        auto as = [](const Tensor& t, const Tensor& like) { return t.to(like.scalar_type()); };
        return {g.x, as(g.AT, v[1]), as(g.AL, v[2]), as(dWx, v[3]), dWT, dbT, dWL, dbL, g.D, Tensor(), Tensor()};
    }
};

// The fused projection kernels' range (the same rule as the op-by-op path's).
bool block_applies(const Tensor& x, const Tensor& AT_log, const Tensor& AL_log, const Tensor& Wx, const Tensor& WT, const Tensor& bT, const Tensor& WL,
                   const Tensor& bL, const Tensor& D) {
    if (!x.is_cuda() || !supported(x) || x.dim() != 4 || AT_log.dim() != 2 || WT.dim() != 2 || Wx.dim() != 2) return false;
    if (at::autocast::is_autocast_enabled(at::kCUDA) && at::autocast::get_autocast_dtype(at::kCUDA) != x.scalar_type()) return false;
    const int64_t E = x.size(3), N = AT_log.size(1), R = WT.size(1), K = 2 * R + 3 * N, P = x.numel() / std::max<int64_t>(E, 1);
    const int64_t bucket = R <= 4 ? 4 : R <= 8 ? 8 : R <= 16 ? 16 : R <= 32 ? 32 : 64;
    if (P < 1 || E < 1 || N < 1 || N > 16 || R < 1 || E > M2D_PROJ_MAX_E || R > M2D_PROJ_MAX_R || E % 4 || K % 4 || 4 * bucket > (E + 31) / 32 * 32) return false;
    if (P * std::max(E, K) >= (1ll << 31) - (1ll << 26)) return false;
    // one type for the parameters: x's own, or fp32 next to a bf16 x (A_log may be any float type: it is
    // used in fp32)
    const auto pt = WT.scalar_type();
    if (pt != x.scalar_type() && pt != at::kFloat) return false;
    for (const Tensor* t : {&Wx, &bT, &WL, &bL, &D})
        if (t->scalar_type() != pt || t->device() != x.device()) return false;
    for (const Tensor* t : {&AT_log, &AL_log, &WT})
        if (!t->is_floating_point() || t->device() != x.device()) return false;
    return AT_log.sizes() == at::IntArrayRef({E, N}) && AL_log.sizes() == AT_log.sizes() && Wx.sizes() == at::IntArrayRef({K, E}) &&
           WT.sizes() == at::IntArrayRef({E, R}) && WL.sizes() == WT.sizes() && bT.sizes() == at::IntArrayRef({E}) && bL.sizes() == bT.sizes() &&
           D.sizes() == bT.sizes();
}

c10::optional<Tensor> block(const Tensor& x, const Tensor& AT_log, const Tensor& AL_log, const Tensor& Wx, const Tensor& WT, const Tensor& bT,
                            const Tensor& WL, const Tensor& bL, const Tensor& D, bool full, bool reverse, bool gelu) {
    if (!block_applies(x, AT_log, AL_log, Wx, WT, bT, WL, bL, D)) return c10::nullopt;
    check_waits();
    bool grad = false;
    if (at::GradMode::is_enabled())
        for (const Tensor* t : {&x, &AT_log, &AL_log, &Wx, &WT, &bT, &WL, &bL, &D}) grad = grad || t->requires_grad();
    if (grad) {
        Tensor y = BlockFn::apply(x, AT_log, AL_log, Wx, WT, bT, WL, bL, D, full, reverse);
        return gelu ? at::gelu(y) : y;
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor xc = x.contiguous();
    const Dims s = block_dims(xc, AT_log, WT);
    const BlockParams p = block_params(xc, AT_log, AL_log, Wx, WT, bT, WL, bL, D);
    return scan_forward(s, block_scan_in(s, xc, p, project(s, xc, p)), block_flags(p, reverse) | (gelu ? M2D_SCAN_GELU_OUT : 0u));
}

// ---- the scan alone -----------------------------------------------------------------------------

// (tensor, pixel pitch): rows of a wider (B,H,W,K) buffer are read in place, anything else is made contiguous.
Tensor pixel_rows(const Tensor& t, const Dims& s, int64_t* pitch) {
    const int64_t K = t.stride(2);
    if (t.stride(3) == 1 && K >= s.N && t.stride(1) == s.W * K && t.stride(0) == s.H * s.W * K) {
        *pitch = K;
        return t;
    }
    *pitch = s.N;
    return t.contiguous();
}

ScanIn scan_in(const Dims& s, const Tensor& x, const Tensor& dT, const Tensor& dL, const Tensor& AT, const Tensor& AL, const Tensor& BT, const Tensor& BL,
               const Tensor& C, const Tensor& D) {
    ScanIn in;
    in.x = x.contiguous(); in.dT = dT.contiguous(); in.dL = dL.contiguous();
    in.AT = AT.contiguous(); in.AL = AL.contiguous(); in.D = D.contiguous();
    in.BT = pixel_rows(BT, s, &in.pBT); in.BL = pixel_rows(BL, s, &in.pBL); in.C = pixel_rows(C, s, &in.pC);
    return in;
}

Dims scan_dims(const Tensor& x, const Tensor& AT) {
    Dims s{};
    s.B = x.size(0); s.H = x.size(1); s.W = x.size(2); s.E = x.size(3); s.N = AT.size(1);
    return s;
}

class ScanFn : public torch::autograd::Function<ScanFn> {
public:
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& dT, const Tensor& dL, const Tensor& AT, const Tensor& AL,
                          const Tensor& BT, const Tensor& BL, const Tensor& C, const Tensor& D, int64_t flags) {
        const c10::cuda::CUDAGuard guard(x.device());
        const Dims s = scan_dims(x, AT);
        Tensor y = scan_forward(s, scan_in(s, x, dT, dL, AT, AL, BT, BL, C, D), (unsigned)flags);
        ctx->save_for_backward({x, dT, dL, AT, AL, BT, BL, C, D});
        ctx->saved_data["flags"] = flags;
        return y;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const at::NoGradGuard no_grad;
        const variable_list v = ctx->get_saved_variables();
        const c10::cuda::CUDAGuard guard(v[0].device());
        const Dims s = scan_dims(v[0], v[3]);
        const Tensor gy = grads[0].to(v[0].scalar_type()).contiguous();
        // one buffer for the three per-pixel gradients of B and C: one memset
        const int64_t n = s.B * s.H * s.W * s.N;
        const Tensor big = at::empty({3, s.B, s.H, s.W, s.N}, v[0].options());
        char* bp = static_cast<char*>(big.data_ptr());
        const int64_t es = big.element_size();
        const ScanGrads g = scan_backward(s, scan_in(s, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]), gy, bp, bp + n * es, bp + 2 * n * es, 0,
                                          (unsigned)ctx->saved_data["flags"].toInt());
        return {g.x, g.dT, g.dL, g.AT, g.AL, big.select(0, 0), big.select(0, 1), big.select(0, 2), g.D, Tensor()};
    }
};

c10::optional<Tensor> scan(const Tensor& x, const Tensor& dT, const Tensor& dL, const Tensor& AT, const Tensor& AL, const Tensor& BT, const Tensor& BL,
                           const Tensor& C, const Tensor& D, bool reverse, bool a_log) {
    // (whatever does not fit goes to the op-by-op path, which names the reason)
    if (!x.is_cuda() || !supported(x) || x.dim() != 4 || AT.dim() != 2 || AT.size(0) != x.size(3)) return c10::nullopt;
    const Dims s = scan_dims(x, AT);
    const int64_t N = s.N;
    for (const Tensor* t : {&dT, &dL})
        if (t->sizes() != x.sizes()) return c10::nullopt;
    for (const Tensor* t : {&BT, &BL, &C})
        if (t->sizes() != at::IntArrayRef({s.B, s.H, s.W, N})) return c10::nullopt;
    if (AL.sizes() != AT.sizes() || D.sizes() != at::IntArrayRef({s.E})) return c10::nullopt;
    for (const Tensor* t : {&dT, &dL, &BT, &BL, &C, &D})
        if (t->scalar_type() != x.scalar_type() || t->device() != x.device()) return c10::nullopt;
    for (const Tensor* t : {&AT, &AL})
        if (t->scalar_type() != (a_log ? at::kFloat : x.scalar_type()) || t->device() != x.device()) return c10::nullopt;
    check_waits();
    return ScanFn::apply(x, dT, dL, AT, AL, BT, BL, C, D, (int64_t)((reverse ? M2D_SCAN_REVERSE : 0u) | (a_log ? M2D_SCAN_A_LOG : 0u)));
}

}  // namespace

PYBIND11_MODULE(_entry, m) {
    m.def("block", &block, "wavefront_scan_cuda as one autograd node; None where it does not apply");
    m.def("scan", &scan, "wf_cuda_fn_pr as a native autograd node; None where it does not apply");
}
