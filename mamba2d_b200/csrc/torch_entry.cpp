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
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/CachingHostAllocator.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDAGuard.h>
#include <cublas_v2.h>
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

// What a call is to do besides its arithmetic; as one number, which a node keeps between its passes.
struct Options {
    unsigned flags = 0;      // of the scan
    bool check = true;       // raise where a launch went wrong, see below
    bool defer = false;      // ... a forward's in the node's backward
    unsigned fwd_hooks = 0, bwd_hooks = 0;      // M2D_SCAN_TEST_... bits
    int64_t packed() const { return (int64_t)flags | (int64_t)check << 16 | (int64_t)defer << 17 | (int64_t)fwd_hooks << 20 | (int64_t)bwd_hooks << 40; }
    static Options of(int64_t v) { return {(unsigned)(v & 0xffff), (v >> 16 & 1) != 0, (v >> 17 & 1) != 0, (unsigned)(v >> 20 & 0xfffff), (unsigned)(v >> 40)}; }
};

// CTAs of one image wait on one another, and a wait that gives up makes the launch's outputs void.  The call that made
// the launch raises then, and no gradient that such a launch is part of is handed out: a pass without gradients and a
// backward pass wait for their scan before they return (not for the kernels behind it), a forward pass with gradients
// is looked at by its backward, so that a training step waits once.  Not where no CTA waits on another, not during a
// stream capture, where nothing can be waited for, and not where the caller does without (M2D_CHECK_STATUS=0).  What
// the waiting costs is the host's lead over the GPU; us a call, without / with: 1x14x14x320 30.7 / 45, 5x37x53x96
// 71.7 / 87, 1x1024x1024x64 2115 / 2135, training 6x45x31x192 346 / 388, 2x200x336x64 bf16 1467 / 1500.
bool looked_at(const Options& opt, int chain) {
    return opt.check && chain > 1 && at::cuda::currentStreamCaptureStatusMayInitCtx() == at::cuda::CaptureStatus::None;
}
[[noreturn]] void raise_void(const char* what) {
    m2d_take_wait_failure();       // told here, not once more by the next call
    TORCH_CHECK(false, what, ": a wait between CTAs timed out; the results of this call are invalid");
}
// A launch's status word is worth reading only where some launch of the process has failed since `mark`.
void check_status(int64_t mark, const void* status, const char* what) {
    if (mark >= 0 && m2d_wait_failure_mark() == mark) return;
    int word = 0;
    C10_CUDA_CHECK(cudaMemcpy(&word, status, sizeof(word), cudaMemcpyDeviceToHost));
    if (word != 0) raise_void(what);
}

// A failed wait of a launch that no call has looked at (one replayed from a graph, one made without the check, or
// the weight gradient's kernel, whose result is then NaN) surfaces here, like any other asynchronous error.
void check_waits() {
    TORCH_CHECK(!m2d_take_wait_failure(), "wavefront scan: a wait between CTAs of an earlier launch timed out; the results of that launch are invalid");
}

// Whether a call on these makes a node.  An input with a forward-mode tangent goes there too, although there is no
// formula for it: the node refuses it, where a pass without one would drop the tangent and say nothing.
bool wants_grad(std::initializer_list<const Tensor*> inputs) {
    bool grad = false;
    for (const Tensor* t : inputs) grad = grad || (at::GradMode::is_enabled() && t->requires_grad()) || t->_fw_grad(0).defined();
    return grad;
}

struct Dims {
    int64_t B, H, W, E, N, R, K;
};

// What the scan reads, as addresses in tensors that the caller holds; BT, BL, C with their pixel pitch.
struct ScanIn {
    const void *x, *dT, *dL, *AT, *AL, *BT, *BL, *C, *D;
    int64_t pBT, pBL, pC;
};
struct ScanGrads {
    void *x, *dT, *dL, *AT, *AL, *BT, *BL, *C, *D;
    int64_t pBC;         // pixel pitch of the gradients of B and C (0: N)
};

m2d_scan_desc scan_desc(const Dims& s, int dtype, const ScanIn& in, unsigned flags) {
    m2d_scan_desc d{};
    d.struct_bytes = sizeof(d);
    d.dtype = dtype;
    d.B = (int)s.B; d.H = (int)s.H; d.W = (int)s.W; d.E = (int)s.E; d.N = (int)s.N;
    d.flags = flags;
    d.x = in.x; d.dT = in.dT; d.dL = in.dL;
    d.AT = in.AT; d.AL = in.AL;
    d.BT = in.BT; d.BL = in.BL; d.C = in.C;
    d.BT_pitch = in.pBT; d.BL_pitch = in.pBL; d.C_pitch = in.pC;
    d.D = in.D;
    return d;
}

void set_grads(m2d_scan_desc& d, const void* gy, const ScanGrads& g) {
    d.gy = gy;
    d.d_x = g.x; d.d_dT = g.dT; d.d_dL = g.dL;
    d.d_AT = g.AT; d.d_AL = g.AL; d.d_D = g.D;
    d.d_BT = g.BT; d.d_BL = g.BL; d.d_C = g.C;
    d.d_BC_pitch = g.pBC;
}

// Several arrays in one allocation (an allocation or a view of a tensor costs the host about 2 us, a third of a
// launch): byte offsets, 256-byte aligned.
struct Carve {
    int64_t bytes = 0;
    int64_t take(int64_t n) {
        const int64_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    }
};

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

// proj (P, K), dT and dL (P, E) in one buffer.
struct Projected {
    int64_t dT, dL, bytes;       // offsets behind proj
    Projected(const Dims& s, int64_t es) {
        Carve c;
        c.take(s.B * s.H * s.W * s.K * es);
        dT = c.take(s.B * s.H * s.W * s.E * es);
        dL = c.take(s.B * s.H * s.W * s.E * es);
        bytes = c.bytes;
    }
};

// out (rows, n) = a (rows, k) @ w, or += ; `w` is (n, k) if transposed, else (k, n).  Row-major operands are what
// the library calls transposed ones.
void gemm(const Tensor& like, int64_t rows, int64_t n, int64_t k, const void* a, const void* w, bool transposed, bool accumulate, void* out) {
    // fp32: the library's tiles are 64 or 128 columns wide and its time for a few rows is several launches' worth.
    // Library / own, us, events around one call with the L2 flushed (which adds about 10), by E (n = K = 56 ... 120 or E):
    //              x @ Wx^T (n = K)                                          d_x += d_proj @ Wx (n = E)
    //     rows     64        128       192       320      384      512       64        128       192       320      384      512
    //     784     26 / 16   17 / 17   20 / 14   24 / 18  25 / 16  29 / 17   23 / 19   16 / 15   17 / 15   17 / 17  18 / 18  19 / 20
    //     2048    17 / 14   17 / 15   20 / 16   23 / 19  25 / 21  28 / 23   16 / 15   16 / 17   18 / 19   20 / 20  21 / 21  21 / 24
    //     6272    19 / 15   20 / 19   23 / 23   28 / 29  30 / 31  38 / 46   18 / 17   19 / 18   21 / 23   29 / 28  29 / 29  38 / 39
    //     12544   19 / 17   23 / 21   29 / 27   43 / 40  39 / 40  55 / 68   20 / 19   22 / 23   28 / 27   41 / 39  44 / 38  58 / 51
    //     25088   23 / 20   29 / 26   41 / 37   55 / 59  61 / 57  92 / 91   22 / 24   31 / 29   46 / 35   63 / 56  70 / 57  97 / 81
    //     37632                                 74 / 63  80 / 71  98 / 109
    //     100352  46 / 29   58 / 49  114 / 78  165 / 137 187 / 160 278 / 294      46 / 38   69 / 56  127 / 81  215 / 144 262 / 160 367 / 233
    // The first product follows its columns: up to 72 (E = 192) always, up to 96 (E = 384) where there are enough rows.  The
    // second is the library's between 2048 and 12000 rows, where neither gains; below that the own kernel's error, a third of
    // the library's, keeps what it has.
    //
    // A caller that allows TF32 products gets them where the library's are faster then, by rows (TF32 / own, us, E = 64, 192, 512):
    //              x @ Wx^T                          d_x += d_proj @ Wx
    //     784      24 / 16   16 / 14   19 / 18       21 / 16   24 / 14   17 / 20
    //     2100     15 / 15   16 / 17   20 / 23       14 / 14   15 / 19   20 / 32
    //     12544    16 / 17   22 / 27   26 / 68       17 / 19   25 / 27   31 / 51
    //     100352   31 / 30   37 / 79   64 / 294      42 / 37   55 / 80   91 / 233
    //     401408   53 / 68                           94 / 89
    auto own = [&] {
        if (like.scalar_type() != at::kFloat) return false;
        if (rows <= 1024) return true;
        const bool tf32 = at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL) == at::Float32Precision::TF32;
        return tf32 ? accumulate && n <= 64 : n <= 72 || rows <= 2048 || (n <= 96 && rows >= 30000) || (accumulate && rows >= 12000);
    };
    if (own()) {
        const int rc = m2d_rows_gemm_f32(rows, (int)n, (int)k, static_cast<const float*>(a), static_cast<const float*>(w), transposed, accumulate,
                                         static_cast<float*>(out), stream_of(like));
        if (rc == M2D_OK) return;
        // (an x that is not 16-byte aligned, or a contraction too long for the kernel's shared memory)
        TORCH_CHECK(rc == M2D_ERR_PITCH || rc == M2D_ERR_TOO_LARGE, "m2d_rows_gemm_f32 failed: ", m2d_strerror(rc));
    }
    const cudaDataType_t type = like.scalar_type() == at::kFloat ? CUDA_R_32F : CUDA_R_16BF;
    const float alpha = 1.f, beta = accumulate ? 1.f : 0.f;
    // (torch's handle: its stream, its workspace, its TF32 setting)
    const cublasStatus_t rc = cublasGemmEx(at::cuda::getCurrentCUDABlasHandle(), transposed ? CUBLAS_OP_T : CUBLAS_OP_N, CUBLAS_OP_N, (int)n, (int)rows, (int)k, &alpha,
                                           w, type, (int)(transposed ? k : n), a, type, (int)k, &beta, out, type, (int)n, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT);
    TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "cublasGemmEx failed: status ", (int)rc);
}

// What the forward scan wants cleared, if the projection kernel should do it: up to 64 MB, which saves the launch of
// a memset (from there on the memset's higher rate is worth more).
uint64_t clear_in_projection(m2d_scan_desc& d) {
    const uint64_t n = m2d_scan_fwd_cleared(&d);
    if (n > (64u << 20)) return 0;
    d.flags |= M2D_SCAN_WS_CLEARED;
    return n;
}

// `clear_bytes` at `clear` are zeroed by the way.
void project(const Dims& s, const Tensor& x, const BlockParams& p, const Projected& o, char* buf, void* clear = nullptr, uint64_t clear_bytes = 0) {
    gemm(x, s.B * s.H * s.W, s.K, s.E, x.data_ptr(), p.Wx.data_ptr(), true, false, buf);
    m2d_proj_desc d = proj_desc(s, x, p);
    d.proj = buf;
    d.dT = buf + o.dT; d.dL = buf + o.dL;
    d.clear = clear; d.clear_bytes = clear_bytes;
    check(m2d_dtproj_fwd(&d, stream_of(x)), "m2d_dtproj_fwd");
}

ScanIn block_scan_in(const Dims& s, const Tensor& x, const BlockParams& p, const Projected& o, const char* buf) {
    const int64_t es = x.element_size();
    ScanIn in;
    in.x = x.data_ptr(); in.dT = buf + o.dT; in.dL = buf + o.dL;
    in.AT = p.AT_log.data_ptr(); in.AL = p.AL_log.data_ptr(); in.D = p.D.data_ptr();
    in.BT = buf + 2 * s.R * es;
    in.BL = buf + (2 * s.R + s.N) * es;
    in.C = buf + (2 * s.R + 2 * s.N) * es;
    in.pBT = in.pBL = in.pC = s.K;
    return in;
}

unsigned block_flags(const BlockParams& p, const Options& opt) { return M2D_SCAN_A_LOG | (p.f32 ? M2D_SCAN_D_F32 : 0u) | opt.flags; }

// y, given the projections in `buf`; the scan's scratch goes to `ws`.  Where the launch is looked at later: its status
// word, on its way to host memory (the scratch does not live that long).
Tensor forward_scan(const Tensor& x, m2d_scan_desc& d, char* ws, const Tensor& y, const Options& opt) {
    d.y = y.data_ptr();
    d.workspace = ws;
    d.flags |= opt.fwd_hooks;
    const bool look = looked_at(opt, m2d_scan_fwd_chain(&d));
    const int64_t mark = m2d_wait_failure_mark();
    check(m2d_scan_fwd(&d, stream_of(x)), "m2d_scan_fwd");
    if (!look) return Tensor();
    const auto stream = at::cuda::getCurrentCUDAStream(x.get_device());
    const void* const status = ws + m2d_scan_fwd_status_offset(&d);
    if (opt.defer) {
        const Tensor word = at::empty({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
        C10_CUDA_CHECK(cudaMemcpyAsync(word.data_ptr(), status, sizeof(int), cudaMemcpyDeviceToHost, stream));
        // (a graph may be dropped, and the word with it, before the copy has landed)
        at::cuda::CachingHostAllocator_recordEvent(word.data_ptr(), word.storage().data_ptr().get_context(), stream);
        return word;
    }
    {
        const pybind11::gil_scoped_release others_run;       // (forward passes come from Python)
        C10_CUDA_CHECK(cudaStreamSynchronize(stream));
    }
    check_status(mark, status, "m2d_scan_fwd");
    return Tensor();
}

// The backward's scan, and the look at both passes once it is through; its status word has to last until then.
class BackwardScan {
public:
    BackwardScan(const m2d_scan_desc& d, const Tensor& x, const Options& opt, const Tensor& forward_word)
        : forward_(forward_word), own_(looked_at(opt, m2d_scan_bwd_chain(&d))), mark_(m2d_wait_failure_mark()),
          status_(static_cast<const char*>(d.workspace) + m2d_scan_bwd_status_offset(&d)) {
        check(m2d_scan_bwd(&d, stream_of(x)), "m2d_scan_bwd");
        if (own_ || forward_.defined()) done_.record(at::cuda::getCurrentCUDAStream(x.get_device()));
    }
    void finish() {
        if (!own_ && !forward_.defined()) return;
        done_.synchronize();       // (the forward's word was copied on this stream, before)
        if (forward_.defined() && *static_cast<const volatile int*>(forward_.data_ptr()) != 0) raise_void("m2d_scan_fwd");
        if (own_) check_status(mark_, status_, "m2d_scan_bwd");
    }

private:
    Tensor forward_;
    bool own_;
    int64_t mark_;
    const void* status_;
    at::cuda::CUDAEvent done_;
};

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
                          const Tensor& bT, const Tensor& WL, const Tensor& bL, const Tensor& D, bool full, int64_t options) {
        const Options opt = Options::of(options);
        const c10::cuda::CUDAGuard guard(x_.device());
        const Tensor x = x_.contiguous();
        const Dims s = block_dims(x, AT_log, WT);
        const BlockParams p = block_params(x, AT_log, AL_log, Wx, WT, bT, WL, bL, D);
        const Projected o(s, x.element_size());
        const Tensor buf = scratch(o.bytes, x);
        char* const bp = static_cast<char*>(buf.data_ptr());
        m2d_scan_desc d = scan_desc(s, dtype_of(x), block_scan_in(s, x, p, o, bp), block_flags(p, opt));
        d.workspace_bytes = m2d_scan_fwd_workspace(&d);
        const Tensor ws = scratch(d.workspace_bytes, x);
        project(s, x, p, o, bp, ws.data_ptr(), clear_in_projection(d));
        Tensor y = at::empty({s.B, s.H, s.W, s.E}, x.options());
        ctx->saved_data["word"] = forward_scan(x, d, static_cast<char*>(ws.data_ptr()), y, opt);
        // "full" recomputation keeps x and the parameters only
        if (full) ctx->save_for_backward({x, AT_log, AL_log, Wx, WT, bT, WL, bL, D});
        else ctx->save_for_backward({x, AT_log, AL_log, Wx, WT, bT, WL, bL, D, buf, p.Wx});
        ctx->saved_data["options"] = options;
        return y;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const at::NoGradGuard no_grad;
        const variable_list v = ctx->get_saved_variables();
        const Tensor& x = v[0];
        const c10::cuda::CUDAGuard guard(x.device());
        const Options opt = Options::of(ctx->saved_data["options"].toInt());
        check_waits();
        const Dims s = block_dims(x, v[1], v[4]);
        const bool saved = v.size() > 9;
        const BlockParams p = block_params(x, v[1], v[2], saved ? v[10] : v[3], v[4], v[5], v[6], v[7], v[8]);
        const int64_t P = s.B * s.H * s.W, es = x.element_size();
        const Projected o(s, es);
        const bool f32 = x.scalar_type() == at::kFloat;      // the fp32 scan accumulates dB and dC in place, the bf16 one in its workspace
        const Tensor gy = grads[0].to(x.scalar_type()).contiguous();

        // scratch: gradients of the projections' outputs, then what the two library workspaces share
        Carve c;
        const int64_t at_dT = c.take(P * s.E * es), at_dL = c.take(P * s.E * es), at_proj = c.take(P * s.K * es), at_buf = saved ? 0 : c.take(o.bytes);
        m2d_scan_desc sd = scan_desc(s, dtype_of(x), ScanIn{}, block_flags(p, opt) | opt.bwd_hooks | (f32 ? M2D_SCAN_BC_ZEROED : 0u));
        sd.BT_pitch = sd.BL_pitch = sd.C_pitch = sd.d_BC_pitch = s.K;
        m2d_proj_desc pd = proj_desc(s, x, p);
        sd.workspace_bytes = m2d_scan_bwd_workspace(&sd);
        pd.workspace_bytes = m2d_proj_workspace(&pd);
        constexpr int64_t kStatus = 256;       // the scan's status word stays as it is while the projections' scratch takes the place of the rest
        const int64_t at_ws = c.take((int64_t)std::max(sd.workspace_bytes, pd.workspace_bytes + kStatus));
        const Tensor tmp = scratch(c.bytes, x);
        char* const t = static_cast<char*>(tmp.data_ptr());
        char* const d_proj = t + at_proj;
        if (f32) C10_CUDA_CHECK(cudaMemsetAsync(d_proj, 0, P * s.K * es, at::cuda::getCurrentCUDAStream(x.get_device())));
        const char* buf = saved ? static_cast<const char*>(v[9].data_ptr()) : t + at_buf;
        if (!saved) project(s, x, p, o, t + at_buf);

        // the parameters' gradients: A_log's in fp32, the others in the parameters' type; neighbours in one buffer
        // where that is the same
        const bool one = f32 || p.f32;
        const auto fp32 = x.options().dtype(at::kFloat);
        const int64_t en = s.E * s.N, er = s.E * s.R, rest = 2 * er + 2 * s.E + s.K * s.E;
        const Tensor a = at::empty({2 * en + (one ? s.E + rest : 0)}, fp32);
        const Tensor w = one ? a : at::empty({s.E + rest}, x.options());
        int64_t at = 0;
        auto view = [&](const Tensor& from, at::IntArrayRef size) {
            const int64_t cols = size.size() == 2 ? size[1] : 1, off = at;
            at += size[0] * cols;
            return size.size() == 2 ? at::as_strided(from, size, {cols, 1}, off) : at::as_strided(from, size, {1}, off);
        };
        Tensor dAT = view(a, {s.E, s.N}), dAL = view(a, {s.E, s.N});
        if (!one) at = 0;
        Tensor dD = view(w, {s.E}), dWT = view(w, {s.E, s.R}), dWL = view(w, {s.E, s.R}), dbT = view(w, {s.E}), dbL = view(w, {s.E}), dWx = view(w, {s.K, s.E});
        Tensor dx = at::empty({s.B, s.H, s.W, s.E}, x.options());

        ScanGrads g;
        g.x = dx.data_ptr(); g.dT = t + at_dT; g.dL = t + at_dL;
        g.AT = dAT.data_ptr(); g.AL = dAL.data_ptr(); g.D = dD.data_ptr();
        g.BT = d_proj + 2 * s.R * es; g.BL = d_proj + (2 * s.R + s.N) * es; g.C = d_proj + (2 * s.R + 2 * s.N) * es;
        g.pBC = s.K;
        const uint64_t ws_bytes = sd.workspace_bytes;
        sd = scan_desc(s, dtype_of(x), block_scan_in(s, x, p, o, buf), sd.flags);
        set_grads(sd, gy.data_ptr(), g);
        sd.workspace = t + at_ws;
        sd.workspace_bytes = ws_bytes;
        BackwardScan scan(sd, x, opt, ctx->saved_data["word"].toTensor());

        pd.x = x.data_ptr(); pd.proj = buf;
        pd.dT = const_cast<char*>(buf) + o.dT; pd.dL = const_cast<char*>(buf) + o.dL;
        pd.g_dT = g.dT; pd.g_dL = g.dL;
        pd.d_proj = d_proj;
        pd.d_WT = dWT.data_ptr(); pd.d_WL = dWL.data_ptr(); pd.d_bT = dbT.data_ptr(); pd.d_bL = dbL.data_ptr();
        pd.d_Wx = dWx.data_ptr();
        pd.workspace = t + at_ws + kStatus;
        check(m2d_proj_bwd(&pd, stream_of(x)), "m2d_proj_bwd");
        gemm(x, P, s.E, s.K, d_proj, p.Wx.data_ptr(), false, true, g.x);      // d_x = (scan's part) + d_proj @ Wx

        scan.finish();
        auto as = [](const Tensor& t, const Tensor& like) { return t.to(like.scalar_type()); };
        return {dx, as(dAT, v[1]), as(dAL, v[2]), as(dWx, v[3]), dWT, dbT, dWL, dbL, dD, Tensor(), Tensor()};
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
                            const Tensor& WL, const Tensor& bL, const Tensor& D, bool full, bool reverse, bool gelu, bool check_status,
                            unsigned fwd_hooks, unsigned bwd_hooks) {
    if (!block_applies(x, AT_log, AL_log, Wx, WT, bT, WL, bL, D)) return c10::nullopt;
    check_waits();
    const bool grad = wants_grad({&x, &AT_log, &AL_log, &Wx, &WT, &bT, &WL, &bL, &D});
    const Options opt{reverse ? M2D_SCAN_REVERSE : 0u, check_status, grad, fwd_hooks, bwd_hooks};
    if (grad) {
        Tensor y = BlockFn::apply(x, AT_log, AL_log, Wx, WT, bT, WL, bL, D, full, opt.packed());
        return gelu ? at::gelu(y) : y;
    }
    const at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor xc = x.contiguous();
    const Dims s = block_dims(xc, AT_log, WT);
    const BlockParams p = block_params(xc, AT_log, AL_log, Wx, WT, bT, WL, bL, D);
    const Projected o(s, xc.element_size());
    m2d_scan_desc d = scan_desc(s, dtype_of(xc), ScanIn{}, block_flags(p, opt) | (gelu ? M2D_SCAN_GELU_OUT : 0u));
    d.BT_pitch = d.BL_pitch = d.C_pitch = s.K;
    const uint64_t ws_bytes = m2d_scan_fwd_workspace(&d);
    const Tensor buf = scratch(o.bytes + ws_bytes, xc);
    char* const bp = static_cast<char*>(buf.data_ptr());
    project(s, xc, p, o, bp, bp + o.bytes, clear_in_projection(d));
    d = scan_desc(s, dtype_of(xc), block_scan_in(s, xc, p, o, bp), d.flags);
    d.workspace_bytes = ws_bytes;
    Tensor y = at::empty({s.B, s.H, s.W, s.E}, xc.options());
    forward_scan(xc, d, bp + o.bytes, y, opt);
    return y;
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

// The scan's inputs, contiguous where they have to be (`keep` holds the copies).
ScanIn scan_in(const Dims& s, const variable_list& v, variable_list& keep) {
    keep.reserve(9);
    for (size_t k = 0; k < 5; ++k) keep.push_back(v[k].contiguous());
    ScanIn in;
    keep.push_back(pixel_rows(v[5], s, &in.pBT));
    keep.push_back(pixel_rows(v[6], s, &in.pBL));
    keep.push_back(pixel_rows(v[7], s, &in.pC));
    keep.push_back(v[8].contiguous());
    const void** dst[] = {&in.x, &in.dT, &in.dL, &in.AT, &in.AL, &in.BT, &in.BL, &in.C, &in.D};
    for (size_t k = 0; k < 9; ++k) *dst[k] = keep[k].data_ptr();
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
                          const Tensor& BT, const Tensor& BL, const Tensor& C, const Tensor& D, int64_t options) {
        const Options opt = Options::of(options);
        const c10::cuda::CUDAGuard guard(x.device());
        const Dims s = scan_dims(x, AT);
        variable_list keep;
        m2d_scan_desc d = scan_desc(s, dtype_of(x), scan_in(s, {x, dT, dL, AT, AL, BT, BL, C, D}, keep), opt.flags);
        d.workspace_bytes = m2d_scan_fwd_workspace(&d);
        const Tensor ws = scratch(d.workspace_bytes, x);
        Tensor y = at::empty({s.B, s.H, s.W, s.E}, x.options());
        ctx->saved_data["word"] = forward_scan(x, d, static_cast<char*>(ws.data_ptr()), y, opt);
        ctx->save_for_backward({x, dT, dL, AT, AL, BT, BL, C, D});
        ctx->saved_data["options"] = options;
        return y;
    }

    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const at::NoGradGuard no_grad;
        const variable_list v = ctx->get_saved_variables();
        const Tensor& x = v[0];
        const c10::cuda::CUDAGuard guard(x.device());
        const Dims s = scan_dims(x, v[3]);
        const Options opt = Options::of(ctx->saved_data["options"].toInt());
        check_waits();
        const Tensor gy = grads[0].to(x.scalar_type()).contiguous();
        variable_list keep;
        m2d_scan_desc d = scan_desc(s, dtype_of(x), scan_in(s, v, keep), opt.flags | opt.bwd_hooks);
        // one buffer for the three per-pixel gradients of B and C, and one for the per-channel gradients where they
        // share a type: the library then clears each with one memset
        const int64_t n = s.B * s.H * s.W * s.N, en = s.E * s.N;
        const Tensor big = at::empty({3, s.B, s.H, s.W, s.N}, x.options());
        const bool one = !(opt.flags & M2D_SCAN_A_LOG) || x.scalar_type() == at::kFloat;
        const Tensor small = at::empty({2 * en + (one ? s.E : 0)}, one ? x.options() : x.options().dtype(at::kFloat));
        Tensor dAT = at::as_strided(small, {s.E, s.N}, {s.N, 1}, 0), dAL = at::as_strided(small, {s.E, s.N}, {s.N, 1}, en);
        Tensor dD = one ? at::as_strided(small, {s.E}, {1}, 2 * en) : at::empty({s.E}, x.options());
        Tensor dx = at::empty(x.sizes(), x.options()), ddT = at::empty(x.sizes(), x.options()), ddL = at::empty(x.sizes(), x.options());
        char* const bp = static_cast<char*>(big.data_ptr());
        const int64_t es = big.element_size();
        set_grads(d, gy.data_ptr(), {dx.data_ptr(), ddT.data_ptr(), ddL.data_ptr(), dAT.data_ptr(), dAL.data_ptr(), bp, bp + n * es, bp + 2 * n * es, dD.data_ptr(), 0});
        d.workspace_bytes = m2d_scan_bwd_workspace(&d);
        const Tensor ws = scratch(d.workspace_bytes, x);
        d.workspace = ws.data_ptr();
        BackwardScan(d, x, opt, ctx->saved_data["word"].toTensor()).finish();
        return {dx, ddT, ddL, dAT, dAL, big.select(0, 0), big.select(0, 1), big.select(0, 2), dD, Tensor()};
    }
};

c10::optional<Tensor> scan(const Tensor& x, const Tensor& dT, const Tensor& dL, const Tensor& AT, const Tensor& AL, const Tensor& BT, const Tensor& BL,
                           const Tensor& C, const Tensor& D, bool reverse, bool a_log, bool check_status, unsigned fwd_hooks, unsigned bwd_hooks) {
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
    return ScanFn::apply(x, dT, dL, AT, AL, BT, BL, C, D,
                         Options{(reverse ? M2D_SCAN_REVERSE : 0u) | (a_log ? M2D_SCAN_A_LOG : 0u), check_status,
                                 wants_grad({&x, &dT, &dL, &AT, &AL, &BT, &BL, &C, &D}), fwd_hooks, bwd_hooks}.packed());
}

}  // namespace

PYBIND11_MODULE(_entry, m) {
    // check_status: raise where a launch whose CTAs wait on one another went wrong (looked_at); the hooks are test hooks of include/m2d_scan.h
    using pybind11::arg;
    m.def("block", &block, "wavefront_scan_cuda as one autograd node; None where it does not apply", arg("x"), arg("AT_log"), arg("AL_log"),
          arg("x_proj_w"), arg("dt_projT_w"), arg("dt_projT_b"), arg("dt_projL_w"), arg("dt_projL_b"), arg("D"), arg("full"), arg("reverse"),
          arg("gelu"), arg("check_status") = true, arg("fwd_hooks") = 0u, arg("bwd_hooks") = 0u);
    m.def("scan", &scan, "wf_cuda_fn_pr as a native autograd node; None where it does not apply", arg("x"), arg("dT"), arg("dL"), arg("AT"),
          arg("AL"), arg("BT"), arg("BL"), arg("C"), arg("D"), arg("reverse"), arg("a_log"), arg("check_status") = true, arg("fwd_hooks") = 0u,
          arg("bwd_hooks") = 0u);
}
