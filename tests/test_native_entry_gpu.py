"""The native entry points (csrc/torch_entry.cpp) against the op-by-op path they replace in eager mode:
same outputs and gradients for every type combination they take, and the fallback for the rest."""
import pytest
import torch

from mamba2d_b200 import _lib
from mamba2d_b200 import wavefront_cuda as wc
from oracle import inputs
from helpers import rel_err

pytestmark = pytest.mark.gpu
NAMES = ("AT_log", "AL_log", "x_proj_w", "dt_projT_w", "dt_projT_b", "dt_projL_w", "dt_projL_b", "D")


def _run(x, ws, gy, **kw):
    leaves = [t.clone().requires_grad_(True) for t in (x, *ws)]
    y = wc.wavefront_scan_cuda(*leaves, **kw)
    return [y.detach(), *torch.autograd.grad(y, leaves, gy)]


@pytest.mark.parametrize("xdt,wdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("shape", [(2, 7, 5, 64), (1, 21, 18, 96)])       # one CTA per image; several
@pytest.mark.parametrize("kw", [{}, {"recomp": "full", "scan_start": "BR", "act_out": "gelu"}])
def test_block_equals_the_op_by_op_path(xdt, wdt, shape, kw, monkeypatch):
    E = shape[-1]
    w = inputs.make_module_params(E, 16, seed=5)
    ws = [w[k].cuda() if k.endswith("_log") else w[k].cuda().to(wdt) for k in NAMES]
    g = torch.Generator().manual_seed(1)
    x, gy = torch.randn(*shape, generator=g).cuda().to(xdt), torch.randn(*shape, generator=g).cuda().to(xdt)
    assert wc._native(x) is _lib.entry()
    got = _run(x, ws, gy, **kw)
    with torch.no_grad():
        y_inf = wc.wavefront_scan_cuda(x, *ws, **kw)
    monkeypatch.setattr(wc, "_native", lambda t: None)
    want = _run(x, ws, gy, **kw)
    tol = 1e-5 if xdt == torch.float32 else 2e-2
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert rel_err(a.float().cpu().numpy(), b.float().cpu().numpy()) < tol
    assert rel_err(y_inf.float().cpu().numpy(), want[0].float().cpu().numpy()) < tol


@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2)])
def test_scan_equals_the_op_by_op_path(dt, tol, monkeypatch):
    inp = inputs.make_inputs(2, 9, 13, 40, 12, seed=3, strided_bc=True)
    args = [inp[k].cuda().to(dt) for k in ("x", "dT", "dL", "AT", "AL", "BT", "BL", "C", "D")]
    gy = inp["gy"].cuda().to(dt)

    def run():
        leaves = [t.detach().requires_grad_(True) for t in args]
        y = wc.wf_cuda_fn_pr.apply(*leaves)
        return [y.detach(), *torch.autograd.grad(y, leaves, gy)]
    got = run()
    monkeypatch.setattr(wc, "_native", lambda t: None)
    for a, b in zip(got, run()):
        assert rel_err(a.float().cpu().numpy(), b.float().cpu().numpy()) < tol


@pytest.mark.parametrize("E", [96, 128, 192])
def test_a_caller_that_allows_tf32_products_gets_them(E, monkeypatch):
    """Many rows: the x projection and what comes back through it, each by itself, show TF32's rounding (2^-11 of a factor) where it
    is allowed and fp32's where it is not."""
    w = inputs.make_module_params(E, 16, seed=5)
    ws = [w[k].cuda() for k in NAMES]
    g = torch.Generator().manual_seed(1)
    x, gy = torch.randn(14, 30, 30, E, generator=g).cuda().requires_grad_(True), torch.randn(14, 30, 30, E, generator=g).cuda()

    def both(fwd, bwd):
        monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", fwd)
        y = wc.wavefront_scan_cuda(x, *ws)
        monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", bwd)
        return y.detach(), torch.autograd.grad(y, x, gy)[0]

    def far(a, b):
        return float((a.double() - b.double()).norm() / b.double().norm())
    y, dx = both(False, False)
    y_f, _ = both(True, False)
    y_b, dx_b = both(False, True)
    assert torch.equal(y_b, y)
    assert 5e-6 < far(y_f, y) < 5e-3
    assert 5e-6 < far(dx_b, dx) < 5e-3


def test_what_the_native_path_does_not_take_goes_op_by_op():
    w = inputs.make_module_params(36, 16, seed=5)                          # 36 channels: dt rank 20 is beyond the kernels' range
    w["dt_projT_w"], w["dt_projL_w"] = torch.randn(36, 20) * 0.2, torch.randn(36, 20) * 0.2
    w["x_proj_w"] = torch.randn(2 * 20 + 48, 36) * 0.1
    ws = [w[k].cuda() for k in NAMES]
    x = torch.randn(1, 4, 5, 36).cuda()
    assert _lib.entry().block(x, *ws, False, False, False) is None
    assert wc.wavefront_scan_cuda(x, *ws).shape == x.shape
    assert _lib.lib().m2d_take_wait_failure() == 0


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("act", [None, "gelu"])
def test_forward_mode_tangents_are_refused(grad, act):
    """There is no forward-mode formula: a call says so and does not return an output without a tangent."""
    import torch.autograd.forward_ad as fw
    w = inputs.make_module_params(64, 16, seed=5)
    ws = [w[k].cuda() for k in NAMES]
    x = torch.randn(2, 7, 5, 64, device="cuda").requires_grad_(grad)
    with fw.dual_level():
        dual = fw.make_dual(x, torch.ones_like(x))
        with pytest.raises(RuntimeError, match="jvp"):
            wc.wavefront_scan_cuda(dual, *ws, act_out=act)
        with torch.no_grad(), pytest.raises(RuntimeError, match="jvp"):
            wc.wavefront_scan_cuda(dual, *ws, act_out=act)
        tangent = fw.make_dual(ws[7], torch.ones_like(ws[7]))                # of a parameter (D)
        with pytest.raises(RuntimeError, match="jvp"):
            wc.wavefront_scan_cuda(x.detach(), *ws[:7], tangent, act_out=act)
