"""The bounded waits of the kernels give up cleanly, and one diverged image does not poison others.

Row-warps of a CTA and, on large maps with few images, CTAs that share an image wait on one another.
Every such wait has a limit; when one runs out the kernel still returns normally and leaves a
nonzero status word in its workspace.  A test hook (descriptor flag M2D_SCAN_TEST_WITHHOLD, honoured
only under M2D_TEST_HOOKS=1) makes exactly that happen: one producer never publishes its progress and
the limits are a few hundred tries.  Nothing here faults or hangs the GPU: a wait runs out and the
kernel ends.

The native entry points (csrc/torch_entry.cpp) read the word before they return: of a pass without gradients, or of
both passes in the backward, so that no gradient of a launch that went wrong is handed out.  A launch they were told
not to look at is reported by the next call."""
import ctypes

import pytest
import torch

from mamba2d_b200 import _lib
from mamba2d_b200 import wavefront_cuda as wc
from oracle import cpu, inputs
from helpers import rel_err

pytestmark = pytest.mark.gpu
ORDER = ("x", "dT", "dL", "AT", "AL", "BT", "BL", "C", "D")


def _launch_fwd(dev, flags):
    L = _lib.lib()
    d, keep = wc._make_desc(*[dev[k] for k in ORDER])
    d.flags = flags
    y = torch.empty_like(dev["x"])
    d.y = y.data_ptr()
    wc._workspace(d, L.m2d_scan_fwd_workspace(ctypes.byref(d)), dev["x"].device, keep)
    rc = L.m2d_scan_fwd(ctypes.byref(d), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return rc, d, keep[-1], y


def test_a_withheld_counter_makes_the_wait_give_up(monkeypatch):
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    inp = inputs.make_inputs(1, 96, 64, 64, 16, seed=3)      # one image on a large map: several CTAs share it
    dev = {k: v.cuda() for k, v in inp.items()}
    L = _lib.lib()
    d0, _ = wc._make_desc(*[dev[k] for k in ORDER])
    assert L.m2d_scan_fwd_chain(ctypes.byref(d0)) > 1
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    rc, d, ws, _ = _launch_fwd(dev, _lib.M2D_SCAN_TEST_WITHHOLD)
    stop.record()
    assert rc == 0
    torch.cuda.synchronize()
    assert start.elapsed_time(stop) < 2000.0                 # it returned promptly
    off = L.m2d_scan_fwd_status_offset(ctypes.byref(d))
    assert off >= 0 and wc._status_word(ws, off) != 0
    with pytest.raises(RuntimeError, match="timed out"):
        wc._check_status("fwd", d, ws)
    # the context is fine and the next, ordinary launch is correct
    rc, d, ws, y = _launch_fwd(dev, 0)
    assert rc == 0
    torch.cuda.synchronize()
    assert wc._status_word(ws, off) == 0
    assert rel_err(y.cpu().numpy(), cpu.forward(inp, "f64")) < 1e-4


def _large_map():
    inp = inputs.make_inputs(1, 96, 64, 64, 16, seed=3)
    return inp, {k: v.cuda() for k, v in inp.items()}


def _grads(y, leaves, gy):
    return torch.autograd.grad(y, leaves, gy)


def _scan(dev, grad, check=True, fwd=0, bwd=0):
    leaves = [dev[k].detach().requires_grad_(grad) for k in ORDER]
    return _lib.entry().scan(*leaves, False, False, check, fwd, bwd), leaves


def _block(dev, grad, check=True, fwd=0, bwd=0):
    w = inputs.make_module_params(64, 16, seed=5)
    names = ("AT_log", "AL_log", "x_proj_w", "dt_projT_w", "dt_projT_b", "dt_projL_w", "dt_projL_b", "D")
    leaves = [t.detach().requires_grad_(grad) for t in (dev["x"], *(w[k].cuda() for k in names))]
    return _lib.entry().block(*leaves, False, False, False, check, fwd, bwd), leaves


DOWN, UP, REPORT = _lib.M2D_SCAN_TEST_WITHHOLD, _lib.M2D_SCAN_TEST_WITHHOLD_UP, _lib.M2D_SCAN_TEST_REPORT


@pytest.mark.parametrize("call", [_scan, _block])
def test_a_native_forward_raises_in_the_call_that_went_wrong(call, monkeypatch):
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    inp, dev = _large_map()
    want, _ = call(dev, False)
    with pytest.raises(RuntimeError, match="m2d_scan_fwd: a wait between CTAs timed out"):
        call(dev, False, fwd=DOWN | REPORT)
    with torch.no_grad(), pytest.raises(RuntimeError, match="m2d_scan_fwd: a wait between CTAs timed out"):
        call(dev, True, fwd=DOWN | REPORT)
    y, _ = call(dev, False)                                  # told once: the next call knows nothing of it
    assert torch.equal(y, want)
    assert _lib.lib().m2d_take_wait_failure() == 0


@pytest.mark.parametrize("call", [_scan, _block])
def test_no_gradient_of_a_forward_that_went_wrong_is_handed_out(call, monkeypatch):
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    inp, dev = _large_map()
    y, leaves = call(dev, True, fwd=DOWN | REPORT)
    assert torch.isnan(y).any()                              # a row that never came reads as NaN
    assert _lib.lib().m2d_take_wait_failure() == 1           # (or the next call would tell, before the backward does)
    with pytest.raises(RuntimeError, match="m2d_scan_fwd: a wait between CTAs timed out"):
        _grads(y, leaves, dev["gy"])
    y, leaves = call(dev, True)
    assert all(torch.isfinite(g).all() for g in _grads(y, leaves, dev["gy"]))
    y, leaves = call(dev, True)
    del y, leaves                                            # a graph that is dropped with its word on the way
    assert _lib.lib().m2d_take_wait_failure() == 0


@pytest.mark.parametrize("call", [_scan, _block])
@pytest.mark.parametrize("hook", [DOWN, UP])                 # the recompute sweep, the adjoint sweep
def test_a_native_backward_raises_before_its_gradients_are_used(call, hook, monkeypatch):
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    inp, dev = _large_map()
    y, leaves = call(dev, True, bwd=hook | REPORT)
    with pytest.raises(RuntimeError, match="m2d_scan_bwd: a wait between CTAs timed out"):
        _grads(y, leaves, dev["gy"])
    y, leaves = call(dev, True)
    assert all(torch.isfinite(g).all() for g in _grads(y, leaves, dev["gy"]))
    assert _lib.lib().m2d_take_wait_failure() == 0


@pytest.mark.parametrize("call", [_scan, _block])
def test_an_unchecked_failure_is_reported_by_the_next_call(call, monkeypatch):
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    inp, dev = _large_map()
    y, leaves = call(dev, True, check=False, bwd=UP | REPORT)
    torch.cuda.synchronize()
    y_bad, _ = call(dev, False, check=False, fwd=DOWN | REPORT)
    torch.cuda.synchronize()
    assert torch.isnan(y_bad).any()                          # a row that never came reads as NaN
    with pytest.raises(RuntimeError, match="earlier launch timed out"):
        _grads(y, leaves, dev["gy"])                         # the backward looks, too
    y, leaves = call(dev, True, check=False, bwd=UP | REPORT)
    _grads(y, leaves, dev["gy"])
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="earlier launch timed out"):
        call(dev, False)
    assert torch.isfinite(call(dev, False)[0]).all()
    assert _lib.lib().m2d_take_wait_failure() == 0


@pytest.mark.parametrize("hook", [DOWN, UP])
def test_the_backwards_waits_give_up(hook, monkeypatch):
    """Through the C interface: the status word, and what the sweep before the withheld row had finished."""
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    inp, dev = _large_map()
    L = _lib.lib()
    want = wc.scan_bwd(*[dev[k] for k in ORDER], dev["gy"])
    d, keep = wc._make_desc(*[dev[k] for k in ORDER])
    d.flags = hook
    assert L.m2d_scan_bwd_chain(ctypes.byref(d)) > 1
    d.gy = dev["gy"].data_ptr()
    outs = [torch.zeros_like(t) for t in want]
    for name, t in zip(("d_x", "d_dT", "d_dL", "d_AT", "d_AL", "d_BT", "d_BL", "d_C", "d_D"), outs):
        setattr(d, name, t.data_ptr())
    wc._workspace(d, L.m2d_scan_bwd_workspace(ctypes.byref(d)), dev["x"].device, keep)
    assert L.m2d_scan_bwd(ctypes.byref(d), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    off = L.m2d_scan_bwd_status_offset(ctypes.byref(d))
    assert wc._status_word(keep[-1], off) != 0
    with pytest.raises(RuntimeError, match="gradients are invalid"):
        wc._check_status("bwd", d, keep[-1])
    assert torch.isnan(outs[1]).any()                        # (d_deltaT, which needs the states and their adjoints)
    last = outs[1][:, 88:]                                   # the last band: complete where only the way up was cut
    if hook == UP:
        assert float((last - want[1][:, 88:]).abs().max()) <= 1e-6 * float(want[1].abs().max())
    else:
        assert torch.isnan(last).any()


def test_the_hook_is_refused_without_the_environment_variable(monkeypatch):
    monkeypatch.delenv("M2D_TEST_HOOKS", raising=False)
    inp = inputs.make_inputs(1, 96, 64, 64, 16, seed=3)
    dev = {k: v.cuda() for k, v in inp.items()}
    rc, _, _, _ = _launch_fwd(dev, _lib.M2D_SCAN_TEST_WITHHOLD)
    assert rc == -10


@pytest.mark.parametrize("shape", [(300, 6, 5, 64, 16), (400, 12, 9, 32, 16)])   # more (image, group) units than resident CTAs
def test_a_diverged_image_leaves_the_others_alone(shape):
    """Image 1 gets infinite inputs.  A CTA walks several images one after the other and carries state
    in registers and shared memory; nothing of a diverged image may leak into the next one (missing
    neighbours are taken as zero, never multiplied by a zero gate)."""
    from mamba2d_b200 import scan_bwd, scan_fwd
    inp = inputs.make_inputs(*shape, seed=8)
    dev = {k: v.cuda() for k, v in inp.items()}
    a = [dev[k] for k in ORDER]
    y0 = scan_fwd(*a)
    g0 = scan_bwd(*a, dev["gy"])
    bad = {k: v.clone() for k, v in dev.items()}
    bad["x"][1] = float("inf")
    bad["gy"][1] = float("inf")
    b = [bad[k] for k in ORDER]
    y1 = scan_fwd(*b)
    g1 = scan_bwd(*b, bad["gy"])
    torch.cuda.synchronize()
    keep = [i for i in range(shape[0]) if i != 1]
    assert torch.equal(y0[keep], y1[keep])
    for idx in (0, 1, 2, 5, 6, 7):       # the per-pixel gradients (the batch sums d_AT, d_AL, d_D include image 1)
        assert torch.isfinite(g1[idx][keep]).all()
        assert float((g0[idx][keep] - g1[idx][keep]).abs().max()) <= 1e-6 * float(g0[idx].abs().max())


def test_a_waiting_call_lets_other_threads_run():
    """The wait for the scan holds no interpreter lock: a thread gets on with its work meanwhile."""
    import threading
    import time
    x = torch.randn(1, 2048, 1024, 64, device="cuda")
    w = inputs.make_module_params(64, 16, seed=5)
    ws = [w[k].cuda() for k in ("AT_log", "AL_log", "x_proj_w", "dt_projT_w", "dt_projT_b", "dt_projL_w", "dt_projL_b", "D")]
    wc.wavefront_scan_cuda(x, *ws)
    torch.cuda.synchronize()
    marks, stop = [], threading.Event()

    def other():
        while not stop.is_set():
            marks.append(time.perf_counter())
    t = threading.Thread(target=other)
    t.start()
    spans = []
    for _ in range(5):
        a = time.perf_counter()
        wc.wavefront_scan_cuda(x, *ws)                       # milliseconds, nearly all of it waiting
        spans.append((a, time.perf_counter()))
    stop.set()
    t.join()
    assert sum(any(a + 0.2 * (b - a) < m < b - 0.2 * (b - a) for m in marks) for a, b in spans) >= 3


def _mid_sized():
    """A batch whose backward runs the batch sweeps with the bands of an image in several CTAs."""
    shape = (24, 57, 50, 64, 16)
    inp = inputs.make_inputs(*shape, seed=6)
    dev = {k: v.cuda() for k, v in inp.items()}
    d, _ = wc._make_desc(*[dev[k] for k in ORDER])
    L = _lib.lib()
    assert L.m2d_scan_bwd_chain(ctypes.byref(d)) == 3
    record, rows = 24 * 57 * 50 * 4 * 1024, 24 * 8 * 50 * 4 * 1024
    assert L.m2d_scan_bwd_workspace(ctypes.byref(d)) < record + 2 * rows + 4096      # (the wave kernels' record is wider: 64 rows of 57 columns)
    return dev


@pytest.mark.parametrize("call", [_scan, _block])
@pytest.mark.parametrize("hook", [DOWN, UP])
def test_a_chained_batch_backward_raises_before_its_gradients_are_used(call, hook, monkeypatch):
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    dev = _mid_sized()
    y, leaves = call(dev, True)
    want = _grads(y, leaves, dev["gy"])
    y, leaves = call(dev, True, bwd=hook | REPORT)
    with pytest.raises(RuntimeError, match="m2d_scan_bwd: a wait between CTAs timed out"):
        _grads(y, leaves, dev["gy"])
    y, leaves = call(dev, True)
    for a, b in zip(_grads(y, leaves, dev["gy"]), want):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
    assert _lib.lib().m2d_take_wait_failure() == 0


@pytest.mark.parametrize("call", [_scan, _block])
def test_a_chained_batch_backward_in_a_graph(call):
    dev = _mid_sized()
    y, leaves = call(dev, True)
    want = [y.detach().clone(), *(_grads(y, leaves, dev["gy"]))]

    def run():
        entry, own = _lib.entry(), [t.detach().requires_grad_() for t in leaves]         # (leaves that no other stream has used)
        y = entry.scan(*own, False, False, True, 0, 0) if call is _scan else entry.block(*own, False, False, False, True, 0, 0)
        return [y.detach(), *_grads(y, own, dev["gy"])]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    for _ in range(2):
        for t in got:
            t.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
    assert _lib.lib().m2d_take_wait_failure() == 0
