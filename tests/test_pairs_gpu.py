"""The batch kernels (a warp owns two rows of 16 channels) at the edges of their tiles: an odd last row, bands cut short by
narrow maps, one row per band, ragged channels and states, lists of several images per CTA, both types of the state record."""
import ctypes

import pytest
import torch

from mamba2d_b200 import _lib, scan_bwd, scan_fwd
from mamba2d_b200 import wavefront_cuda as wc
from oracle import cpu, inputs
from helpers import rel_err

pytestmark = pytest.mark.gpu
ORDER = ("x", "dT", "dL", "AT", "AL", "BT", "BL", "C", "D")
SHAPES = [
    (200, 2, 3, 16, 16),      # one pair of rows, the narrowest map
    (150, 7, 3, 20, 16),      # bands of one row: no second row anywhere; ragged second group
    (130, 9, 4, 32, 16),      # bands of two rows, an odd last one
    (600, 3, 6, 48, 12),      # an odd last row in a single band, lists of images
    (140, 33, 5, 34, 16),     # 17 bands, the last of one row
    (700, 7, 7, 40, 16),      # the last stage of a model, lists of images, ragged group
    (90, 17, 19, 66, 5),      # scalar loads, ragged states
    (70, 31, 12, 96, 16),
    (12, 20, 20, 128, 16),    # bf16: few images, the record stays fp32
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("reverse", [False, True])
def test_batch_kernels_against_the_oracle(shape, dt, tol, reverse):
    assert _chains(shape) == (1, 1)
    _check(shape, 1, dt, tol, reverse)


def _chains(shape):
    d = _lib.ScanDesc()
    d.struct_bytes = ctypes.sizeof(d)
    d.B, d.H, d.W, d.E, d.N = shape
    d.BT_pitch = d.BL_pitch = d.C_pitch = shape[4]
    return _lib.lib().m2d_scan_fwd_chain(ctypes.byref(d)), _lib.lib().m2d_scan_bwd_chain(ctypes.byref(d))


def _check(shape, chain, dt, tol, reverse):
    assert _chains(shape)[1] == chain
    inp = inputs.make_inputs(*shape, seed=sum(shape), strided_bc=True)
    inp = {k: v.to(dt).float() for k, v in inp.items()}
    dev = {k: v.cuda().to(dt) for k, v in inp.items()}
    ref = {k: (v.flip(1, 2).contiguous() if v.dim() == 4 else v) for k, v in inp.items()} if reverse else inp

    def back(a):
        return a[:, ::-1, ::-1] if reverse and a.ndim == 4 else a
    y = scan_fwd(*[dev[k] for k in ORDER], reverse=reverse)
    assert rel_err(y.float().cpu().numpy(), back(cpu.forward(ref, "f64"))) < tol
    grads = scan_bwd(*[dev[k] for k in ORDER], dev["gy"], reverse=reverse)
    want = cpu.backward(ref, mode="f64")
    for name, t in zip(cpu.GRAD_NAMES, grads):
        assert rel_err(t.float().cpu().numpy(), back(want[name])) < tol, name


# the same sweeps with the bands of an image in several CTAs, backward only: an image's bands in one round and in two, an odd
# last band, ragged channels
CHAINED = [((40, 56, 56, 64, 16), 3), ((4, 70, 64, 320, 16), 3), ((2, 75, 80, 500, 12), 4), ((9, 61, 60, 130, 5), 3)]


@pytest.mark.parametrize("shape,chain", CHAINED)
@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("reverse", [False, True])
def test_chained_sweeps_against_the_oracle(shape, chain, dt, tol, reverse):
    _check(shape, chain, dt, tol, reverse)


@pytest.mark.parametrize("hook", [_lib.M2D_SCAN_TEST_WITHHOLD, _lib.M2D_SCAN_TEST_WITHHOLD_UP])
def test_waits_of_chained_sweeps_give_up(hook, monkeypatch):
    """A band that hands nothing on: the launch ends, says so, and the next one is right."""
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    shape = (4, 70, 64, 320, 16)
    dev = {k: v.cuda() for k, v in inputs.make_inputs(*shape, seed=3).items()}
    want = scan_bwd(*[dev[k] for k in ORDER], dev["gy"])
    d, keep = wc._make_desc(*[dev[k] for k in ORDER])
    d.flags = hook
    L = _lib.lib()
    d.gy = dev["gy"].data_ptr()
    outs = [torch.zeros_like(t) for t in want]
    for name, t in zip(("d_x", "d_dT", "d_dL", "d_AT", "d_AL", "d_BT", "d_BL", "d_C", "d_D"), outs):
        setattr(d, name, t.data_ptr())
    wc._workspace(d, L.m2d_scan_bwd_workspace(ctypes.byref(d)), dev["x"].device, keep)
    assert L.m2d_scan_bwd(ctypes.byref(d), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert wc._status_word(keep[-1], L.m2d_scan_bwd_status_offset(ctypes.byref(d))) != 0
    assert torch.isnan(outs[1]).any()                        # (d_deltaT: a row that never came reads as NaN)
    again = scan_bwd(*[dev[k] for k in ORDER], dev["gy"])
    for a, b in zip(again, want):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("shape,chain", [((4, 70, 64, 320, 16), 3), ((2, 75, 80, 500, 12), 4),      # chained batch sweeps backward
                                         ((2, 41, 64, 96, 16), 6), ((1, 200, 9, 64, 16), 25)])      # wave kernels, which all take forward
@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
def test_launches_with_fewer_ctas_than_planned(shape, chain, dt, tol, monkeypatch):
    """What a launch does where fewer CTAs are resident than its plan says: half the chain, down to one CTA per image."""
    monkeypatch.setenv("M2D_TEST_HOOKS", "1")
    assert _chains(shape)[0] > 1 and _chains(shape)[1] == chain
    inp = {k: v.to(dt).float() for k, v in inputs.make_inputs(*shape, seed=4).items()}
    dev = {k: v.cuda().to(dt) for k, v in inp.items()}
    L = _lib.lib()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    d, keep = wc._make_desc(*[dev[k] for k in ORDER])
    d.flags = _lib.M2D_SCAN_TEST_SHORT
    y = torch.full_like(dev["x"], float("nan"))
    d.y = y.data_ptr()
    wc._workspace(d, L.m2d_scan_fwd_workspace(ctypes.byref(d)), y.device, keep)
    assert L.m2d_scan_fwd(ctypes.byref(d), stream) == 0
    assert rel_err(y.float().cpu().numpy(), cpu.forward(inp, "f64")) < tol
    want = cpu.backward(inp, mode="f64")
    outs = [torch.full_like(dev[k], float("nan")) for k in ("x", "dT", "dL", "AT", "AL", "BT", "BL", "C", "D")]
    for name, t in zip(("d_x", "d_dT", "d_dL", "d_AT", "d_AL", "d_BT", "d_BL", "d_C", "d_D"), outs):
        setattr(d, name, t.data_ptr())
    d.gy = dev["gy"].data_ptr()
    wc._workspace(d, L.m2d_scan_bwd_workspace(ctypes.byref(d)), y.device, keep)
    assert L.m2d_scan_bwd(ctypes.byref(d), stream) == 0
    torch.cuda.synchronize()
    assert wc._status_word(keep[-1], L.m2d_scan_bwd_status_offset(ctypes.byref(d))) == 0
    got = dict(zip(("d_x", "d_dT", "d_dL", "d_AT", "d_AL", "d_BT", "d_BL", "d_C", "d_D"), outs))
    for name in cpu.GRAD_NAMES:
        assert rel_err(got[name].float().cpu().numpy(), want[name]) < tol, name
