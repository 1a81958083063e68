"""The wave kernels (few images: eight rows per warp, several CTAs per image) at the edges of their tiles:
last bands of one row, maps narrower than a chunk of columns, ragged channels and states, chains that are
shorter than the number of bands, lists of several images, both corners, both I/O types."""
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
    (1, 8, 12, 32, 16),      # one band: no boundary rows
    (1, 9, 5, 16, 16),       # a band of one row; fewer columns than lane rows
    (2, 17, 2, 40, 12),      # two columns
    (1, 16, 3, 6, 4),        # scalar loads, ragged channel group
    (1, 33, 4, 34, 16),      # one chunk of columns
    (3, 24, 13, 18, 5),      # states that are not a multiple of four
    (1, 200, 9, 64, 16),     # 25 bands, a CTA each
    (3, 57, 33, 192, 16),    # 8 bands for 3 CTAs: a CTA comes back for a second and third band while others wait on it
    (2, 140, 26, 128, 12),   # 18 bands for 2 CTAs, ragged states
    (2, 41, 64, 96, 16),
    (60, 17, 7, 64, 16),     # more (image, group) pairs than SMs
    (400, 9, 2, 16, 16),     # lists of several images per CTA
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("reverse", [False, True])
def test_wave_kernels_against_the_oracle(shape, dt, tol, reverse):
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


@pytest.mark.parametrize("shape,chains", [((1, 200, 9, 64, 16), (25, 25)), ((3, 57, 33, 192, 16), (3, 3)), ((2, 140, 26, 128, 12), (2, 2)),
                                          ((400, 9, 2, 16, 16), (1, 1))])
def test_the_shapes_above_get_the_chains_they_are_there_for(shape, chains):
    d = _lib.ScanDesc()
    d.struct_bytes = ctypes.sizeof(d)
    d.B, d.H, d.W, d.E, d.N = shape
    d.BT_pitch = d.BL_pitch = d.C_pitch = shape[4]
    L = _lib.lib()
    assert (L.m2d_scan_fwd_chain(ctypes.byref(d)), L.m2d_scan_bwd_chain(ctypes.byref(d))) == chains


def test_boundary_rows_are_kept_where_a_later_sweep_needs_them():
    """The workspace of a forward list holds two boundary rows in turn, not one per band."""
    d, _ = wc._make_desc(*[torch.zeros(s) for s in ((1, 2, 2, 2),) * 3 + ((2, 2),) * 2 + ((1, 2, 2, 2),) * 3 + ((2,),)])
    L = _lib.lib()
    d.B, d.H, d.W, d.E, d.N = 400, 80, 2, 16, 16
    d.BT_pitch = d.BL_pitch = d.C_pitch = 16
    few = L.m2d_scan_fwd_workspace(ctypes.byref(d))
    d.H = 160
    assert L.m2d_scan_fwd_workspace(ctypes.byref(d)) == few


def _is_wave_backward(shape, dt):
    """Whether the backward is planned for the wave kernels, by the size of its workspace (mamba2d_b200/csrc/m2d_scan_bwd.cu)."""
    B, H, W, E, N = shape
    d = _lib.ScanDesc()
    d.struct_bytes = ctypes.sizeof(d)
    d.dtype = _lib.M2D_F32 if dt == torch.float32 else _lib.M2D_BF16
    d.B, d.H, d.W, d.E, d.N = shape
    d.BT_pitch = d.BL_pitch = d.C_pitch = N

    def up(v):
        return (v + 255) // 256 * 256
    sums = 0 if dt == torch.float32 else up(4 * (3 * B * H * W * N + 2 * E * N + E))
    bands, groups = (H + 7) // 8, (E + 15) // 16
    edge = up(B * ((E + 1) // 2) * (bands if bands > 1 else 0) * W * 32 * 4)
    return _lib.lib().m2d_scan_bwd_workspace(ctypes.byref(d)) == 256 + sums + 2 * edge + up(B * groups * 8 * bands * (W + 7) * 1024)


@pytest.mark.parametrize("shape", [(2, 41, 64, 96, 16), (1, 21, 18, 96, 16), (3, 24, 13, 18, 5)])
@pytest.mark.parametrize("columns", ["neighbours", "apart", "flag"])
@pytest.mark.parametrize("kind", ["f32", "bf16"])
def test_wave_gradients_of_b_and_c_as_columns_of_a_wider_buffer(shape, columns, kind):
    import test_scan_gpu
    assert _is_wave_backward(shape, torch.float32 if kind == "f32" else torch.bfloat16)
    test_scan_gpu.test_gradients_of_b_and_c_as_columns_of_a_wider_buffer(shape, columns, kind)


@pytest.mark.parametrize("shape", [(1, 700, 6, 32, 16), (1, 33, 4, 34, 16)])     # 88 bands that one CTA walks; a band each for five
@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
def test_wave_backward_of_narrow_maps(shape, dt, tol):
    assert _is_wave_backward(shape, dt)
    test_wave_kernels_against_the_oracle(shape, dt, tol, False)
