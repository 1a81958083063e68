"""Chained forwards that hand their boundary rows over in pairs of columns (few images, four channels per lane, a chain whose
start-up is three tenths of the steps or more, the line of fp32; bf16 has a lower one): maps that end inside a pair or a
chunk, a last band of one row, a CTA that comes back for a later band, ragged channels.  The bounds are those of the other
tests of these kernels."""
import ctypes

import pytest
import torch

from mamba2d_b200 import _lib, scan_fwd
from oracle import cpu, inputs
from helpers import rel_err

pytestmark = pytest.mark.gpu
ORDER = ("x", "dT", "dL", "AT", "AL", "BT", "BL", "C", "D")
SHAPES = [(1, 136, 90, 512, 16), (1, 137, 93, 500, 16), (1, 200, 200, 320, 16), (4, 129, 81, 126, 7)]


def _edge_columns(shape, dtype):
    d = _lib.ScanDesc()
    d.struct_bytes, d.dtype = ctypes.sizeof(d), dtype
    d.B, d.H, d.W, d.E, d.N = shape
    d.BT_pitch = d.BL_pitch = d.C_pitch = shape[4]
    return _lib.lib().m2d_scan_fwd_edge_columns(ctypes.byref(d))


@pytest.mark.parametrize("dtype", [_lib.M2D_F32, _lib.M2D_BF16])
def test_the_shapes_here_are_handed_over_in_pairs(dtype):
    assert [_edge_columns(s, dtype) for s in SHAPES] == [2] * len(SHAPES)
    assert _edge_columns((1, 400, 400, 384, 16), dtype) == 4               # (a start-up of 7 % of the steps)
    assert _edge_columns((2, 200, 336, 64, 16), dtype) == 4                # (two channels per lane)
    assert _edge_columns((128, 56, 56, 64, 16), dtype) == 0                # (a CTA per image and 32 channels)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt,tol", [(torch.float32, 1e-4), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("reverse", [False, True])
def test_boundary_rows_in_pairs_against_the_oracle(shape, dt, tol, reverse):
    inp = inputs.make_inputs(*shape, seed=sum(shape), strided_bc=True)
    inp["D"] = torch.zeros_like(inp["D"])                # the skip term cannot mask an error in the recurrence
    inp = {k: v.to(dt).float() for k, v in inp.items()}
    ref = {k: (v.flip(1, 2).contiguous() if v.dim() == 4 else v) for k, v in inp.items()} if reverse else inp
    want = cpu.forward(ref, "f64")
    y = scan_fwd(*[inp[k].cuda().to(dt) for k in ORDER], reverse=reverse)
    assert rel_err(y.float().cpu().numpy(), want[:, ::-1, ::-1] if reverse else want) < tol
