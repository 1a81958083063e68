"""GELU folded into the batch kernel's store, which a warp makes in its next step: rows, bands, images of one CTA's list and
the last cell of all must each get their own value.  Against erf-GELU in fp64 of the y that the kernel without it returns: its
formula is within 2.4e-7 of that over |y| <= 8 (4.5e-7 counting erf's own), and three fp32 roundings at the size of y, 0.6e-7
each, lie between."""
import pytest
import torch

from oracle import inputs
from test_scan_gpu import ORDER, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,E", [(300, 2, 3, 32), (310, 8, 5, 4), (301, 9, 7, 40), (168, 17, 21, 96), (149, 23, 12, 64)])
@pytest.mark.parametrize("reverse", [False, True])
def test_gelu_one_step_late(B, H, W, E, reverse):
    from mamba2d_b200 import scan_fwd
    d = to_dev(inputs.make_inputs(B, H, W, E, 16, seed=B + W), torch.float32)
    args = [d[k] for k in ORDER]
    y = scan_fwd(*args, reverse=reverse).double()
    got = scan_fwd(*args, reverse=reverse, gelu_out=True).double()
    want = 0.5 * y * (1.0 + torch.erf(y * 0.5 ** 0.5))
    assert float(((got - want).abs() - 2e-7 * y.abs()).max()) < 4.5e-7


@pytest.mark.parametrize("B,H,W,E", [(300, 2, 3, 32), (301, 9, 7, 40), (149, 23, 12, 64)])
def test_gelu_one_step_late_bf16(B, H, W, E):
    """The y to compare with is rounded to bf16, whose 8 bits leave 2^-8 of a value (times GELU's slope of 1.13 at most), and so is
    the result, which is no larger than y."""
    from mamba2d_b200 import scan_fwd
    d = to_dev(inputs.make_inputs(B, H, W, E, 16, seed=B + W), torch.bfloat16)
    args = [d[k] for k in ORDER]
    y = scan_fwd(*args).double()
    got = scan_fwd(*args, gelu_out=True).double()
    want = 0.5 * y * (1.0 + torch.erf(y * 0.5 ** 0.5))
    assert float(((got - want).abs() - 2.14 * 2.0 ** -8 * y.abs()).max()) < 4.5e-7
