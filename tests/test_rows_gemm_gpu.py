"""fp32 products of pixel rows with a small matrix (csrc/m2d_gemm.cu) against fp64: both kernels, row tiles, column
chunks and steps of the contraction that are not full, with and without accumulation."""
import ctypes

import pytest
import torch

from mamba2d_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transposed,accumulate", [(1, 0), (0, 1)])
@pytest.mark.parametrize("rows,n,k", [(1, 4, 4), (15, 60, 96), (196, 88, 320), (2047, 132, 640), (2500, 8, 12), (4801, 56, 64), (9805, 60, 96),
                                      (19073, 16, 36), (20001, 64, 128), (30011, 36, 68), (40037, 44, 100), (9000, 148, 600)])
def test_rows_gemm(rows, n, k, transposed, accumulate):
    g = torch.Generator(device="cuda").manual_seed(rows + n + k)
    a = torch.randn(rows, k, generator=g, device="cuda")
    w = torch.randn(*((n, k) if transposed else (k, n)), generator=g, device="cuda")
    out = torch.randn(rows, n, generator=g, device="cuda")
    want = a.double() @ (w.t() if transposed else w).double() + (out.double() if accumulate else 0.0)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = _lib.lib().m2d_rows_gemm_f32(ctypes.c_int64(rows), n, k, ptr(a), ptr(w), transposed, accumulate, ptr(out),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    scale = (k + 1) ** 0.5                           # of one result
    assert float((out.double() - want).abs().max()) < 2e-6 * scale
    assert float((out.double() - want).norm() / want.norm()) < 3e-7


@pytest.mark.parametrize("rows,n,k", [(12000, 96, 60), (12001, 128, 64), (12543, 192, 72), (13000, 320, 88), (12289, 512, 112), (12017, 576, 120)])
def test_rows_gemm_adds_to_wide_rows(rows, n, k):
    """d_x += d_proj @ Wx at the widths and row counts that no longer go to the GEMM library."""
    test_rows_gemm(rows, n, k, 0, 1)


@pytest.mark.parametrize("rows,n,k", [(30000, 76, 224), (30011, 88, 320), (40001, 96, 384)])
def test_rows_gemm_of_many_rows_and_more_columns(rows, n, k):
    """The x projection at the column and row counts around its line to the GEMM library."""
    test_rows_gemm(rows, n, k, 1, 0)


@pytest.mark.parametrize("transposed,accumulate", [(1, 0), (0, 1)])
@pytest.mark.parametrize("rows,n,k", [(40, 60, 68), (5000, 12, 20), (20011, 64, 56), (12017, 112, 64)])
def test_rows_gemm_of_values_that_bf16_parts_cannot_hold(rows, n, k, transposed, accumulate):
    """Infinities, NaNs and floats that round to infinity in bf16, in either factor and in what is added to: each result is
    the infinity, the NaN or the number that fp64 gives (rounded to fp32: a product beyond its range is infinite)."""
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    inf, nan, most = float("inf"), float("nan"), 3.4e38
    a = torch.randn(rows, k, generator=g, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda")
    w[:, k // 2:] = w[:, k // 2:].bfloat16().float()          # exact in one part: the others are zeros
    w[1] = 0.0
    w[3:9] *= 0.1                                             # no two large terms meet that only an fp32 sum would take
    a[:, k - 1] *= 0.1                                        # out of range on its way, by the order of its terms
    for i, v in enumerate((inf, -inf, nan, most, -most)):
        a[7 * i, 3 * i] = v
        a[rows - 1 - i, k - 1 - i] = v
    w[5, 2], w[6, k - 7], w[8, k - 1] = inf, -inf, -most
    out = torch.randn(rows, n, generator=g, device="cuda")
    out[2, 3], out[rows - 3, 9], out[4, 4] = inf, -inf, nan
    want = (a.double() @ w.double().t() + (out.double() if accumulate else 0.0)).float()
    m = w if transposed else w.t().contiguous()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = _lib.lib().m2d_rows_gemm_f32(ctypes.c_int64(rows), n, k, ptr(a), ptr(m), transposed, accumulate, ptr(out),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out.isinf(), want.isinf()) and torch.equal(out[out.isinf()], want[want.isinf()])
    ok = want.isfinite()
    small = ok & (want.abs() < 1e30)
    assert int(small.sum()) > 0.5 * rows * n
    assert float((out.double() - want.double())[small].abs().max()) < 2e-6 * (k + 1) ** 0.5      # of one result, as above
    large = ok & ~small                                       # at most three terms are large: a rounding of fp32 (6e-8) each
    size = a.double().abs() @ w.double().abs().t()
    assert int(large.sum()) > 0 and float(((out.double() - want.double()).abs() / size)[large].max()) < 1.8e-7
