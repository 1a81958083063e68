"""What the projection kernels do on the side: memory cleared by the forward, and both halves of the backward with one
launch for their sums, against the two calls."""
import ctypes

import pytest
import torch

from mamba2d_b200 import _lib

pytestmark = pytest.mark.gpu


def _desc(dt, P, E, R, t):
    d = _lib.ProjDesc()
    d.struct_bytes, d.dtype, d.P, d.E, d.R, d.N = ctypes.sizeof(d), int(dt == torch.bfloat16), P, E, R, 16
    d.proj_pitch = 2 * R + 48
    for name, v in t.items():
        setattr(d, name, v.data_ptr())
    return d


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("dt,P,E,R", [(torch.float32, 196, 320, 20), (torch.float32, 46900, 64, 4), (torch.bfloat16, 33, 64, 4),
                                      (torch.bfloat16, 9000, 384, 24)])
@pytest.mark.parametrize("pieces", [0, 1, 17, 70001])
def test_forward_clears(dt, P, E, R, pieces):
    K = 2 * R + 48
    z = lambda *s: torch.zeros(*s, dtype=dt, device="cuda")
    t = {"proj": z(P, K), "WT": z(E, R), "WL": z(E, R), "bT": z(E), "bL": z(E), "dT": z(P, E), "dL": z(P, E)}
    d = _desc(dt, P, E, R, t)
    mem = torch.full((pieces * 4 + 8,), -1, dtype=torch.int32, device="cuda")
    d.clear, d.clear_bytes = mem[4:].data_ptr(), pieces * 16
    assert _lib.lib().m2d_dtproj_fwd(ctypes.byref(d), _stream()) == 0
    assert bool((mem[4:4 + pieces * 4] == 0).all()) and bool((mem[:4] == -1).all()) and bool((mem[4 + pieces * 4:] == -1).all())
    assert bool(((t["dL"].float() - 0.6931).abs() < 4e-3).all())


@pytest.mark.parametrize("dt,P,E,R", [(torch.float32, 333, 96, 6), (torch.bfloat16, 784, 384, 24), (torch.bfloat16, 5000, 64, 4), (torch.bfloat16, 77, 36, 3)])
@pytest.mark.parametrize("f32_params", [0, 1])
def test_backward_in_one_call(dt, P, E, R, f32_params):
    K = 2 * R + 48 + (-2 * R) % 4
    g = torch.Generator(device="cuda").manual_seed(P)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda")
    pt = torch.float32 if f32_params else dt
    t = {"x": n(P, E).to(dt), "proj": n(P, K).to(dt), "WT": n(E, R).to(pt), "WL": n(E, R).to(pt), "dT": n(P, E).abs().to(dt),
         "dL": n(P, E).abs().to(dt), "g_dT": n(P, E).to(dt), "g_dL": n(P, E).to(dt)}
    cols = n(P, K).to(dt)
    outs = []
    for both in (False, True):
        o = {"d_proj": cols.clone(), "d_WT": torch.empty(E, R, dtype=pt, device="cuda"), "d_WL": torch.empty(E, R, dtype=pt, device="cuda"),
             "d_bT": torch.empty(E, dtype=pt, device="cuda"), "d_bL": torch.empty(E, dtype=pt, device="cuda"),
             "d_Wx": torch.empty(2 * R + 48, E, dtype=pt, device="cuda")}
        d = _desc(dt, P, E, R, {**t, **o})
        d.proj_pitch, d.flags = K, f32_params
        L = _lib.lib()
        d.workspace_bytes = L.m2d_proj_workspace(ctypes.byref(d))
        ws = torch.empty(d.workspace_bytes, dtype=torch.uint8, device="cuda")
        d.workspace = ws.data_ptr()
        for fn in ((L.m2d_proj_bwd,) if both else (L.m2d_dtproj_bwd, L.m2d_xproj_wgrad)):
            assert fn(ctypes.byref(d), _stream()) == 0
        outs.append(o)
    # (d_r of the CUDA-core kernel is summed by atomic adds below 32 ranks: not the same bits twice)
    for k in outs[0]:
        a, b = (o[k].float() for o in outs)
        assert float((a - b).norm()) <= (1e-6 if dt == torch.float32 else 1e-3) * float(a.norm()), k
