"""The dt projections on the tensor cores (csrc/proj_mma.cuh) against fp64: sizes on both sides of the rule
that picks them, last tiles of pixels, channel chunks and rank tiles that are not full, every shipped width, and the
ranks around the last one whose fp32 products fit into shared memory (48 to 53, by the width)."""
import pytest
import torch
import torch.nn.functional as F

from mamba2d_b200 import wavefront_cuda as wc
from helpers import rel_err

pytestmark = pytest.mark.gpu
WIDTHS = [(64, 4), (72, 7), (96, 6), (128, 8), (136, 8), (192, 12), (200, 16), (320, 20), (384, 24), (512, 32), (576, 36), (640, 39),
          (512, 48), (232, 49), (640, 53), (256, 64), (640, 64)]


def _inputs(P, E, R, dt):
    g = torch.Generator(device="cuda").manual_seed(P + E)
    n = lambda *s: torch.randn(*s, generator=g, device="cuda")
    K = 2 * R + 48 + (-2 * R) % 4
    W, b = [n(E, R) * R ** -0.5 for _ in range(2)], [n(E) - 3.0 for _ in range(2)]
    return n(1, 1, P, K).to(dt), [t.to(dt) for t in W], [t.to(dt) for t in b], [n(1, 1, P, E).to(dt) for _ in range(2)]


@pytest.mark.parametrize("E,R", WIDTHS)
@pytest.mark.parametrize("dt,P", [(torch.bfloat16, 131), (torch.bfloat16, 4797), (torch.float32, 0)])
def test_dt_projections_and_their_backward(E, R, dt, P):
    P = P or 3000000 // E + 45                       # fp32: just enough elements for the tensor cores
    proj, W, b, g = _inputs(P, E, R, dt)
    dT, dL = wc._dtproj_fwd(proj, W[0], b[0], W[1], b[1], 16)
    want = [F.softplus(proj[..., k * R:(k + 1) * R].double() @ W[k].double().t() + b[k].double()) for k in range(2)]
    tol = 2e-6 if dt == torch.float32 else 4e-3
    for got, ref in zip((dT, dL), want):
        assert float(((got.double() - ref).abs() / (ref.abs() + 1e-3)).max()) < (2e-5 if dt == torch.float32 else 8e-3)
        assert rel_err(got.float().cpu().numpy(), ref.cpu().numpy()) < tol
    zeros = torch.zeros(1, 1, P, 16, dtype=dt, device="cuda")
    d_proj, dWT, dbT, dWL, dbL = wc._dtproj_bwd(g[0], g[1], dT, dL, proj, W[0], W[1], zeros, zeros, zeros)
    btol = 1e-5 if dt == torch.float32 else 8e-3
    for k, (dW, db) in enumerate(((dWT, dbT), (dWL, dbL))):
        s = g[k].double() * -torch.expm1(-(dT, dL)[k].double())
        s = s.reshape(P, E)
        assert rel_err(dW.float().cpu().numpy(), (s.t() @ proj.reshape(P, -1)[:, k * R:(k + 1) * R].double()).cpu().numpy()) < btol
        assert rel_err(db.float().cpu().numpy(), s.sum(0).cpu().numpy()) < btol
        assert rel_err(d_proj.reshape(P, -1)[:, k * R:(k + 1) * R].float().cpu().numpy(), (s @ W[k].double()).cpu().numpy()) < btol
