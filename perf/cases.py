"""The calls whose speed this package is judged by: the 2-D selective scan as models use it.

Two entry points: ``wavefront_scan_cuda`` (what a block calls: projections and scan, from the activation
and the block's own fp32 parameters) and ``wf_cuda_fn_pr`` (the scan alone, its nine inputs given).  A
"train" case is one forward and one backward pass with every gradient; an "infer" case is a forward
pass without gradients.  Channel counts, map sizes and the batch of 128 are the shipped models' four
stages; the batch-2 map of 200x336 and the batch-1 map of 1024x1024 are detection fine-tuning and
high-resolution inference; odd sizes stand for images of any size given to a convolutional backbone.
"""
import math

import torch
import torch.nn.functional as F

from mamba2d_b200 import wavefront_cuda as wf

N = 16          # states per channel, the same in every shipped model

# Stage widths of the shipped models, by the downsampling of their stage relative to the first one.
WIDTHS = {1: (64, 96), 2: (128, 192), 4: (320, 384), 8: (512, 576)}


def listed():
    def case(name, call, kind, B, H, W, E, dtype, **more):
        return dict(name=name, call=call, kind=kind, B=B, H=H, W=W, E=E, dtype=dtype,
                    **{"recomp": "partial", "start": "TL", "act": "", **more})

    return [
        # one image, third stage: what a single-image request waits for
        case("infer_1x14x14x320_f32", "block", "infer", 1, 14, 14, 320, "f32"),
        # a few images of an odd size, bottom-right block, activation folded in
        case("infer_5x37x53x96_f32_br", "block", "infer", 5, 37, 53, 96, "f32", start="BR", act="gelu"),
        # batched classification, first stage (the largest activation of the model)
        case("infer_128x56x56x64_bf16", "block", "infer", 128, 56, 56, 64, "bf16", act="gelu"),
        # high-resolution map, one image
        case("infer_1x1024x1024x64_f32", "block", "infer", 1, 1024, 1024, 64, "f32"),
        # fine-tuning with a small batch, launch-bound
        case("train_4x14x14x384_bf16", "block", "train", 4, 14, 14, 384, "bf16"),
        # ragged training map, fp32
        case("train_6x45x31x192_f32", "block", "train", 6, 45, 31, 192, "f32"),
        # the four stages of a training step, batch 128 (bf16 activations as under autocast, or fp32)
        case("train_128x56x56x64_f32", "block", "train", 128, 56, 56, 64, "f32"),
        case("train_128x28x28x128_bf16", "block", "train", 128, 28, 28, 128, "bf16"),
        case("train_128x14x14x320_bf16_br", "block", "train", 128, 14, 14, 320, "bf16", start="BR"),
        case("train_128x7x7x512_f32_full", "block", "train", 128, 7, 7, 512, "f32", recomp="full"),
        # detection fine-tuning: two large images
        case("train_2x200x336x64_bf16", "block", "train", 2, 200, 336, 64, "bf16"),
        # the scan alone, forward and backward, at the shape the kernels are quoted on
        case("scan_128x56x56x64_f32", "scan", "train", 128, 56, 56, 64, "f32"),
    ]


def draw(rng):
    """Any stage width, batch and map of the ranges above, odd sizes among them."""
    kind = rng.choice(("infer", "train"))
    call = "scan" if rng.random() < 0.2 else "block"
    level = rng.choice((1, 2, 4, 8))
    E = rng.choice(WIDTHS[level])
    # mostly maps of classification images of 160 ... 512 pixels, sometimes large images
    big = rng.random() < 0.25
    lo, hi = (math.log(112), math.log(1024 if kind == "infer" else 336)) if big else (math.log(40), math.log(128))

    def side():
        return max(5, int(math.exp(rng.uniform(lo, hi)) / level))

    H = side()
    W = max(5, min(int(math.exp(hi)) // level, int(H * math.exp(rng.uniform(-0.6, 0.6)))))
    cap = (1 << 25 if kind == "infer" else 3 << 23) // (H * W * E)          # elements of the largest listed cases
    if cap < 1:
        H, W, cap = max(5, H // 2), max(5, W // 2), 1
    B = max(1, min(128, cap, int(math.exp(rng.uniform(0, math.log(160)))) if not big else rng.choice((1, 2, 3, 4, 8))))
    act = rng.choice(("", "gelu")) if (kind == "infer" and call == "block") else ""
    recomp = rng.choice(("partial", "partial", "full")) if (kind == "train" and call == "block") else "partial"
    return dict(call=call, kind=kind, B=B, H=H, W=W, E=E, dtype=rng.choice(("f32", "bf16")), recomp=recomp,
                start=rng.choice(("TL", "BR")), act=act)


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def _rank(case):
    return math.ceil(case["E"] / 16)


def prepare(case, seed):
    B, H, W, E, dt = case["B"], case["H"], case["W"], case["E"], _dtype(case)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo

    train = case["kind"] == "train"
    x = normal(B, H, W, E).to(dt)
    gy = normal(B, H, W, E).to(dt) if train else None
    if case["call"] == "scan":
        delta = [F.softplus(normal(B, H, W, E) * 0.5 - 2.0).to(dt) for _ in range(2)]
        A = [(-torch.exp(uniform(0.0, math.log(16.0), E, N))).to(dt) for _ in range(2)]
        BC = [(normal(B, H, W, N) * N ** -0.5).to(dt) for _ in range(3)]
        args = [x, *delta, *A, *BC, normal(E).to(dt)]
    else:
        # a block's own parameters as it initialises them, a little way into training
        R = _rank(case)
        n = torch.arange(1, N + 1, dtype=torch.float32, device="cuda").repeat(E, 1)
        A_log = [torch.log(n) + 0.05 * normal(E, N) for _ in range(2)]
        x_proj = uniform(-1.0, 1.0, 2 * R + 3 * N, E) * E ** -0.5
        dt_w = [uniform(-1.0, 1.0, E, R) * R ** -0.5 for _ in range(2)]
        step = torch.exp(uniform(math.log(1e-3), math.log(0.1), E)).clamp(min=1e-4)
        bias = step + torch.log(-torch.expm1(-step))
        D = 1.0 + 0.1 * normal(E)
        args = [x, *A_log, x_proj, dt_w[0], bias.clone(), dt_w[1], bias.clone(), D]
    if train:
        args = [a.requires_grad_(True) for a in args]
    return {"case": dict(case), "args": args, "gy": gy}


def run(state):
    case, args, gy = state["case"], state["args"], state["gy"]
    if gy is None:
        with torch.no_grad():
            return _call(case, args)
    y = _call(case, args)
    return (y, *torch.autograd.grad(y, args, gy))


def _call(case, args):
    if case["call"] == "scan":
        return wf.wf_cuda_fn_pr.apply(*args, case["start"] == "BR")
    return wf.wavefront_scan_cuda(*args, recomp=case["recomp"], scan_start=case["start"], act_out=case["act"] or None)


def work(case):
    """Inputs once, outputs once.  Per element and state the forward does 14 operations (two gates, the
    input term, the recurrence, the readout), the backward 40; the projections are 2 per multiply-add and
    their backward is twice their forward."""
    E, R, s = case["E"], _rank(case), 4 if case["dtype"] == "f32" else 2
    P = case["B"] * case["H"] * case["W"]
    train = case["kind"] == "train"
    state_ops = P * E * N * (54 if train else 14)
    if case["call"] == "scan":
        inputs = s * (P * (3 * E + 3 * N) + 2 * E * N + E)
        grads = inputs + s * P * E if train else 0          # the nine gradients, and the upstream one
        return {"bytes": inputs + s * P * E + grads, "flops": state_ops}
    K = 2 * R + 3 * N
    weights = 4 * (2 * E * N + K * E + 2 * E * R + 3 * E)
    proj_ops = 2 * P * E * (K + 2 * R)
    return {"bytes": s * P * E * (4 if train else 2) + weights * (2 if train else 1),
            "flops": state_ops + proj_ops * (3 if train else 1)}


def tolerance(case):
    # fp32: sums of up to 4e5 terms in another order; bf16: inputs, projections and results rounded to 8 bits
    return {"rel": 2e-5, "max": 2e-3} if case["dtype"] == "f32" else {"rel": 1e-2, "max": 0.4}
