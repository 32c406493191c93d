"""What users of this package have it do, as cases that can be timed: training steps of a box
convolution block, inference on single frames, the integral image on its own, and the four
functions of the extension interface.

A case is a dict of plain values.  `prepare` makes what a program holds before the call, `run` is
one pass through the public entry points.  Shapes are written N (samples), C (input planes), F
(filters per plane), h, w; a training or inference case has N*C*F output planes of h x w.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "box-convolutions_b200"))
import box_convolution as bc  # noqa: E402

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}

# The box blocks of one 512 x 1024 frame: (count, C, F, frame height / h, frame width / w)
FRAME_BLOCKS = [(8, 32, 4, 8, 8), (3, 16, 4, 4, 4), (1, 8, 2, 2, 2)]


def block(op, name, N, C, F, h, w, dtype="float32", exact=True, normalize=True):
    return {"name": name, "op": op, "N": N, "C": C, "F": F, "h": h, "w": w, "dtype": dtype,
            "exact": exact, "normalize": normalize}


def listed():
    return [
        # fine-tuning on one small crop: nothing but latency, launches and host work
        block("train", "train_crop", 1, 8, 4, 32, 32),
        # the block at 1/8 of a 512 x 1024 frame, one GPU's ordinary batch
        block("train", "train_eighth", 16, 32, 4, 64, 128),
        # the same block on a large batch
        block("train", "train_eighth_batch256", 256, 32, 4, 64, 128),
        # the blocks at 1/4 of a 512 x 1024 frame: planes of 128 x 256
        block("train", "train_quarter_512", 8, 16, 4, 128, 256),
        # 1/4 of a 1024 x 2048 frame: planes of 256 x 512, long-range boxes
        block("train", "train_quarter_1024", 8, 16, 4, 256, 512),
        # feature maps whose sides are no multiple of anything, an odd filter count
        block("train", "train_odd", 6, 20, 3, 93, 157),
        # a module cast to bfloat16
        block("train", "train_bf16", 32, 32, 4, 64, 128, dtype="bfloat16"),
        # one frame through a module in eval mode, whole-pixel boxes: single-frame latency
        block("eval", "eval_eighth", 1, 32, 4, 64, 128, exact=False),
        # the fused inference tail of one block: ReLU, boxes, folded BatchNorm, skip, ReLU
        block("tail", "tail_quarter_512", 1, 16, 4, 128, 256, exact=False),
        # the 12 block tails of one frame replayed as a CUDA graph
        {"name": "frame_graph", "op": "frame", "N": 1, "h": 512, "w": 1024},
        # the integral image on its own, many large planes
        {"name": "integral_1024_planes", "op": "integral", "planes": 1024, "h": 512, "w": 1024},
        # code written against the four functions: integral image, forward, backward, clipping
        block("functions", "functions_mid", 4, 16, 4, 96, 160),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: sizes over their logarithm, odd ones among them."""
    op = rng.choice(["train"] * 10 + ["eval", "tail", "tail", "frame", "integral", "integral", "functions", "functions"])
    if op == "frame":
        # frames are multiples of 8 so that the 1/8-resolution maps exist
        h = 8 * _log_int(rng, 32, 96)
        return {"op": op, "N": rng.choice([1, 1, 2]), "h": h, "w": 8 * _log_int(rng, h // 8, h // 4)}
    if op == "integral":
        h, w = _log_int(rng, 24, 640), _log_int(rng, 24, 1280)
        most = (1 << 29) // (h * w)
        return {"op": op, "planes": _log_int(rng, 1, max(1, min(4096, most))), "h": h, "w": w}
    h, w = _log_int(rng, 20, 280), _log_int(rng, 24, 560)
    if rng.random() < 0.5:                      # half of the maps come from frames with even sides
        h, w = -(-h // 8) * 8, -(-w // 8) * 8
    C, F = _log_int(rng, 4, 64), rng.choice([1, 2, 3, 4, 4, 4, 6, 8])
    most = (1 << 27) // (h * w * C * F) if op == "train" else (1 << 25) // (h * w * C * F)
    N = _log_int(rng, 1, max(1, min(128, most))) if op in ("train", "functions") else rng.choice([1, 1, 1, 2, 4])
    case = block(op, "", N, C, F, h, w, exact=rng.random() < (0.8 if op in ("train", "functions") else 0.4),
                 normalize=rng.random() < 0.85)
    del case["name"]
    if op in ("train", "eval"):
        case["dtype"] = rng.choice(["float32"] * 7 + ["bfloat16"] * 2 + ["float16"])
    return case


def _boxes(rng, C, F, h, w):
    """Pixel-unit boxes (x_min, x_max, y_min, y_max): centres within half the map, half-extents of
    1 pixel up to a quarter of it, no border closer than 1e-3 to a whole pixel."""
    def some(n):
        ch, cw = rng.uniform(-h / 2, h / 2, n), rng.uniform(-w / 2, w / 2, n)
        eh, ew = rng.uniform(1.0, max(1.5, h / 4), n), rng.uniform(1.0, max(1.5, w / 4), n)
        return np.stack([ch - eh, ch + eh, cw - ew, cw + ew]).astype(np.float32)

    b = some(C * F)
    while (bad := (np.abs(b - np.round(b)) < 1e-3).any(axis=0)).any():
        b[:, bad] = some(int(bad.sum()))
    return b.reshape(4, C, F)


def _module(rng, C, F, h, w, dtype=torch.float32, exact=True, normalize=True):
    m = bc.BoxConv2d(C, F, h, w, normalize=normalize)
    m.exact = exact
    b = _boxes(rng, C, F, h, w)
    with torch.no_grad():
        for p, v, rep in zip((m.x_min, m.x_max, m.y_min, m.y_max), b,
                             (m.reparametrization_h, m.reparametrization_h, m.reparametrization_w, m.reparametrization_w)):
            p.copy_(torch.from_numpy(v / np.float32(rep)))
    return m.cuda().to(dtype)


def _frame_layers(case):
    return [(C, F, case["h"] // dh, case["w"] // dw) for n, C, F, dh, dw in FRAME_BLOCKS for _ in range(n)]


def prepare(case, seed):
    rng = np.random.RandomState(seed % (1 << 31))
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, dtype=torch.float32):
        return torch.randn(*shape, device="cuda", generator=gen).to(dtype)

    op = case["op"]
    if op == "integral":
        x = torch.rand(case["planes"], case["h"], case["w"], device="cuda", generator=gen)
        return {"op": op, "x": x}
    if op == "frame":
        layers = _frame_layers(case)
        modules = [_module(rng, C, F, h, w, exact=False).eval() for C, F, h, w in layers]
        inputs = []
        for C, F, h, w in layers:
            inputs += [randn(case["N"], C, h, w), randn(case["N"], C * F, h, w)]

        def tails(*t):
            return [bc.fused_box_block(m, t[2 * i], input_relu=True, residual=t[2 * i + 1], output_relu=True)
                    for i, m in enumerate(modules)]

        return {"op": op, "graph": bc.GraphedForward(tails, *inputs), "modules": modules}
    N, C, F, h, w = (case[k] for k in ("N", "C", "F", "h", "w"))
    dtype = DTYPES[case["dtype"]]
    state = {"op": op, "x": randn(N, C, h, w, dtype=dtype)}
    if op == "functions":
        m = _module(rng, C, F, h, w, dtype, case["exact"], case["normalize"])
        state["stored"] = [p.detach().clone() for p in (m.x_min, m.x_max, m.y_min, m.y_max)]
        state["pixels"] = [p.clone() for p in m.get_actual_parameters()]
        state["rep"] = (m.reparametrization_h, m.reparametrization_w)
        state["flags"] = (case["normalize"], case["exact"])
        state["max"] = (h, w)
        state["g"] = randn(N, C * F, h, w, dtype=dtype)
        return state
    state["m"] = _module(rng, C, F, h, w, dtype, case["exact"], case["normalize"])
    if op == "train":
        state["x"].requires_grad_()
        state["g"] = randn(N, C * F, h, w, dtype=dtype)
        state["m"].train()
    else:
        state["m"].eval()
    if op == "tail":
        state["scale"] = torch.rand(C * F, device="cuda", generator=gen) + 0.5
        state["shift"] = torch.rand(C * F, device="cuda", generator=gen) - 0.5
        state["residual"] = randn(N, C * F, h, w)
    return state


def run(state):
    op = state["op"]
    if op == "train":
        m, x = state["m"], state["x"]
        m.zero_grad(set_to_none=True)
        x.grad = None
        y = m(x)
        y.backward(state["g"])
        ps = (m.x_min, m.x_max, m.y_min, m.y_max)
        return [y, x.grad, [p.grad for p in ps], list(ps)]
    if op == "eval":
        with torch.no_grad():
            return state["m"](state["x"])
    if op == "tail":
        return bc.fused_box_block(state["m"], state["x"], input_relu=True, scale=state["scale"], shift=state["shift"],
                                  residual=state["residual"], output_relu=True)
    if op == "frame":
        return state["graph"].replay()
    if op == "integral":
        return bc.integral_image(state["x"])
    pixels, (rep_h, rep_w) = state["pixels"], state["rep"]
    normalize, exact = state["flags"]
    bc.clip_parameters(*state["stored"], rep_h, rep_w, *state["max"], exact)
    integ = bc.integral_image(state["x"])
    out = bc.box_convolution_forward(integ, *pixels, normalize, exact)
    grads = bc.box_convolution_backward(integ, *pixels, state["g"], out, rep_h, rep_w, normalize, exact,
                                        True, True, True, True, True)
    return [integ, out, grads, state["stored"]]


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: a 2-D prefix sum takes 2 additions
    a pixel; an output (or the grad-input share) of one box 16 taps, i.e. about 30 operations, the
    four parameter gradients about as many again."""
    op = case["op"]
    if op == "integral":
        n, h, w = case["planes"], case["h"], case["w"]
        return {"bytes": 4 * n * (h * w + (h + 1) * (w + 1)), "flops": 2 * n * h * w}
    if op == "frame":
        total = {"bytes": 0, "flops": 0}
        for C, F, h, w in _frame_layers(case):
            E = case["N"] * C * h * w
            total["bytes"] += 4 * E * (1 + 2 * F)
            total["flops"] += E * (2 + 32 * F)
        return total
    N, C, F, h, w = (case[k] for k in ("N", "C", "F", "h", "w"))
    E, size = N * C * h * w, 4 if case["dtype"] == "float32" else 2
    if op == "train":       # x, output, grad_output, x again, grad_input
        return {"bytes": size * E * (2 * F + 3), "flops": E * (2 + 92 * F)}
    if op == "eval":
        return {"bytes": size * E * (1 + F), "flops": E * (2 + 30 * F)}
    if op == "tail":        # x, residual, output
        return {"bytes": size * E * (1 + 2 * F), "flops": E * (2 + 34 * F)}
    integ = N * C * (h + 1) * (w + 1)
    return {"bytes": size * (2 * E + integ + 2 * F * E), "flops": E * (2 + 92 * F)}


def tolerance(case):
    """Sums of up to h*w 32-bit values, taken as differences of prefix sums; 16-bit tensors are
    rounded once when they are stored."""
    if case.get("dtype", "float32") == "bfloat16":
        return {"rel": 1e-2}
    if case.get("dtype", "float32") == "float16":
        return {"rel": 2e-3}
    return {"rel": 1e-5, "max": 1e-3}
