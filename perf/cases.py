"""Workloads by which the speed of this package is measured, through its public entry points.

The path is what a model with NVFP4 lattice weights does: forward passes (`F.linear` under `bl.compute`), training
steps (forward, input and weight gradients, the lattice update from the gradient hooks), the optimizer on its own, and
the conversion of dense weights to NVFP4 and back. `listed()` names the workloads, `draw()` gives further ones from the
same ranges, `prepare()` builds what a program holds before the call, `run()` is one pass.

A case is a dict of plain values:

    kind       forward | train | step | convert
    block      layer (q, k, v from one input; o; gate and up from one input -> SwiGLU -> down), mlp (gate, up -> SwiGLU
               -> down) or linear (one projection hidden -> inter)
    tokens     rows of the activations
    hidden, kv, inter   widths of the block (kv: output features of k and v)
    dtype      of activations and gradients
    compute    the compute policy: fp4 and fp4_all (the NVIDIA operand recipe), exact, or a recipe of backend.FP4_RECIPES
    direction, phase_bits   of the lattice update
    shard      the weights are 1 / shard of the rows of the block's (row shards of a model split over GPUs)
    blocks     how many blocks the optimizer holds (kind step)
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import bitlattice_b200 as bl
from bitlattice_b200.parallel import shared_input_linears

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed() -> list:
    decoder = dict(block="layer", hidden=4096, kv=1024, inter=12288, dtype="bf16")          # the 8B-class decoder layer
    mlp = dict(block="mlp", hidden=1024, kv=0, inter=3072, dtype="bf16")                    # the small SwiGLU block
    colnorm = dict(direction="colnorm", phase_bits=4, shard=1)
    sign = dict(direction="sign", phase_bits=4, shard=1)
    return [
        # serving, one step of 16 sequences: launches and the reading of the weights count
        dict(name="decode_16", kind="forward", tokens=16, compute="fp4", **decoder),
        # serving, a prompt of odd length, four-over-six activations
        dict(name="prefill_1903", kind="forward", tokens=1903, compute="4over6", **decoder),
        # training of the smallest layer of the test configurations: host work and launches
        dict(name="train_linear_256", kind="train", block="linear", hidden=1024, kv=0, inter=1024, dtype="bf16",
             tokens=256, compute="fp4_all", **sign),
        # the SwiGLU block of the test configurations
        dict(name="train_mlp_8k", kind="train", tokens=8192, compute="fp4_all", **mlp, **sign),
        # a decoder layer on one sequence, and on the 16 x 4096 tokens of the benchmark
        dict(name="train_layer_4k", kind="train", tokens=4096, compute="fp4_all", **decoder, **colnorm),
        dict(name="train_layer_64k", kind="train", tokens=65536, compute="fp4_all", **decoder, **colnorm),
        # a wide projection in fp16 on a batch that fills no tile
        dict(name="train_wide_4999", kind="train", block="linear", hidden=5120, kv=0, inter=25600, dtype="fp16",
             tokens=4999, compute="fp4_all", direction="raw", phase_bits=2, shard=1),
        # the 128-point rotation recipe: MS-EDEN gradients, four-over-six activations
        dict(name="train_quartet2_16k", kind="train", block="linear", hidden=4096, kv=0, inter=4096, dtype="bf16",
             tokens=16384, compute="quartet2", **colnorm),
        # the default policy: dequantized weights and dense products
        dict(name="train_exact_1k", kind="train", tokens=1024, compute="exact", **mlp, **sign),
        # the optimizer on its own: whole matrices, and the shards of an 8-way split with fp32 gradients
        dict(name="step_3_layers", kind="step", blocks=3, **decoder, **colnorm),
        dict(name="step_shards", kind="step", blocks=3, block="layer", hidden=4096, kv=1024, inter=12288, dtype="fp32",
             direction="sign", phase_bits=2, shard=8),
        # loading a dense checkpoint and exporting it
        dict(name="convert_12288", kind="convert", block="linear", hidden=4096, kv=0, inter=12288, dtype="fp32"),
    ]


# ---------------------------------------------------------------------------------------------------- drawn cases

def _log_int(rng, lo: int, hi: int, multiple: int = 1) -> int:
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(multiple, round(v / multiple) * multiple))


def draw(rng) -> dict:
    kind = rng.choice(["forward", "forward", "train", "train", "train", "step", "convert"])
    block = rng.choice(["layer", "mlp", "linear"])
    rotated = kind == "train" and rng.random() < 0.25
    hidden = _log_int(rng, 512, 5120, 128)
    inter = _log_int(rng, 1024, 12288, 128 if rotated else 32)
    case = dict(kind=kind, block=block, hidden=hidden, inter=inter,
                kv=max(128, hidden // 4 // 128 * 128) if block == "layer" else 0)
    if kind == "convert":
        case.update(block="linear", kv=0, dtype=rng.choice(["fp32", "bf16"]))
        return case
    if kind == "forward":
        case.update(tokens=_log_int(rng, 1, 16384), dtype=rng.choice(["bf16", "bf16", "fp16"]),
                    compute=rng.choice(["fp4", "fp4", "4over6"]))
        return case
    case.update(direction=rng.choice(["colnorm", "colnorm", "sign", "raw"]), phase_bits=rng.choice([2, 4, 4]))
    if kind == "step":
        case.update(blocks=rng.choice([1, 2, 3]), shard=rng.choice([1, 2, 4, 8]), dtype=rng.choice(["bf16", "bf16", "fp32"]))
        return case
    case.update(tokens=_log_int(rng, 64, 16384), dtype=rng.choice(["bf16", "bf16", "fp16"]), shard=1)
    case["compute"] = (rng.choice(["quartet2", "quartet2", "quartet2_4o6"]) if rotated
                       else rng.choice(["fp4_all", "fp4_all", "fp4_all", "4over6"]))
    return case


# ---------------------------------------------------------------------------------------------------- shapes, bounds

def _shapes(case) -> list:
    """(name, out_features, in_features) of a block's projections."""
    h, kv, i, s = case["hidden"], case["kv"], case["inter"], case.get("shard", 1)
    block = {"layer": [("q", h, h), ("k", kv, h), ("v", kv, h), ("o", h, h), ("gate", i, h), ("up", i, h), ("down", h, i)],
             "mlp": [("gate", i, h), ("up", i, h), ("down", h, i)],
             "linear": [("w", i, h)]}[case["block"]]
    if s == 1:
        return block
    return [(name, max(32, n // s // 32 * 32), k) for name, n, k in block]


def _weights(case) -> int:
    return sum(n * k for _, n, k in _shapes(case)) * case.get("blocks", 1)


def _phase_container(bits: int) -> int:
    return bits if bits <= 2 else 4 if bits <= 4 else 8


def work(case) -> dict:
    w, m = _weights(case), case.get("tokens", 0)
    size = torch.empty((), dtype=DTYPES[case["dtype"]]).element_size()
    update = w * (2 * 0.5625 + 2 * _phase_container(case.get("phase_bits", 0)) / 8)         # codes, scales, phase: r + w
    if case["kind"] == "convert":
        return {"bytes": w * (size + 2 * 0.5625 + 2), "flops": 0}                           # dense in, NVFP4, bf16 out
    if case["kind"] == "step":
        return {"bytes": w * size + update, "flops": 0}
    h, kv, i = case["hidden"], case["kv"], case["inter"]
    ins = {"layer": 3 * h, "mlp": h, "linear": h}[case["block"]]                            # widths of inputs, outputs
    outs = {"layer": 3 * h + 2 * kv, "mlp": h, "linear": i}[case["block"]]
    if case["kind"] == "forward":
        return {"bytes": m * (ins + outs) * size + 0.5625 * w, "flops": 2.0 * m * w}
    return {"bytes": 2 * m * (ins + outs) * size + update, "flops": 6.0 * m * w}


def tolerance(case):
    # The optimizer and the conversion fix the order of every sum: their bytes are reproducible. The products may sum in
    # another order. With every product formed in 64 bits instead, forward passes moved by up to 1.4e-5 (single elements
    # by one step of the 16-bit output, or of a re-quantized activation), training steps by up to 3.4e-4 (single
    # elements by 0.045: a gradient code that fell on the other side of its draw) and 1.1e-4 of the updated bytes.
    if case["kind"] in ("step", "convert"):
        return "exact"
    if case["kind"] == "forward":
        return {"rel": 6e-5, "max": 0.03}
    return {"rel": 1.4e-3, "max": 0.2, "differ": 5e-4}


# ---------------------------------------------------------------------------------------------------- state, one pass

def _generator(seed: int):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, shape, std, dtype):
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(dtype)


def _parameters(case, gen) -> list:
    """The blocks' weights, N(0, 0.02^2), quantized to NVFP4."""
    logical = DTYPES[case["dtype"]]                          # the gradients of a weight have its logical type
    out = []
    for _ in range(case.get("blocks", 1)):
        for _, n, k in _shapes(case):
            dense = torch.randn(n, k, device="cuda", generator=gen) * 0.02
            out.append(torch.nn.Parameter(bl.LatticeTensor.from_float(dense, "nvfp4", method="rtn", dtype=logical)))
    return out


def prepare(case, seed) -> dict:
    gen = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    kind, h, kv, i = case["kind"], case["hidden"], case["kv"], case["inter"]
    s = dict(case=case, passes=0, seed=seed)
    if kind == "convert":
        s["dense"] = _normal(gen, (i, h), 0.02, dtype)
        return s
    s["params"] = ps = _parameters(case, gen)
    if kind in ("train", "step"):
        # hooks apply the updates during backward; a decoder layer's go out as one batch beside the backward pass
        hooks = {} if kind == "step" else dict(fused_backward=True)
        if kind == "train" and case["block"] == "layer":
            hooks.update(overlap=True, hook_batch=len(ps), hook_flush="reader")
        s["opt"] = bl.Lattice(ps, lr=3e-3, direction=case["direction"], phase_bits=case["phase_bits"], rounding="sr",
                              scale_rule="fit", trust=0.1, trust_lr=0.0, seed=1234, **hooks)
    if kind == "step":
        # gradients of successive steps point both ways, so that the weights stay where training keeps them
        first = [_normal(gen, (p.shape[0], p.shape[1]), 1e-3, dtype) for p in ps]
        s["grads"] = (first, [-g for g in first])
        return s
    m = case["tokens"]
    ins = {"layer": (h, h, h), "mlp": (h,), "linear": (h,)}[case["block"]]
    outs = {"layer": (h, kv, kv, h, h), "mlp": (h,), "linear": (i,)}[case["block"]]
    s["x"] = [_normal(gen, (m, k), 1.0, dtype) for k in ins]
    if kind == "train":
        first = [_normal(gen, (m, n), 1e-2, dtype) for n in outs]
        s["gy"] = (first, [-g for g in first])
    return s


def _forward(case, x: list, ps: list) -> list:
    if case["block"] == "linear":
        return [F.linear(x[0], ps[0])]
    ys = []
    if case["block"] == "layer":
        ys += shared_input_linears(x[0], ps[0:3])
        ys.append(F.linear(x[1], ps[3]))
    gate, up = shared_input_linears(x[-1], ps[-3:-1])
    ys.append(F.linear(bl.swiglu(gate, up), ps[-1]))
    return ys


def _stored(ps: list, opt) -> list:
    return [(p.packed, p.scales.view(torch.uint8), opt.state[p]["phase"]) for p in ps]


def run(s):
    case, n = s["case"], s["passes"]
    s["passes"] = n + 1
    kind = case["kind"]
    if kind == "convert":
        w = bl.LatticeTensor.from_float(s["dense"], "nvfp4", method="rtn", dtype=torch.bfloat16)
        return w.packed, w.scales.view(torch.uint8), w.global_scale, w.dequantize()
    if kind == "step":
        for p, g in zip(s["params"], s["grads"][n % 2]):
            p.grad = g
        s["opt"].step()
        return _stored(s["params"], s["opt"])
    if kind == "forward":
        with torch.no_grad(), bl.compute(case["compute"]):
            return _forward(case, [x.detach() for x in s["x"]], s["params"])
    bl.backend.set_sr_seed(1 + (s["seed"] % 1000) * 100003 + 64 * n)     # the rounding draws of this step, reproducible
    xs = [x.detach().requires_grad_(True) for x in s["x"]]
    with bl.compute(case["compute"]):
        ys = _forward(case, xs, s["params"])
        torch.autograd.backward(ys, s["gy"][n % 2])
    s["opt"].step()
    return [y.detach() for y in ys], [x.grad for x in xs], _stored(s["params"], s["opt"])
