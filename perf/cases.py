"""Performance cases of mixfp4_b200: what a program that uses the framework has it do, through the public
entry points, with sizes of the decoder shapes that the benchmark and the tests use.

    listed()               the fixed cases
    draw(rng)              one more case of the same ranges
    prepare(case, seed)    inputs, packed weights, captured decode step: what the program holds before a call
    run(state)             one pass
    work(case)             bytes and floating-point operations that a pass cannot do without
    tolerance(case)        how far another correct implementation may be from the result

A case's "kind" says which path it takes:

    decode    one token step of `batch` sequences through the linears of `layers` decoder layers (q/k/v and
              gate/up grouped, o and down single, every launch chained to the one before), recorded once in a
              CUDA graph and replayed on new activations: how a decode loop runs the linears
    linear    one `mixfp4_linear` call on new activations, weight in the layout the layers keep; `transform`:
              the rotation folded into the weight, which the call applies to x; `activation`: the format
              region of the W4A4 forward, "" for bf16 activations
    block     the seven linears of one decoder layer called one after the other on `m` prompt tokens
    convert   `MixFP4Linear.from_linear`: rotate, quantize and lay out a dense weight for the kernels
    fake      `quant_mixfp4_granularity`: the quantize-dequantize of a tensor with a format region
"""

from __future__ import annotations

import math

import torch

import mixfp4_b200 as mx

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # one sequence generating tokens: a quarter of an 8B model's decoder layers, 1 GB of packed weights
        {"name": "decode_batch1", "kind": "decode", "layers": 8, "batch": 1, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # the same step for a small, odd number of sequences
        {"name": "decode_batch12", "kind": "decode", "layers": 8, "batch": 12, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # a server's batch: more sequences than the matrix-vector kernels take
        {"name": "decode_batch48", "kind": "decode", "layers": 8, "batch": 48, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # the smallest call: one k or v projection of one token, called eagerly
        {"name": "linear_kv_m1", "kind": "linear", "m": 1, "n": 1024, "k": 4096, "transform": "", "activation": "", "out": "bf16"},
        # a short prompt with a ragged number of tokens through one layer
        {"name": "block_m777", "kind": "block", "m": 777, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # an ordinary prefill of the square projection
        {"name": "linear_q_m4096", "kind": "linear", "m": 4096, "n": 4096, "k": 4096, "transform": "", "activation": "", "out": "bf16"},
        # the largest: a 70B-shaped gate or up projection on a long prompt
        {"name": "linear_70b_m4096", "kind": "linear", "m": 4096, "n": 28672, "k": 8192, "transform": "", "activation": "", "out": "bf16"},
        # a rotated projection: the activations take the weight's block Hadamard on the way in
        {"name": "linear_h128_m2048", "kind": "linear", "m": 2048, "n": 4096, "k": 4096, "transform": "H128", "activation": "", "out": "bf16"},
        # quantized activations: rotate, quantize-dequantize, multiply
        {"name": "linear_w4a4_m2048", "kind": "linear", "m": 2048, "n": 4096, "k": 14336, "transform": "H128", "activation": "oracle16",
         "out": "bf16"},
        # loading a model: one dense gate or up projection becomes a packed layer
        {"name": "convert_gate", "kind": "convert", "n": 14336, "k": 4096, "dtype": "bf16", "transform": "H128"},
        # studying a format: quantize-dequantize of a weight with one format per 16 values
        {"name": "fake_oracle16", "kind": "fake", "n": 4096, "k": 4096, "dtype": "bf16", "region": "oracle16"},
        # the same for float32 weights, a format per 8 x 64 region and ragged edges
        {"name": "fake_n8k64_f32", "kind": "fake", "n": 3001, "k": 4100, "dtype": "f32", "region": "n8k64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _to(value, multiple):
    return max(multiple, value // multiple * multiple)


def draw(rng):
    kind = rng.choice(["decode", "decode", "linear", "linear", "linear", "block", "convert", "fake"])
    if kind in ("decode", "block"):
        hidden = _to(_log(rng, 1024, 8192), 128)
        shape = {"hidden": hidden, "kv": _to(hidden // rng.choice([1, 4, 8]), 64), "ffn": _to(int(hidden * rng.uniform(2.5, 4.0)), 64)}
    if kind == "decode":
        return {"kind": kind, "layers": rng.choice([1, 2, 4]) if hidden <= 4096 else 1, "batch": _log(rng, 1, 128), **shape}
    if kind == "block":
        case = {"kind": kind, "m": _log(rng, 130, 3000), **shape}
        while work(case)["flops"] > 1.5e12:
            case["m"] //= 2
        return case
    n, k = _log(rng, 256, 28672), _log(rng, 512, 14336)
    if rng.random() < 0.75:          # most layers have round sizes; the rest take any
        n, k = _to(n, 64), _to(k, 128)
    if kind == "linear":
        transform = rng.choice(["", "", "H128", "H64"])
        activation = rng.choice(["", "", "", "oracle16"])
        m = _log(rng, 1, 8192)
        while 2.0 * m * n * k > 1.5e12 and m > 1:
            m //= 2
        return {"kind": kind, "m": m, "n": n, "k": k, "transform": transform, "activation": activation, "out": rng.choice(["bf16", "bf16", "f32"])}
    dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
    while n * k > 6e7:               # a projection of the larger models at most
        n //= 2
    if kind == "convert":
        return {"kind": kind, "n": n, "k": k, "dtype": dtype, "transform": rng.choice(["", "H128"])}
    return {"kind": kind, "n": n, "k": k, "dtype": dtype, "region": rng.choice(["oracle16", "oracle16", "all_e2m1", "n8k64", "k64_row"])}


# ------------------------------------------------------------------------------------------ inputs
def _weight(n, k, gen, dtype=torch.bfloat16):
    """Heavy-tailed weight, Student-t with 4 degrees of freedom times 0.02 (the benchmark's)."""
    z = torch.randn((n, k), generator=gen, device="cuda")
    chi = torch.zeros((n, k), device="cuda")
    for _ in range(4):
        d = torch.randn((n, k), generator=gen, device="cuda")
        chi.addcmul_(d, d)
    return (z / torch.sqrt(chi / 4) * 0.02).to(dtype)


def _tokens(m, k, gen):
    return torch.randn((m, k), generator=gen, device="cuda").to(torch.bfloat16)


def _packed(n, k, gen, transform=""):
    w = _weight(n, k, gen)
    if transform:
        w = mx.apply_transform(w, transform)
    return mx.quantize_packed(w, rotation=transform or None)[0].to_stream_layout()


def _layer(case, gen):
    h, kv, ffn = case["hidden"], case["kv"], case["ffn"]
    shapes = {"q": (h, h), "k": (kv, h), "v": (kv, h), "o": (h, h), "gate": (ffn, h), "up": (ffn, h), "down": (h, ffn)}
    return {name: _packed(n, k, gen) for name, (n, k) in shapes.items()}


def _decode_step(layers, x):
    outs = []
    for w in layers:
        q, k, v = mx.mixfp4_linear_grouped(x, [w["q"], w["k"], w["v"]], overlap_previous=True)
        o = mx.mixfp4_linear(q, w["o"], overlap_previous=True)
        gate, up = mx.mixfp4_linear_grouped(o, [w["gate"], w["up"]], overlap_previous=True)
        outs += [q, k, v, o, gate, up, mx.mixfp4_linear(gate, w["down"], overlap_previous=True)]
    return outs


@torch.no_grad()
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, state = case["kind"], {"kind": case["kind"]}
    if kind == "decode":
        layers = [_layer(case, gen) for _ in range(case["layers"])]
        x = _tokens(case["batch"], case["hidden"], gen)
        slot = x.clone()
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            _decode_step(layers, slot)
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                outs = _decode_step(layers, slot)
        torch.cuda.synchronize()
        state.update(layers=layers, x=x, slot=slot, graph=graph, outs=outs)
    elif kind == "linear":
        state.update(w=_packed(case["n"], case["k"], gen, case["transform"]), x=_tokens(case["m"], case["k"], gen),
                     activation=case["activation"] or None, out=DTYPES[case["out"]])
    elif kind == "block":
        state.update(w=_layer(case, gen), x=_tokens(case["m"], case["hidden"], gen))
    elif kind == "convert":
        n, k = case["n"], case["k"]
        dense = torch.nn.Linear(k, n, bias=False, device="meta", dtype=DTYPES[case["dtype"]])
        dense.weight = torch.nn.Parameter(_weight(n, k, gen, DTYPES[case["dtype"]]), requires_grad=False)
        state.update(dense=dense, transform=case["transform"] or None)
    else:
        state.update(w=_weight(case["n"], case["k"], gen, DTYPES[case["dtype"]]), region=case["region"])
    return state


# -------------------------------------------------------------------------------------------- pass
@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "decode":
        state["slot"].copy_(state["x"])
        state["graph"].replay()
        return state["outs"]
    if kind == "linear":
        return mx.mixfp4_linear(state["x"], state["w"], activation_mode=state["activation"], out_dtype=state["out"])
    if kind == "block":
        w, x = state["w"], state["x"]
        q, k, v = mx.mixfp4_linear_grouped(x, [w["q"], w["k"], w["v"]])
        o = mx.mixfp4_linear(q, w["o"])
        gate, up = mx.mixfp4_linear_grouped(o, [w["gate"], w["up"]])
        return [q, k, v, o, gate, up, mx.mixfp4_linear(gate, w["down"])]
    if kind == "convert":
        layer = mx.MixFP4Linear.from_linear(state["dense"], rotation=state["transform"])
        return [layer.codes, layer.global_scale, layer.lut]
    return mx.quant_mixfp4_granularity(state["w"], format_region=state["region"])


# ------------------------------------------------------------------------------------ what it takes
def work(case):
    kind = case["kind"]
    if kind in ("decode", "block"):
        h, kv, ffn = case["hidden"], case["kv"], case["ffn"]
        m = case["batch"] if kind == "decode" else case["m"]
        shapes = [(h + 2 * kv, h), (h, h), (2 * ffn, h), (h, ffn)]          # weights that share an input read it once
        layers = case.get("layers", 1)
        return {"bytes": layers * sum(mx.packed_nbytes(n, k) + 2 * m * k + 2 * m * n for n, k in shapes),
                "flops": layers * sum(2.0 * m * n * k for n, k in shapes)}
    n, k = case["n"], case["k"]
    if kind == "linear":
        m, out = case["m"], 4 if case["out"] == "f32" else 2
        return {"bytes": mx.packed_nbytes(n, k) + 2 * m * k + out * m * n, "flops": 2.0 * m * n * k}
    size = 4 if case["dtype"] == "f32" else 2
    if kind == "convert":
        return {"bytes": size * n * k + mx.packed_nbytes(n, k), "flops": 0}
    return {"bytes": 2 * size * n * k, "flops": 0}


def tolerance(case):
    if case["kind"] in ("convert", "fake"):
        return "exact"                                                      # bytes and bit patterns of the format
    # Measured against the same path with its sums in double precision, times four.  One linear with bf16
    # output: results on either side of a rounding boundary, 1.8e-4 (one unit in the last place, 7.8e-3).
    # Linears in a chain carry such differences on: 2.3e-3 and 1.7e-2 after four.
    if case["kind"] in ("decode", "block"):
        return {"rel": 8e-3, "max": 0.07}
    if case["out"] == "f32":
        return {"rel": 1e-5, "max": 1e-4}                                   # fp32 sums of up to 14336 products
    return {"rel": 8e-4, "max": 0.04}
