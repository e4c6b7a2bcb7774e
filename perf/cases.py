"""The work that is timed: what a program that serves or converts W4A16 models has this package do.

Four kinds of case:

  linear      one `QuantizedLinear` forward, called eagerly
  layer       the linear work of decoder layers through the fused modules: residual + RMSNorm + qkv
              (`RmsNormLinear`), the attention output projection, gate/up with SiLU (`GateUpSilu`) and the
              down projection; `qkv` = 0 leaves the attention half out (an MLP alone)
  quantize    `QuantizedLinear.from_float` of a trained weight: codes, steps, zero points and the device image
  dequantize  `dequantize_int4` of a checkpoint's tensors: the device image and from it the FP32 weights

`graph` = True replays the calls from a CUDA graph, as a serving loop does with its decode step; otherwise every
call is made from Python.  Layer shapes are those of the benchmark configurations (Qwen3-0.6B, Qwen3-8B,
Llama-3-70B MLP and the stress sweep); weights, activations and quantized states have their distributions.
"""
import math

import torch

import dandan_ops_b200 as ops

_DEVICE = "cuda"


def listed():
    return [
        # The smallest call: one token through the smallest projection of the smallest model, from Python.
        {"name": "token-o-0.6b", "kind": "linear", "n": 1024, "k": 2048, "m": 1, "bias": False, "steps": "fp32", "graph": False},
        # One token through a stack of small decoder layers, the serving loop's graph.
        {"name": "decode1-0.6b", "kind": "layer", "hidden": 1024, "qkv": 4096, "attn": 2048, "inter": 3072, "layers": 12,
         "m": 1, "graph": True},
        # One token through a decoder layer of a mid-size model.
        {"name": "decode1-8b", "kind": "layer", "hidden": 4096, "qkv": 6144, "attn": 4096, "inter": 12288, "layers": 2,
         "m": 1, "graph": True},
        # Sixteen sequences decoded together.
        {"name": "decode16-8b", "kind": "layer", "hidden": 4096, "qkv": 6144, "attn": 4096, "inter": 12288, "layers": 2,
         "m": 16, "graph": True},
        # The MLP of a large model, eight sequences, called from Python.
        {"name": "decode8-70b-mlp", "kind": "layer", "hidden": 8192, "qkv": 0, "attn": 0, "inter": 28672, "layers": 1,
         "m": 8, "graph": False},
        # A checkpoint with FP16 steps, ragged output width, bias and a ragged batch (the stress sweep).
        {"name": "ragged17-bias", "kind": "linear", "n": 12289, "k": 3072, "m": 17, "bias": True, "steps": "fp16", "graph": False},
        # A serving batch of sixty-four sequences on a mid-size layer.
        {"name": "batch64-8b", "kind": "layer", "hidden": 4096, "qkv": 6144, "attn": 4096, "inter": 12288, "layers": 1,
         "m": 64, "graph": True},
        # A prompt through a small layer.
        {"name": "prefill512-0.6b", "kind": "layer", "hidden": 1024, "qkv": 4096, "attn": 2048, "inter": 3072, "layers": 1,
         "m": 512, "graph": False},
        # Prompts through a mid-size layer.
        {"name": "prefill2048-8b", "kind": "layer", "hidden": 4096, "qkv": 6144, "attn": 4096, "inter": 12288, "layers": 1,
         "m": 2048, "graph": False},
        # The largest: a long prompt through the MLP of a large model.
        {"name": "prefill4096-70b-mlp", "kind": "layer", "hidden": 8192, "qkv": 0, "attn": 0, "inter": 28672, "layers": 1,
         "m": 4096, "graph": False},
        # Converting a model: FP16 weights to the INT4 format (and the image the kernels read).
        {"name": "quantize-down-8b", "kind": "quantize", "n": 4096, "k": 12288, "dtype": "float16"},
        # Exporting or checking one: checkpoint tensors back to FP32 weights.
        {"name": "dequantize-qkv-8b", "kind": "dequantize", "n": 6144, "k": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, of):
    return max(lo, _log(rng, lo, hi) // of * of)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "layer", "layer", "layer", "quantize", "dequantize"])
    if kind == "layer":
        m = _log(rng, 1, 2048)
        hidden = _multiple(rng, 1024, 4096, 64)
        attn = _multiple(rng, 1024, 4096, 64)
        inter = _multiple(rng, 2048, 12288, 64)
        qkv = rng.choice([0, attn + 2 * _multiple(rng, 512, 1024, 64)])
        return {"kind": kind, "hidden": hidden, "qkv": qkv, "attn": attn if qkv else 0, "inter": inter,
                "layers": rng.randint(1, 3), "m": m, "graph": rng.random() < 0.7 if m <= 64 else False}
    n = _multiple(rng, 1024, 28672, 64)
    if rng.random() < 0.5:
        n += rng.randint(1, 63)
    k = _multiple(rng, 1024, 12288, 64)
    if kind == "linear":
        m = _log(rng, 1, 4096)
        if m <= 64 and rng.random() < 0.25:
            k += rng.randint(1, 63)
        return {"kind": kind, "n": n, "k": k, "m": m, "bias": rng.random() < 0.3, "steps": rng.choice(["fp32", "fp32", "fp16"]),
                "graph": False}
    if rng.random() < 0.5:
        k += rng.randint(1, 63)
    if kind == "quantize":
        return {"kind": kind, "n": n, "k": k, "dtype": rng.choice(["float16", "float32"])}
    return {"kind": kind, "n": n, "k": k}


# ---- inputs ------------------------------------------------------------------------------------------------


def _weight(gen, n, k, sigma, dtype=torch.float16):
    return (torch.randn(n, k, generator=gen, device=_DEVICE) * sigma).to(dtype)


def _layer(gen, n, k, sigma, bias=False):
    b = torch.randn(n, generator=gen, device=_DEVICE).half() if bias else None
    return ops.QuantizedLinear.from_float(_weight(gen, n, k, sigma), b, group_size=64)


def _checkpoint_state(gen, n, k):
    """Uniform codes and zero points, log-normal steps that FP16 can hold, one group in a hundred fifty times larger."""
    groups = -(-k // 64)
    codes = torch.randint(0, 16, (n, k), generator=gen, device=_DEVICE, dtype=torch.uint8)
    zeros = torch.randint(0, 16, (n, groups), generator=gen, device=_DEVICE, dtype=torch.int32)
    steps = torch.exp(torch.randn(n, groups, generator=gen, device=_DEVICE) * 0.5 - 5.0)
    steps = torch.where(torch.rand(n, groups, generator=gen, device=_DEVICE) < 0.01, steps * 50.0, steps).half().float()
    return ops.pack_int4(codes), steps, zeros


def _x(gen, m, k):
    return torch.randn(m, k, generator=gen, device=_DEVICE).half()


def _decoder_layer(gen, case):
    sigma = 0.015 if case["hidden"] >= 8192 else 0.02
    hidden, inter, m = case["hidden"], case["inter"], case["m"]
    part = {"mlp_in": _x(gen, m, hidden),
            "gate_up": ops.GateUpSilu(_layer(gen, inter, hidden, sigma), _layer(gen, inter, hidden, sigma)),
            "down": _layer(gen, hidden, inter, sigma)}
    if case["qkv"]:
        norm = 1.0 + 0.1 * torch.randn(hidden, generator=gen, device=_DEVICE)
        part.update(qkv=ops.RmsNormLinear(norm, _layer(gen, case["qkv"], hidden, sigma), eps=1e-6),
                    o=_layer(gen, hidden, case["attn"], sigma), block_in=_x(gen, m, hidden), residual=_x(gen, m, hidden),
                    attn_out=_x(gen, m, case["attn"]))
    return part


def _calls(state):
    case = state["case"]
    if case["kind"] == "linear":
        return [state["layer"](state["x"])]
    outputs = []
    for part in state["parts"]:
        if "qkv" in part:
            outputs.extend(part["qkv"](part["block_in"], part["residual"]))
            outputs.append(part["o"](part["attn_out"]))
        outputs.append(part["down"](part["gate_up"](part["mlp_in"])))
    return outputs


def prepare(case, seed):
    gen = torch.Generator(device=_DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "quantize":
        return {"case": case, "weight": _weight(gen, case["n"], case["k"], 0.02, getattr(torch, case["dtype"]))}
    if kind == "dequantize":
        codes, steps, zeros = ops.quantize_int4(_weight(gen, case["n"], case["k"], 0.02), 64)
        return {"case": case, "packed": ops.pack_int4(codes), "scales": steps, "zeros": zeros}
    state = {"case": case, "graph": None}
    if kind == "linear":
        n, k = case["n"], case["k"]
        if case["steps"] == "fp16":
            bias = torch.randn(n, generator=gen, device=_DEVICE).half() if case["bias"] else None
            state["layer"] = ops.QuantizedLinear(*_checkpoint_state(gen, n, k), in_features=k, bias=bias)
        else:
            state["layer"] = _layer(gen, n, k, 0.02, case["bias"])
        state["x"] = _x(gen, case["m"], k)
    else:
        state["parts"] = [_decoder_layer(gen, case) for _ in range(case["layers"])]
    if case["graph"]:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _calls(state)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["outputs"] = _calls(state)
        state["graph"] = graph
    return state


@torch.no_grad()
def run(state):
    case = state["case"]
    if case["kind"] == "quantize":
        layer = ops.QuantizedLinear.from_float(state["weight"], group_size=64)
        return [layer.packed_weight, layer.scales, layer.zeros]
    if case["kind"] == "dequantize":
        return ops.dequantize_int4(state["packed"], state["scales"], state["zeros"], case["k"])
    if state["graph"] is not None:
        state["graph"].replay()
        return state["outputs"]
    return _calls(state)


# ---- what a pass cannot do without, and how far two correct ones differ -------------------------------------


def _state_bytes(n, k):
    """4-bit codes, and an FP32 step and a 4-bit zero point per row and group of 64."""
    return n * k / 2 + n * (-(-k // 64)) * 4.5


def _linear_work(n, k, m, out=None):
    return _state_bytes(n, k) + 2 * m * k + 2 * m * (n if out is None else out), 2.0 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "quantize":
        n, k = case["n"], case["k"]
        return {"bytes": n * k * (2 if case["dtype"] == "float16" else 4) + n * k / 2 + n * (-(-k // 64)) * 8, "flops": 0}
    if kind == "dequantize":
        n, k = case["n"], case["k"]
        return {"bytes": n * k / 2 + n * (-(-k // 64)) * 8 + 4 * n * k, "flops": 0}
    if kind == "linear":
        size, flops = _linear_work(case["n"], case["k"], case["m"])
        return {"bytes": size, "flops": flops}
    m, hidden, inter = case["m"], case["hidden"], case["inter"]
    parts = [_linear_work(2 * inter, hidden, m, inter), _linear_work(hidden, inter, m)]
    if case["qkv"]:
        # the norm reads its input and the residual and writes their sum
        parts += [_linear_work(case["qkv"], hidden, m), (4 * m * hidden, 0.0), _linear_work(hidden, case["attn"], m)]
    return {"bytes": case["layers"] * sum(p[0] for p in parts), "flops": case["layers"] * sum(p[1] for p in parts)}


def tolerance(case):
    if case["kind"] in ("quantize", "dequantize"):
        return "exact"
    # FP16 outputs of FP32 sums: another order of the sums flips the last bit of a few per cent of them.  Against the
    # same product with 64-bit sums a projection is off by up to 6e-5 (2-norm), the MLP, whose FP16 activation goes
    # through a second projection, by up to 2.6e-4; single values by up to 2e-3.
    return {"rel": 2.4e-4 if case["kind"] == "linear" else 1e-3, "max": 8e-3}
