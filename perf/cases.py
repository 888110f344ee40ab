"""The work this framework is measured on: FPx x fp16 linear layers as a user's program calls them, from one small layer
to the prefill of a large decoder block, and the weight conversion that comes before them.

A case is a dict with an "op":

  "layers"   single layers through `linear_forward_eXmY_cuda`, the operator drop-in programs use
  "block"    the four linear layers of a decoder block through the modules (`FPxLinear`, `FPxGateUpLinear`)
  "load"     an fp16 layer of a checkpoint turned into a module (`FPxLinear.from_linear`, `enable_native`)
  "convert"  unpacked codes packed for the kernels and expanded to fp16 (prepack, both dequantisers)
  "host"     layers whose activations arrive and whose results are wanted in host memory (`linear_forward_host_batch`)
"""
import math

import torch

import fp6_llm_b200 as fpx
from fp6_llm_b200.formats import bit_width

SMS = 148   # what a program passes to the split-K heuristic on this GPU


def _block(name, hidden, qkv, ffn, tokens, e, m, native, bias=False):
    return {"name": name, "op": "block", "hidden": hidden, "qkv": qkv, "ffn": ffn, "tokens": tokens, "e": e, "m": m,
            "native": native, "bias": bias}


def listed():
    return [
        # the quick-start call: one small FP6 layer, a handful of tokens, no split; launches and host work count
        {"name": "layer-4096-8tok", "op": "layers", "oc": 4096, "ic": 4096, "ffn": 0, "tokens": 8, "e": 3, "m": 2, "split": "one"},
        # a chat with one user: one token per step through a small model, weights also kept in the decode layout
        _block("7b-fp6-decode-1", 4096, 12288, 11008, 1, 3, 2, True),
        # decode of a served batch through a large model: streaming 640 MB of weights is the work
        _block("70b-fp6-decode-16", 8192, 10240, 28672, 16, 3, 2, True),
        # the drop-in operator on FP5 weights with the split-K heuristic, as the original project's programs call it
        {"name": "13b-fp5-op-16tok", "op": "layers", "oc": 5120, "ic": 5120, "ffn": 13824, "tokens": 16, "e": 2, "m": 2, "split": "heuristic"},
        # a busy server: 64 and 128 sequences decoded at once, between the memory-bound and the compute-bound regime
        _block("70b-fp6-batch-64", 8192, 10240, 28672, 64, 3, 2, True),
        _block("7b-fp6-batch-128", 4096, 12288, 11008, 128, 3, 2, False),
        # prompts: a ragged one through FP5 layers with biases, one of a few hundred tokens, one long (the largest case)
        _block("13b-fp5-prompt-333", 5120, 15360, 13824, 333, 2, 2, False, True),
        _block("70b-fp6-prompt-512", 8192, 10240, 28672, 512, 3, 2, True),
        _block("70b-fp6-prompt-2048", 8192, 10240, 28672, 2048, 3, 2, True),
        # start of a server: a large fp16 layer is scaled, quantised and laid out on the GPU
        {"name": "load-fp6-8192x28672", "op": "load", "oc": 8192, "ic": 28672, "e": 3, "m": 2, "native": True},
        # a checkpoint that already holds codes: packed for the kernels, and expanded to fp16 for checks and fp16 layers
        {"name": "convert-fp6-10240x8192", "op": "convert", "oc": 10240, "ic": 8192, "e": 3, "m": 2},
        # an engine that keeps activations on the host: the block's layers as one pipelined batch
        {"name": "host-13b-fp6-16tok", "op": "host", "oc": 5120, "ic": 5120, "ffn": 13824, "tokens": 16, "e": 3, "m": 2, "native": True},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _multiple(x, of):
    return max(of, int(round(x / of)) * of)


def draw(rng):
    """One more case of the ranges above: hidden sizes 1024 .. 8192, any token count up to 2048, every format."""
    most = _flops(listed()[8])
    op = rng.choices(["block", "layers", "load", "convert", "host"], [10, 5, 2, 2, 1])[0]
    e, m = rng.choice([(3, 2), (3, 2), (3, 2), (2, 2), (2, 2), (2, 3), (3, 1), (2, 1)])
    while True:
        if op == "block":
            hidden = _multiple(_log_uniform(rng, 1024, 8192), 256)
            kv = rng.choice([hidden, max(256, _multiple(hidden / 8, 128))])
            ffn = min(28672, _multiple(hidden * rng.uniform(2.0, 4.0), 128))
            case = {"op": op, "hidden": hidden, "qkv": hidden + 2 * kv, "ffn": ffn, "tokens": int(_log_uniform(rng, 1, 2049)),
                    "e": e, "m": m, "native": rng.random() < 0.6, "bias": rng.random() < 0.3}
        elif op == "layers":
            case = {"op": op, "oc": _multiple(_log_uniform(rng, 1024, 16384), 256), "ic": _multiple(_log_uniform(rng, 1024, 16384), 64),
                    "ffn": 0, "tokens": int(_log_uniform(rng, 1, 513)), "e": e, "m": m, "split": rng.choice(["one", "heuristic", "auto"])}
        elif op == "host":
            hidden = _multiple(_log_uniform(rng, 2048, 6144), 256)
            case = {"op": op, "oc": hidden, "ic": hidden, "ffn": _multiple(hidden * rng.uniform(2.0, 3.5), 128),
                    "tokens": int(_log_uniform(rng, 1, 65)), "e": e, "m": m, "native": rng.random() < 0.5}
        else:
            case = {"op": op, "oc": _multiple(_log_uniform(rng, 1024, 16384), 256), "ic": _multiple(_log_uniform(rng, 1024, 16384), 64),
                    "e": e, "m": m}
            if op == "load":
                case["native"] = rng.random() < 0.7
        if _flops(case) <= most:
            return case


def _shapes(case):
    """(output channels, input channels) of the layers a case runs."""
    if case["op"] == "block":
        h, f = case["hidden"], case["ffn"]
        return [(case["qkv"], h), (h, h), (2 * f, h), (h, f)]
    if case.get("ffn"):   # the four layers of a block with full-width keys and values
        h, f = case["ic"], case["ffn"]
        return [(3 * h, h), (h, h), (2 * f, h), (h, f)]
    return [(case["oc"], case["ic"])]


def _flops(case):
    return sum(2 * oc * ic for oc, ic in _shapes(case)) * case.get("tokens", 0)


def work(case):
    bw = bit_width(case["e"], case["m"])
    if case["op"] == "load":     # fp16 weights in; codes (once per layout) and scales out
        n = case["oc"] * case["ic"]
        return {"bytes": 2 * n + n * bw / 8 + (n * 6 / 8 if case["native"] else 0) + 2 * case["oc"], "flops": 0}
    if case["op"] == "convert":  # pack: codes in, codes out; each dequantiser: codes in, fp16 out
        n = case["oc"] * case["ic"]
        return {"bytes": 4 * n * bw / 8 + 2 * 2 * n + 2 * 2 * case["oc"], "flops": 0}
    t = case["tokens"]
    total = sum(oc * ic * bw / 8 + 2 * oc + 2 * t * (oc + ic) for oc, ic in _shapes(case))
    if case["op"] == "block":
        total -= 2 * t * case["ffn"]   # gate and up leave their layer as one product
        if case["bias"]:
            total += sum(2 * oc for oc, _ in _shapes(case))
    return {"bytes": total, "flops": _flops(case)}


def tolerance(case):
    if case["op"] in ("load", "convert"):
        return "exact"
    # Measured against the same sums in 64 bits: one layer is off by rel 2.1e-4 and max 5e-4 (the rounding of the result to
    # fp16; 8.9e-4 at most with K = 28672), gate/up followed by the down layer by 3.0e-4 and 1.3e-3 (its fp16 input is rounded too).
    return {"rel": 1e-3, "max": 5e-3}


def _weights(gen, oc, ic):
    return torch.randn(oc, ic, generator=gen, device="cuda", dtype=torch.float16).mul_(0.02)


def _linear(gen, oc, ic, bias):
    layer = torch.nn.utils.skip_init(torch.nn.Linear, ic, oc, bias=bias, device="cuda", dtype=torch.float16)
    layer.weight.data = _weights(gen, oc, ic)
    if bias:
        layer.bias.data = torch.randn(oc, generator=gen, device="cuda", dtype=torch.float16).mul_(0.1)
    return layer


def _activations(gen, tokens, ic):
    return torch.randn(tokens, ic, generator=gen, device="cuda", dtype=torch.float16)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, e, m = case["op"], case["e"], case["m"]
    state = {"op": op, "e": e, "m": m}
    with torch.no_grad():
        if op == "block":
            bias, shapes = case["bias"], _shapes(case)
            f = case["ffn"]
            layers = [fpx.FPxLinear.from_linear(_linear(gen, oc, ic, bias), e, m) for oc, ic in shapes[:2]]
            layers.append(fpx.FPxGateUpLinear.from_linears(_linear(gen, f, case["hidden"], bias), _linear(gen, f, case["hidden"], bias), e, m))
            layers.append(fpx.FPxLinear.from_linear(_linear(gen, *shapes[3], bias), e, m))
            if case["native"]:
                for layer in layers:
                    layer.enable_native()
            state["layers"] = layers
            state["x"] = [_activations(gen, case["tokens"], case["hidden"]) for _ in range(3)]
        elif op in ("layers", "host"):
            calls = []
            for oc, ic in _shapes(case):
                w = _weights(gen, oc, ic)
                scales = fpx.FPxLinear.row_scales(w, e, m)
                packed = fpx.quantize_prepack_cuda(w, scales, e, m)
                x = _activations(gen, case["tokens"], ic)
                if op == "layers":
                    split = {"one": 1, "auto": 0}.get(case["split"])
                    if split is None:
                        split = fpx.HeuristicFuntion_SplitK(oc, case["tokens"], SMS)
                    calls.append((x, packed, scales, split))
                else:
                    call = (e, m, x.cpu().pin_memory(), packed, scales,
                            torch.empty(case["tokens"], oc, dtype=torch.float16, pin_memory=True), 0)
                    calls.append(call + (fpx.native_repack(e, m, packed),) if case["native"] else call)
            state["calls"] = calls
        elif op == "load":
            state["linear"] = _linear(gen, case["oc"], case["ic"], False)
            state["native"] = case["native"]
        else:
            cols = case["ic"] * bit_width(e, m) // 32
            state["codes"] = torch.randint(-2**31, 2**31, (case["oc"], cols), generator=gen, device="cuda", dtype=torch.int32)
            state["scales"] = torch.rand(case["oc"], generator=gen, device="cuda").mul_(9e-3).add_(1e-3).half()
    return state


@torch.no_grad()
def run(state):
    op, e, m = state["op"], state["e"], state["m"]
    if op == "block":   # what lies between the layers (attention, norms) is not this framework's: o has an input of its own
        qkv, o, gate_up, down = state["layers"]
        x_attn, x_o, x_mlp = state["x"]
        h = gate_up(x_mlp)
        return [qkv(x_attn), o(x_o), h, down(h)]
    if op == "layers":
        return [fpx.linear_forward_eXmY_cuda(e, m, x, packed, scales, split) for x, packed, scales, split in state["calls"]]
    if op == "host":
        fpx.linear_forward_host_batch(state["calls"])
        return [call[5] for call in state["calls"]]
    if op == "load":
        layer = fpx.FPxLinear.from_linear(state["linear"], e, m)
        if state["native"]:
            layer.enable_native()
            return [layer.weight, layer.scales, layer.weight_native]
        return [layer.weight, layer.scales]
    packed = fpx.weight_prepacking_eXmY_cpu(e, m, state["codes"])
    return [packed, fpx.weight_dequant_eXmY_cpu(e, m, state["codes"], state["scales"]), fpx.dequant_packed_cuda(e, m, packed, state["scales"])]
