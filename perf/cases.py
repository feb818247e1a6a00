"""The work a user of the hybrid MXFP4/MXFP8 linear layer has it do, as cases that can be timed and compared.

Four kinds of pass, all through the package's public entry points:

* "block":   the linears of one decoder block, as a serving engine calls them through the registered ops: qkv_proj,
             o_proj, gate_up_proj and SwiGLU + down_proj (`ops.linear`, `ops.linear_silu`).  Attention lies between
             them and belongs to the engine, so each linear but down_proj has an input of its own.  With `graph` the
             calls are captured once and a pass replays them (decode runs under full CUDA graphs); without it they
             are eager (prefill).
* "linear":  one layer called directly (`DualLinear.__call__`), eager: quantise the activations and multiply.
* "load":    packing of one 16-bit weight matrix into the two partitions (`DualLinear.__init__`), once per layer when
             a model is loaded.
* "offline": the exponent search behind offline banks (`fp4_quant.quantize`) on one chunk of rows, with statistics.

Values follow the benchmark configurations: activations ~N(0,1) with 1 % of the K columns scaled by 20, weights
~N(0,0.02), a seeded sorted selection of MXFP8 channels.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "comp2029-hybridgemm_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from hygemm_vllm import fp4_quant, native, ops  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _block(name, tokens, hidden, qkv, attention, inter, dtype="bf16", graph=True, fraction=0.1):
    return {"name": name, "kind": "block", "tokens": tokens, "hidden": hidden, "qkv": qkv, "attention": attention,
            "inter": inter, "dtype": dtype, "graph": graph, "fraction": fraction}


def listed():
    qwen = dict(hidden=3584, qkv=4608, attention=3584, inter=18944)      # Qwen2.5-7B
    mistral = dict(hidden=4096, qkv=6144, attention=4096, inter=14336)   # Mistral-7B
    return [
        # The smallest call: the Qwen2.5-0.5B gate shape at eight tokens, eager.  Host work and launches decide.
        {"name": "linear_small_8", "kind": "linear", "tokens": 8, "k": 896, "outputs": 4864, "high": 486, "dtype": "bf16"},
        # An ordinary eager call with nothing round about it: odd tokens, odd width, IEEE half.
        {"name": "linear_odd_77", "kind": "linear", "tokens": 77, "k": 2432, "outputs": 7003, "high": 701, "dtype": "fp16"},
        # Decode of a 7B model under CUDA graphs: one user, a few users, a busy server, a full one.
        _block("decode_1", 1, **qwen),
        _block("decode_16", 16, **qwen),
        _block("decode_64", 64, **qwen),
        _block("decode_128", 128, **qwen),
        # The other 7B architecture in IEEE half at a batch that is no multiple of a tile.
        _block("decode_odd_37", 37, dtype="fp16", **mistral),
        # One rank's shard of it at tensor parallel 4, batch 128: column-parallel N / 4, row-parallel K / 4.
        _block("decode_shard_128", 128, hidden=4096, qkv=1536, attention=1024, inter=3584),
        # Prefill, eager: a ragged prompt, and a full chunk.
        _block("prefill_777", 777, dtype="fp16", graph=False, **qwen),
        _block("prefill_2048", 2048, graph=False, **qwen),
        # Model load: the widest layer of the 7B model.
        {"name": "load_gate_up", "kind": "load", "k": 3584, "outputs": 37888, "high": 3840, "dtype": "bf16"},
        # Bank writing: one chunk of rows, errors weighted by the input channels' second moments.
        {"name": "offline_chunk", "kind": "offline", "rows": 4096, "k": 3584, "dtype": "bf16", "weighted": True},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "linear", "linear", "load", "offline"))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    if kind in ("decode", "prefill"):
        hidden = 128 * rng.randint(7, 28)
        attention = rng.choice((hidden, hidden, 128 * rng.randint(4, hidden // 128)))
        case = _block("", _log_int(rng, 1, 128) if kind == "decode" else _log_int(rng, 129, 2048), hidden,
                      attention + 256 * rng.randint(1, 4), attention,
                      min(18944, 128 * round(hidden * rng.uniform(1.0, 5.4) / 128)), dtype, kind == "decode",
                      rng.choice((0.05, 0.1, 0.1, 0.2)))
        del case["name"]
        return case
    k = 128 * _log_int(rng, 4, 48)
    outputs = _log_int(rng, 640, 12000)
    if kind == "linear":
        return {"kind": "linear", "tokens": _log_int(rng, 1, 512), "k": k, "outputs": outputs,
                "high": round(outputs * rng.choice((0.05, 0.1, 0.1, 0.2))), "dtype": dtype}
    if kind == "load":
        return {"kind": "load", "k": k, "outputs": outputs, "high": round(outputs * rng.choice((0.05, 0.1, 0.2))), "dtype": dtype}
    return {"kind": "offline", "rows": _log_int(rng, 256, 4096), "k": k, "dtype": dtype, "weighted": rng.random() < 0.5}


def _quota(outputs, fraction):
    """A fraction of the channels, rounded to a multiple of 128, at least one multiple."""
    return max(128, round(outputs * fraction / 128) * 128)


def _linears(case):
    """(outputs, k) of the four linears of a block."""
    return [(case["qkv"], case["hidden"]), (case["hidden"], case["attention"]), (2 * case["inter"], case["hidden"]),
            (case["hidden"], case["inter"])]


class _State:
    """Inputs, layers and (for decode) the captured graph; the layers' device memory is given back with it."""

    def __init__(self, case):
        self.case, self.layers, self.handles, self.graph, self.outputs = case, [], [], None, None

    def __del__(self):
        self.graph = self.outputs = None
        for handle in self.handles:
            ops._runtimes.pop(handle, None)
        for layer in self.layers:
            layer.close()


def _activations(tokens, k, dtype, generator):
    x = torch.randn(tokens, k, device="cuda", generator=generator)
    outliers = torch.randperm(k, device="cuda", generator=generator)[:max(1, -(-k // 100))]
    x[:, outliers] *= 20
    return x.to(dtype)


def _weight(outputs, k, dtype, generator):
    return torch.randn(outputs, k, device="cuda", generator=generator, dtype=dtype) * 0.02


def _selection(outputs, high, generator):
    return torch.sort(torch.randperm(outputs, device="cuda", generator=generator)[:high]).values


def prepare(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _DTYPES[case["dtype"]]
    state = _State(case)
    if case["kind"] == "linear":
        layer = native.DualLinear(_weight(case["outputs"], case["k"], dtype, generator),
                                  _selection(case["outputs"], case["high"], generator))
        state.layers = [layer]
        state.x = _activations(case["tokens"], case["k"], dtype, generator)
    elif case["kind"] == "block":
        for outputs, k in _linears(case):
            state.layers.append(native.DualLinear(_weight(outputs, k, dtype, generator),
                                                  _selection(outputs, _quota(outputs, case["fraction"]), generator)))
        state.handles = [ops.register_runtime(layer) for layer in state.layers]
        state.inputs = [_activations(case["tokens"], k, dtype, generator) for _, k in _linears(case)[:3]]
        if case["graph"]:
            _block_pass(state)                       # every shape is warmed before the capture
            torch.cuda.synchronize()
            state.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state.graph):
                state.outputs = _block_pass(state)
    elif case["kind"] == "load":
        state.weight = _weight(case["outputs"], case["k"], dtype, generator)
        state.ids = _selection(case["outputs"], case["high"], generator)
    else:
        state.weight = _weight(case["rows"], case["k"], dtype, generator)
        state.importance = (_activations(64, case["k"], torch.float32, generator).square().mean(0)
                            if case["weighted"] else None)
    return state


def _block_pass(state):
    (qkv, o_proj, gate_up, down), (x, attention, hidden) = state.handles, state.inputs
    case = state.case
    y_qkv = ops.linear(x, qkv, case["qkv"])
    y_o = ops.linear(attention, o_proj, case["hidden"])
    y_gate_up = ops.linear(hidden, gate_up, 2 * case["inter"])
    y_down = ops.linear_silu(y_gate_up, down, case["hidden"], 0)
    return y_qkv, y_o, y_gate_up, y_down


def run(state):
    kind = state.case["kind"]
    if kind == "linear":
        return state.layers[0](state.x)
    if kind == "block":
        if state.graph is None:
            return _block_pass(state)
        state.graph.replay()
        return state.outputs
    if kind == "load":
        layer = native.DualLinear(state.weight, state.ids)
        return layer.w4, layer.sf4, layer.w8, layer.sf8, layer.lo, layer.hi
    return fp4_quant.quantize(state.weight, state.importance)


def _packed_bytes(outputs, k, high):
    """Codes, scales and channel maps of a packed layer."""
    return (outputs - high) * k / 2 + high * k + outputs * k / 32 + 4 * outputs


def work(case):
    if case["kind"] == "linear":
        m, n, k = case["tokens"], case["outputs"], case["k"]
        return {"bytes": _packed_bytes(n, k, case["high"]) + 2 * m * k + 2 * m * n, "flops": 2 * m * n * k}
    if case["kind"] == "block":
        m = case["tokens"]
        weights = sum(_packed_bytes(n, k, _quota(n, case["fraction"])) for n, k in _linears(case))
        # down_proj's input is gate_up's output: written once, and no input of the pass
        activations = sum(2 * m * k for _, k in _linears(case)[:3]) + sum(2 * m * n for n, _ in _linears(case))
        return {"bytes": weights + activations, "flops": sum(2 * m * n * k for n, k in _linears(case))}
    if case["kind"] == "load":
        n, k = case["outputs"], case["k"]
        return {"bytes": 2 * n * k + 8 * case["high"] + _packed_bytes(n, k, case["high"]), "flops": 0}
    rows, k = case["rows"], case["k"]
    return {"bytes": 2 * rows * k + (4 * k if case["weighted"] else 0) + rows * k / 2 + rows * k / 32, "flops": 0}


def tolerance(case):
    """Codes, scale bytes and maps are exact.  A linear's fp32 sums may be added in another order and are rounded once
    to 16 bits (half an ulp is 2^-9 of the value in bf16, 2^-12 in fp16); in a block, values that rounded the other
    way reach down_proj through an 8-bit quantisation.  The statistics of the offline search are sums of 32-bit terms."""
    if case["kind"] == "load":
        return "exact"
    if case["kind"] == "offline":
        return {"rel": 1e-5, "differ": 0.0}
    return {"rel": 5e-3} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 0.04}
