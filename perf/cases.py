"""What the framework is timed on: the MoE expert layer as its users run it.

A user holds layers (`ExpertLayerSlice`), a stack of them (`MoeLayerStack`) or one expert's
feed-forward network (`ExpertFfn`) and passes token rows through.  Shapes and value
distributions are those of the repository's own configurations: the benchmark layer (hidden
2688, 128 experts x 1856, top-6, shared expert 3712, all NVFP4) and the reference checkpoint's
latent layer (hidden 4096, latent 1024, 512 experts x 2688, top-22, shared expert 5376; fc1_latent
and shared_up in scaled FP8, fc2_latent in bf16).  What varies from call to call is the number
of token rows, their type and how evenly the router spreads them.

Passes run on one stream of the caller's own, as in a serving loop.
"""
import importlib
import math

import torch

package = importlib.import_module("nemotron-inference_b200")
synthetic = importlib.import_module("nemotron-inference_b200.synthetic")
stack_module = importlib.import_module("nemotron-inference_b200.stack")

STACK_LAYERS = 3


def _case(kind, tokens, name=None, dtype="bf16", skewed=False, trace=False):
    """kind: "layer", "stack", "latent" or "ffn"; dtype: of the rows that go in and come out
    ("fp32" is what the caller's loop hands from layer to layer); skewed: popular and unpopular
    experts; trace: the layer keeps every intermediate for inspection, its default."""
    case = {"kind": kind, "tokens": tokens, "dtype": dtype, "skewed": skewed, "trace": trace}
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # one sequence being decoded: ten small kernels, launches and latency
        _case("layer", 1, "decode_1"),
        # a few sequences: reads the weights of about 36 experts
        _case("layer", 7, "decode_7"),
        # a full decode batch: nearly every expert is read, few rows each
        _case("layer", 64, "decode_64"),
        # the decode batch of the 23-layer configuration, rows handed on in FP32
        _case("stack", 256, "stack_decode_256", dtype="fp32"),
        # a prompt of odd length: every expert gets some 47 rows, tiles are ragged
        _case("layer", 1003, "prefill_1003"),
        # the prefill chunk of the 23-layer configuration, FP32 in and out, default settings
        _case("layer", 4096, "prefill_4096_fp32", dtype="fp32", trace=True),
        # popular and empty experts
        _case("layer", 8192, "prefill_8192_skewed", skewed=True),
        # the largest batch of the benchmark
        _case("layer", 16384, "prefill_16384"),
        # the checkpoint's latent layer: one sequence, a decode batch, an odd prompt
        _case("latent", 1, "latent_decode_1"),
        _case("latent", 40, "latent_decode_40"),
        _case("latent", 1000, "latent_prefill_1000"),
        # one expert's feed-forward network alone, called synchronously
        _case("ffn", 64, "ffn_64"),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "latent", "latent", "stack", "ffn"])
    if kind == "decode":
        return _case("layer", _log_int(rng, 1, 256), dtype=rng.choice(["bf16", "bf16", "fp32"]),
                     skewed=rng.random() < 0.2)
    if kind == "prefill":
        return _case("layer", _log_int(rng, 257, 16383), dtype=rng.choice(["bf16", "bf16", "fp32"]),
                     skewed=rng.random() < 0.3, trace=rng.random() < 0.3)
    if kind == "latent":
        return _case("latent", _log_int(rng, 1, 1000), dtype=rng.choice(["bf16", "fp32"]))
    if kind == "stack":
        return _case("stack", _log_int(rng, 1, 4000), dtype="fp32")
    return _case("ffn", _log_int(rng, 1, 4000), dtype=rng.choice(["bf16", "fp32"]))


class State:
    pass


_streams = []


def _serving_stream():
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _make_layer(case, seed):
    tokens = case["tokens"]
    if case["kind"] == "latent":
        config = synthetic.checkpoint_shape_config(max_tokens=max(256, tokens))
        data = synthetic.make_layer(config, seed, device="cuda", norm_weight_uniform=True,
                                    latent_family="fp8", shared_up_family="fp8")
    else:
        config = synthetic.baseline_config(max_tokens=max(256, tokens))
        data = synthetic.make_layer(config, seed, device="cuda", skewed=case["skewed"],
                                    norm_weight_uniform=case["kind"] == "stack")
    layer = package.ExpertLayerSlice.create(config, data.bindings)
    if layer is None:
        raise RuntimeError("layer creation failed: " + package.ExpertLayerSlice.create_error)
    if not case["trace"]:
        layer.keep_trace(False)
    return layer


def prepare(case, seed):
    state = State()
    state.kind = case["kind"]
    tokens, seed = case["tokens"], seed * 16
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    hidden = 4096 if state.kind == "latent" else synthetic.HIDDEN
    state.x = synthetic.make_tokens(tokens, hidden, seed + 15, device="cuda").to(dtype)
    state.out = torch.empty_like(state.x)
    if state.kind == "ffn":
        up, down = synthetic.make_ffn_weights(hidden, synthetic.ROUTED_INTERMEDIATE, seed,
                                              device="cuda")
        state.ffn = package.ExpertFfn(up, down, max_rows=tokens)
    elif state.kind == "stack":
        layers = [_make_layer(case, seed + i) for i in range(STACK_LAYERS)]
        state.stack = stack_module.MoeLayerStack(layers, hidden, tokens)
    else:
        state.layer = _make_layer(case, seed)
    state.stream = _serving_stream()
    torch.cuda.synchronize()
    return state


def run(state):
    with torch.cuda.stream(state.stream):
        if state.kind == "ffn":
            return state.ffn.run(state.x)
        if state.kind == "stack":
            state.stack.run(state.x, state.out)
        else:
            state.layer.run_async(state.x, state.out)
        return state.out


def _nvfp4(rows, cols):
    """Bytes of an NVFP4 matrix: codes and block scales."""
    return rows * cols * 9 // 16


def work(case):
    """Every weight that the rows need and every row read once, every result row written once."""
    tokens = case["tokens"]
    row = 2 if case["dtype"] == "bf16" else 4
    if case["kind"] == "ffn":
        hidden, inter = synthetic.HIDDEN, synthetic.ROUTED_INTERMEDIATE
        return {"bytes": 2 * _nvfp4(inter, hidden) + tokens * hidden * (row + 4),
                "flops": tokens * 4 * hidden * inter}
    if case["kind"] == "latent":
        hidden, latent, inter, shared, experts, top_k = 4096, 1024, 2688, 5376, 512, 22
        dense = latent * hidden + shared * hidden + 2 * latent * hidden  # FP8, FP8, bf16
        dense_flops = 2 * (2 * latent * hidden + shared * hidden)
        shared_nvfp4, shared_nvfp4_flops = _nvfp4(hidden, shared), 2 * shared * hidden
    else:
        hidden, inter, shared, experts, top_k = (synthetic.HIDDEN, synthetic.ROUTED_INTERMEDIATE,
                                                 synthetic.SHARED_INTERMEDIATE, synthetic.EXPERTS,
                                                 synthetic.TOP_K)
        latent, dense, dense_flops = hidden, 0, 0
        shared_nvfp4, shared_nvfp4_flops = 2 * _nvfp4(shared, hidden), 4 * shared * hidden
    # experts that some token selects, were every selection equally likely
    touched = experts * (1.0 - (1.0 - top_k / experts) ** tokens)
    layers = STACK_LAYERS if case["kind"] == "stack" else 1
    weights = touched * 2 * _nvfp4(inter, latent) + shared_nvfp4 + dense + 2 * experts * hidden
    per_token = top_k * 4 * latent * inter + shared_nvfp4_flops + dense_flops + 2 * experts * hidden
    return {"bytes": int(layers * (weights + 2 * tokens * hidden * row)),
            "flops": layers * tokens * per_token}


def tolerance(case):
    # The sums are FP32, but what they make is rounded to FP4 codes: a sum on a rounding boundary
    # to within its own noise may take the neighbouring code, which moves one row by a few
    # percent.  Such rows are rare in one layer; the next layer's codes follow from them.
    if case["kind"] == "stack":
        return {"rel": 1e-2, "max": 0.5}
    if case["kind"] == "ffn" or case["dtype"] == "fp32":
        return {"rel": 2e-3, "max": 0.2}
    return {"rel": 5e-3, "max": 0.2}
