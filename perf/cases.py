"""The work that users of the packed linear layer have it do, as timed cases.

Sizes are the Llama-3-8B linears and the square benchmark layers (``matgptq_b200.synth``, the published kernel
benchmark up to 8192), the Llama-3.1-8B decoder harness cut to a few layers, and ragged sizes between them.  Every
case goes through an entry point that a user's program calls:

* ``linear``   ``MatGPTQLinear.forward`` as the HF-transformers path calls it, one layer after the other
* ``grouped``  ``matmul_matgptq_grouped``, a fused layer whose parts have their own bitwidths (the vLLM method)
* ``zeros``    ``matmul_matgptq_zeros``, checkpoints with per-group zero points (the vLLM method with ``zero_points``)
* ``repack``   ``slice_pack_matgptq_qweights``, loading a layer or switching its bitwidth from the master codes
* ``decode``   one token for every sequence of a batch: ``PackedLlama.forward`` as a replayed CUDA graph, which is how
               ``generate`` and the serving loops run it
* ``prefill``  ``PackedLlama.forward`` over whole prompts, eager
"""
import torch

from matgptq_b200 import decode as llama
from matgptq_b200 import ops  # noqa: F401  registers torch.ops.matgptq_cuda.*
from matgptq_b200 import synth
from matgptq_b200.matgptq_linear import MatGPTQLinear

FLAGS = 1 | 4  # asynchronous, programmatic dependent launch: what the module and the vLLM method pass
HEADS, KV_HEADS, HIDDEN, INTER = 32, 8, 4096, 14336  # the Llama-3.1-8B architecture
VOCAB_PER_LAYER = 128256 // 32  # the head keeps the share of a step that it has in the whole model
MOST_WEIGHTS = 8192 * 8192
MOST_FLOPS = 2 * 2048 * 14336 * 4096


def _linear(name, m, n, k, bits, group, dtype):
    return {"name": name, "kind": "linear", "m": m, "n": n, "k": k, "bits": bits, "group": group, "dtype": dtype}


def listed():
    return [
        # one token through the narrowest layer of a model: what a chat with one user does most often
        _linear("kv_1_b4", 1, 1024, 4096, 4, 128, "fp16"),
        # four sequences through the layer with the longest sums, at the lowest bitwidth
        _linear("down_4_b2", 4, 4096, 14336, 2, 128, "bf16"),
        # sizes that are not multiples of anything large (pruned or otherwise odd models), small groups
        _linear("ragged_13_b3", 13, 2064, 2944, 3, 32, "fp16"),
        # a serving batch
        _linear("qo_40_b6", 40, 4096, 4096, 6, 128, "bf16"),
        # a short prompt through a large layer at the master bitwidth, one scale per row
        _linear("square8k_300_b8", 300, 8192, 8192, 8, -1, "fp16"),
        # a long prompt: the dense contraction
        _linear("gate_2048_b4", 2048, 14336, 4096, 4, 128, "bf16"),
        # fused q, k, v with a bitwidth each, a batch of 16
        {"name": "qkv_16_mixed", "kind": "grouped", "m": 16, "n0": 4096, "n1": 1024, "n2": 1024, "b0": 3, "b1": 6, "b2": 4,
         "k": 4096, "group": 128, "dtype": "bf16"},
        # a checkpoint with zero points, a short prompt
        {"name": "zeros_128_b4", "kind": "zeros", "m": 128, "n": 4096, "k": 4096, "bits": 4, "group": 128, "dtype": "fp16"},
        # a layer is loaded, or switched to another bitwidth
        {"name": "repack_8_to_3", "kind": "repack", "n": 14336, "k": 4096, "bits": 3},
        # decode steps: one user, and a full serving batch
        {"name": "decode_1", "kind": "decode", "batch": 1, "layers": 4, "mean_bits": 3.0, "context": 192, "max_seq": 256,
         "dtype": "fp16"},
        {"name": "decode_32", "kind": "decode", "batch": 32, "layers": 4, "mean_bits": 3.0, "context": 192, "max_seq": 256,
         "dtype": "bf16"},
        # one prompt of 512 tokens
        {"name": "prefill_512", "kind": "prefill", "batch": 1, "seq": 512, "layers": 4, "mean_bits": 3.5, "max_seq": 768,
         "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over the logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def _width(rng, step, lo, hi):
    return max(lo, _log(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choices(("linear", "grouped", "zeros", "repack", "decode", "prefill"), (8, 3, 2, 1, 2, 1))[0]
    dtype, group = rng.choice(("fp16", "bf16")), rng.choice((128, 128, 128, 32, -1))
    if kind in ("decode", "prefill"):
        case = {"kind": kind, "layers": rng.randint(2, 4), "mean_bits": rng.choice((3.0, 3.5, 4.0, 6.0)), "dtype": dtype}
        if kind == "decode":
            max_seq = rng.choice((256, 512, 768))
            return {**case, "batch": _log(rng, 1, 32), "context": rng.randint(16, max_seq - 1), "max_seq": max_seq}
        batch = rng.choice((1, 1, 2, 4))
        return {**case, "batch": batch, "seq": _log(rng, 16, 512 // batch), "max_seq": rng.choice((512, 768))}
    while True:
        n, k = _width(rng, 16, 256, 14336), _width(rng, 128, 256, 14336)
        if n * k <= MOST_WEIGHTS:
            break
    bits = rng.choice(synth.BITWIDTHS)
    if kind == "repack":
        return {"kind": kind, "n": n, "k": k, "bits": bits}
    m = _log(rng, 1, {"linear": 2048, "grouped": 512, "zeros": 512}[kind])
    m = max(1, min(m, MOST_FLOPS // (2 * n * k)))
    case = {"kind": kind, "m": m, "k": k, "group": group, "dtype": dtype}
    if kind == "grouped":
        n1 = max(16, n // rng.choice((2, 4, 8)) // 16 * 16)
        b = [rng.choice(synth.BITWIDTHS) for _ in range(3)]
        return {**case, "n0": n, "n1": n1, "n2": n1, "b0": b[0], "b1": b[1], "b2": b[2]}
    return {**case, "n": n, "bits": bits}


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float16


def _flag(case):
    return FLAGS | (2 if case["dtype"] == "bf16" else 0)


def _model(case, seed):
    """A few layers of the 8B architecture with seeded per-layer bitwidths, its caches filled as by an earlier prompt."""
    shape = llama.LlamaShape(HIDDEN, INTER, HEADS, KV_HEADS, case["layers"], VOCAB_PER_LAYER * case["layers"])
    # the bitwidths belong to the model, not to its weights: every seed runs the same mixture
    bits = llama.mixed_bitwidths(shape, case["mean_bits"], seed=0)
    model = llama.PackedLlama(shape, bits, dtype=_dtype(case), batch=case["batch"], max_seq=case["max_seq"], seed=seed % 9973)
    return model, torch.Generator(device="cuda").manual_seed(seed + 29)


@torch.no_grad()
def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        w = synth.make_layer(case["n"], case["k"], case["group"], seed=seed, dtype=_dtype(case), device="cuda")
        layer = MatGPTQLinear.from_master(w.qweight, w.scales, 8, case["bits"], case["group"])
        x = synth.make_activations(case["m"], case["k"], seed=seed, dtype=_dtype(case), device="cuda")
        # [batch, tokens, features]: one token each for a decode batch, one prompt otherwise
        return {"kind": kind, "layer": layer, "x": x.unsqueeze(1) if case["m"] <= 32 else x.unsqueeze(0)}
    if kind == "grouped":
        x = synth.make_activations(case["m"], case["k"], seed=seed, dtype=_dtype(case), device="cuda")
        rows, bits = [case["n0"], case["n1"], case["n2"]], [case["b0"], case["b1"], case["b2"]]
        weights, scales = [], []
        for i, (n, b) in enumerate(zip(rows, bits)):
            w = synth.make_layer(n, case["k"], case["group"], seed=3 * seed + i, dtype=_dtype(case), device="cuda")
            weights.append(torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(w.qweight, n, case["k"], 8, b, case["group"], _flag(case)))
            scales.append(torch.ops.matgptq_cuda.reorder_matgptq_scales(w.scales, n, case["k"], case["group"]))
        return {"kind": kind, "args": (x, weights, scales, rows, case["k"], bits, case["group"], _flag(case))}
    if kind == "zeros":
        n, k, g = case["n"], case["k"], case["group"]
        w = synth.make_layer(n, k, g, seed=seed, sym=False, dtype=_dtype(case), device="cuda")
        x = synth.make_activations(case["m"], k, seed=seed, dtype=_dtype(case), device="cuda")
        packed = torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(w.qweight, n, k, 8, case["bits"], g, _flag(case))
        s, z = (torch.ops.matgptq_cuda.reorder_matgptq_scales(t, n, k, g) for t in (w.scales, w.zeros))
        return {"kind": kind, "args": (x, packed, s, z, n, k, case["bits"], g, _flag(case))}
    if kind == "repack":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        # master codes cluster around the zero point: weights are normal inside their group's range
        q = (torch.randn(case["n"], case["k"], generator=gen, device="cuda") * 48 + 128).round().clamp(0, 255).to(torch.uint8)
        return {"kind": kind, "args": (q, case["n"], case["k"], 8, case["bits"], 128, FLAGS)}
    model, gen = _model(case, seed)
    vocab = model.shape.vocab
    if kind == "prefill":
        tokens = torch.randint(0, vocab, (case["batch"], case["seq"]), generator=gen, device="cuda")
        return {"kind": kind, "model": model, "tokens": tokens, "positions": torch.arange(case["seq"], device="cuda")}
    for cache in model.k_cache + model.v_cache:
        cache[:, :, :case["context"]] = torch.randn(cache[:, :, :case["context"]].shape, generator=gen, device="cuda").to(cache.dtype)
    tokens = torch.randint(0, vocab, (case["batch"], 1), generator=gen, device="cuda")
    position = torch.full((1,), case["context"], dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        model.forward(tokens, position, fp32_logits=False)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            logits = model.forward(tokens, position, fp32_logits=False)
    torch.cuda.current_stream().wait_stream(stream)
    return {"kind": kind, "graph": graph, "model": model, "inputs": (tokens, position), "logits": logits}


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "grouped":
        return torch.ops.matgptq_cuda.matmul_matgptq_grouped(*state["args"])
    if kind == "zeros":
        return torch.ops.matgptq_cuda.matmul_matgptq_zeros(*state["args"])
    if kind == "repack":
        return torch.ops.matgptq_cuda.slice_pack_matgptq_qweights(*state["args"]).view(torch.int32)
    model = state["model"]
    if kind == "decode":
        state["graph"].replay()
        return {"logits": state["logits"], "k": model.k_cache, "v": model.v_cache}
    return {"logits": model.forward(state["tokens"], state["positions"]), "k": model.k_cache, "v": model.v_cache}


def _matmul_work(m, n, k, bits, group, zeros=False):
    return synth.algorithmic_bytes(n, k, m, bits, group, zeros), 2 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "repack":
        return {"bytes": case["n"] * case["k"] * (8 + case["bits"]) // 8, "flops": 0}
    if kind in ("linear", "zeros"):
        b, f = _matmul_work(case["m"], case["n"], case["k"], case["bits"], case["group"], kind == "zeros")
        return {"bytes": b, "flops": f}
    if kind == "grouped":
        parts = [_matmul_work(case["m"], case["n%d" % i], case["k"], case["b%d" % i], case["group"]) for i in range(3)]
        # the activations are read once for all parts
        return {"bytes": sum(p[0] for p in parts) - 2 * case["m"] * case["k"] * 2, "flops": sum(p[1] for p in parts)}
    # a decoder: the packed weights with their scales, the head, the keys and values of the sequences
    shape = llama.LlamaShape(HIDDEN, INTER, HEADS, KV_HEADS, case["layers"], VOCAB_PER_LAYER * case["layers"])
    sizes, bits = llama.layer_names(shape), llama.mixed_bitwidths(shape, case["mean_bits"], seed=0)
    batch, seq = case["batch"], case.get("seq", 1)
    keys = case.get("context", 0) + seq
    weights = sum(n * bits[name] / 8 + n / 128 * 2 for name, n in sizes.items()) + shape.vocab * HIDDEN * 2
    cache = case["layers"] * batch * (keys + seq) * 2 * KV_HEADS * shape.head_dim * 2
    pairs = batch * (keys if seq == 1 else seq * (seq + 1) // 2)  # query and key positions that meet
    return {"bytes": int(weights + cache),
            "flops": int(2 * batch * (seq * sum(sizes.values()) + shape.vocab * HIDDEN) + case["layers"] * 4 * pairs * HIDDEN)}


def tolerance(case):
    if case["kind"] == "repack":
        return "exact"
    if case["kind"] in ("decode", "prefill"):
        # a chain of layers, every intermediate rounded to the model's type
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
    # one product: its inputs and result rounded to the type, the weights too where the kernel builds them densely
    return {"rel": 5e-3 if case["dtype"] == "bf16" else 1e-3}
