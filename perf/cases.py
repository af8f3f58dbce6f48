"""What is measured: the decode step and the single kernels behind it, as a user's program calls them.

Two ways into the framework are covered.  A server drives `Engine.decode`: the whole captured step of the
27B-shaped hybrid model (64 layers, three DeltaNet layers to one attention layer, NVFP4 projections, e4m3
vocabulary tables) over a ragged batch of up to 32 rows.  A program with an executor of its own calls
the kernels one by one through the C ABI (`qwencore_b200.ops`), eagerly, on its own stream.

Shapes, number formats and distributions are those of the benchmark configurations, the tests and
`qwencore_b200/synth.py`.  Everything is drawn on the GPU from the seed.
"""

import math

import numpy as np
import torch

from qwencore_b200 import abi, engine, ops

HIDDEN, INTERMEDIATE, VOCAB = 5120, 17408, 151936

# (rows, columns) of the model's projections with 32 and with 48 value heads, and the small ones of the tests
MATRICES = [(34816, 5120), (5120, 17408), (12352, 5120), (16480, 5120), (14336, 5120), (5120, 6144), (5120, 4096),
            (1040, 512), (264, 256)]


def listed():
    return [
        # a server under load: 32 requests of very different ages, the benchmark's own step
        {"name": "step_c32_loguniform", "kind": "step", "rows": 32, "low": 128, "high": 32768, "heads": 32, "page": 16,
         "layers": 64},
        # one interactive user: the latency of a token at context 2048
        {"name": "step_c1_2k", "kind": "step", "rows": 1, "low": 2048, "high": 2048, "heads": 32, "page": 16, "layers": 64},
        # a partly filled batch of short chats, with the reference's own dimensions (48 value heads, pages of 64)
        {"name": "step_c9_short_v48", "kind": "step", "rows": 9, "low": 128, "high": 2048, "heads": 48, "page": 64,
         "layers": 64},
        # a few requests over long documents: attention outweighs the projections
        {"name": "step_c20_long", "kind": "step", "rows": 20, "low": 8192, "high": 32768, "heads": 32, "page": 16,
         "layers": 64},
        # a single NVFP4 matrix-vector product, the width of the fused gate and up projection
        {"name": "projection_m1_34816x5120", "kind": "projection", "rows": 1, "out": 34816, "in": 5120},
        # a narrow output with a long sum at an odd batch: the MLP's down projection
        {"name": "projection_m13_5120x17408", "kind": "projection", "rows": 13, "out": 5120, "in": 17408},
        # the gate and up pair with SwiGLU at the full batch
        {"name": "swiglu_m32_17408x5120", "kind": "swiglu", "rows": 32, "out": 17408, "in": 5120},
        # packed attention over a ragged batch of chats
        {"name": "attention_c32_uniform", "kind": "attention", "rows": 32, "low": 128, "high": 2048, "page": 16,
         "gated": False, "scaled": True},
        # ... and over three long contexts, gated, pages of 64
        {"name": "attention_c3_long", "kind": "attention", "rows": 3, "low": 16001, "high": 32768, "page": 64,
         "gated": True, "scaled": False},
        # the recurrent update of 32 slots through eight layers (as many as L2 does not hold)
        {"name": "delta_c32_v32", "kind": "delta", "rows": 32, "heads": 32, "layers": 8},
        # the smallest call of a step: one slot's recurrent update
        {"name": "delta_c1_v48", "kind": "delta", "rows": 1, "heads": 48, "layers": 1},
        # the vocabulary head and greedy sampling at an odd batch
        {"name": "head_m5_argmax", "kind": "head", "rows": 5, "vocab": VOCAB, "in": HIDDEN},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "projection", "swiglu", "attention", "delta", "head"])
    rows = rng.randint(1, 32)
    if kind == "step":
        high = _log_int(rng, 256, 32768)
        low = _log_int(rng, 128, high)
        while rows > 1 and rows * (low + high) > 400000:  # no more tokens than the listed cases attend to
            rows -= 1
        return {"kind": kind, "rows": rows, "low": low, "high": high, "heads": rng.choice([32, 48]),
                "page": rng.choice([16, 64]), "layers": 4 * _log_int(rng, 1, 15)}
    if kind == "projection":
        out, width = rng.choice(MATRICES)
        return {"kind": kind, "rows": rows, "out": out, "in": width}
    if kind == "swiglu":
        return {"kind": kind, "rows": rows, "out": 8 * _log_int(rng, 64, INTERMEDIATE // 8),
                "in": 256 * _log_int(rng, 2, HIDDEN // 256)}
    if kind == "attention":
        high = _log_int(rng, 64, 32768)
        low = _log_int(rng, 1, high)
        while rows > 1 and rows * (low + high) > 400000:
            rows -= 1
        return {"kind": kind, "rows": rows, "low": low, "high": high, "page": rng.choice([16, 64]),
                "gated": rng.random() < 0.5, "scaled": rng.random() < 0.5}
    if kind == "delta":
        return {"kind": kind, "rows": rows, "heads": rng.choice([32, 48]), "layers": _log_int(rng, 1, 8)}
    return {"kind": kind, "rows": rows, "vocab": 8 * _log_int(rng, 1000, VOCAB // 8),
            "in": rng.choice([512, 2048, HIDDEN])}


# ---- inputs ----------------------------------------------------------------------------------------------

class _Device:
    """A tensor of the engine as torch sees it; holds the engine, whose memory it is."""

    def __init__(self, handle, name, layer, shape, typestr):
        self.handle = handle
        pointer, _ = handle.tensor_ptr(name, layer)
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (pointer, False), "version": 3}


def _contexts(case, seed):
    """Log-uniform lengths in [low, high]; the longest one is always there."""
    rng = np.random.default_rng([seed, 7])
    low, high = math.log(case["low"]), math.log(case["high"])
    contexts = np.exp(rng.uniform(low, high, case["rows"])).astype(np.int64).clip(case["low"], case["high"])
    contexts[rng.integers(case["rows"])] = case["high"]
    return contexts


def _expected_tokens(case):
    low, high = case["low"], case["high"]
    mean = low if low == high else (high - low) / math.log(high / low)
    return (case["rows"] - 1) * mean + high


def _generator(seed):
    generator = torch.Generator(device="cuda")
    generator.manual_seed(seed)
    return generator


def _bf16(shape, generator, std=1.0):
    return (torch.randn(shape, device="cuda", generator=generator) * std).to(torch.bfloat16)


def _linear(out, width, generator):
    """Codes uniform over the 16 e2m1 values; block scales |N(0,1)| * 0.05 rounded to e4m3."""
    packed = torch.randint(0, 256, (out, width // 2), dtype=torch.uint8, device="cuda", generator=generator)
    count = ops.block_scale_storage_len(out, width)
    scales = torch.randn(count, device="cuda", generator=generator).abs_().mul_(0.05).to(torch.float8_e4m3fn)
    return ops.Linear(packed, scales.view(torch.uint8), 1.0, out, width)


def _prepare_step(case, seed):
    contexts = _contexts(case, seed)
    page, rows, layers = case["page"], case["rows"], case["layers"]
    blocks = (contexts + page - 1) // page
    handle = engine.Engine(engine.default_config(
        num_layers=layers, delta_value_heads=case["heads"], kv_page_size=page, max_batch=rows,
        max_context=-(-case["high"] // 1024) * 1024, kv_pool_blocks=int(blocks.sum()) + 1, state_slots=rows + 1,
        write_logits=1, seed=seed))
    # Divisors as a loader sets them: the inner projections keep the scale of what they read; the two that
    # write the residual stream are scaled down with depth, so that 64 random layers do not amplify the
    # last bit of a bf16 activation beyond what logits can be compared at.
    for layer in range(layers):
        full = (layer + 1) % 4 == 0
        for name in ("gate", "up", "qkv" if full else "in_proj"):
            handle.set_weight_global_scale(name, layer, 32.0)
        for name in ("down", "o" if full else "la_out"):
            handle.set_weight_global_scale(name, layer, 262144.0)
    rng = np.random.default_rng([seed, 9])
    slots = rng.permutation(rows + 1)[:rows].astype(np.uint32)
    pages = rng.permutation(int(blocks.sum()) + 1)
    first = 0
    for slot, context, count in zip(slots, contexts, blocks):
        handle.install_sequence(int(slot), int(context), pages[first:first + count])
        first += int(count)
    tokens = rng.integers(0, VOCAB, rows).astype(np.uint32)
    # what the cache manager hands over with a step: the length of every row's sequence
    edits = np.array([(slot, 0, context, 1) for slot, context in zip(slots, contexts)], dtype=np.uint32)
    views = {"logits": torch.as_tensor(_Device(handle, "logits", 0, (rows, VOCAB), "<f4"), device="cuda")}
    for layer in range(layers):
        if (layer + 1) % 4 != 0:
            views["state_scales.%d" % layer] = torch.as_tensor(
                _Device(handle, "state_scales", layer, (rows + 1, case["heads"], 128), "<f4"), device="cuda")
    for _ in range(2):  # a server's engine has its step captured: the first step runs eagerly, the second captures
        handle.decode(slots, tokens, edits)
    return {"kind": "step", "engine": handle, "slots": slots, "tokens": tokens, "edits": edits, "views": views}


def _prepare_attention(case, seed, generator):
    contexts = _contexts(case, seed)
    page, rows = case["page"], case["rows"]
    blocks = (contexts + page - 1) // page
    pool, widest = int(blocks.sum()) + 3, int(blocks.max())
    tables = np.zeros((rows, widest), dtype=np.int32)
    pages = np.random.default_rng([seed, 11]).permutation(pool)
    first = 0
    for row, count in enumerate(blocks):
        tables[row, :count] = pages[first:first + count]
        first += int(count)
    state = {"kind": "attention", "rows": rows, "page": page, "widest": widest,
             "tables": torch.from_numpy(tables).cuda(), "contexts": torch.from_numpy(contexts.astype(np.int32)).cuda(),
             "query": _bf16((rows, ops.NUM_ATTN_HEADS, ops.ATTN_HEAD_DIM), generator), "gate": None, "scales": None,
             "output": torch.zeros((rows, ops.NUM_ATTN_HEADS, ops.ATTN_HEAD_DIM), dtype=torch.bfloat16, device="cuda")}
    if case["gated"]:
        state["gate"] = _bf16((rows, ops.NUM_ATTN_HEADS, 2 * ops.ATTN_HEAD_DIM), generator)
    scale = torch.ones(ops.NUM_KV_HEADS, device="cuda")
    if case["scaled"]:
        scale = (0.5 + torch.rand(ops.NUM_KV_HEADS, device="cuda", generator=generator)) / 64.0
        state["scales"] = scale
    for name in ("keys", "values"):
        cache = torch.empty((pool, ops.NUM_KV_HEADS, page, ops.ATTN_HEAD_DIM), dtype=torch.float8_e4m3fn, device="cuda")
        for at in range(0, pool, 4096):
            part = torch.randn(cache[at:at + 4096].shape, device="cuda", generator=generator)
            cache[at:at + 4096] = part.div_(scale[None, :, None, None]).clamp_(-448, 448).to(torch.float8_e4m3fn)
        state[name] = cache.view(torch.uint8)
    state["partitions"] = ops.packed_partition_count(rows, int(contexts.max()))
    state["workspace"] = torch.zeros(max(16, ops.packed_workspace_bytes(rows, state["partitions"])), dtype=torch.uint8,
                                     device="cuda")
    return state


def _prepare_delta(case, seed, generator):
    rows, heads, layers = case["rows"], case["heads"], case["layers"]
    abi.configure(heads, abi.get_shape()[1])
    state = {"kind": "delta", "rows": rows, "capacity": rows + 1, "layers": []}
    state["slots"] = torch.randperm(rows + 1, device="cuda", generator=generator)[:rows].to(torch.int32)
    for _ in range(layers):
        values = torch.randn((rows + 1, heads, 128, 128), device="cuda", generator=generator) * 0.1
        peak = values.abs().amax(-1)
        q, k = (torch.nn.functional.normalize(_bf16((rows, 16, 128), generator).float(), dim=-1) for _ in range(2))
        q = q / math.sqrt(128.0)
        gates = torch.randn((2, rows, heads), device="cuda", generator=generator)
        state["layers"].append({
            "codes": (values * (127.0 / peak)[..., None]).round_().to(torch.int8), "scales": peak * (1.0 / 127.0),
            "q": q, "k": k, "v": _bf16((rows, heads, 128), generator).float(), "kq": (q * k).sum(-1),
            "alpha": torch.exp(-torch.nn.functional.softplus(gates[0])), "beta": torch.sigmoid(gates[1]),
            "out": torch.zeros((rows, heads, 128), device="cuda")})
    return state


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    generator = _generator(seed)
    if case["kind"] == "attention":
        return _prepare_attention(case, seed, generator)
    if case["kind"] == "delta":
        return _prepare_delta(case, seed, generator)
    rows = case["rows"]
    if case["kind"] == "head":
        vocab, width = case["vocab"], case["in"]
        weights = torch.randn((vocab, width), dtype=torch.bfloat16, device="cuda", generator=generator)
        return {"kind": "head", "rows": rows, "vocab": vocab, "in": width, "x": _bf16((rows, width), generator),
                "weights": weights.mul_(16).to(torch.float8_e4m3fn).view(torch.uint8),
                "row_scales": 0.002 + 0.002 * torch.rand(vocab, device="cuda", generator=generator),
                "logits": torch.zeros((rows, vocab), device="cuda"),
                "part_values": torch.zeros((rows, 256), device="cuda"),
                "part_indices": torch.zeros((rows, 256), dtype=torch.int32, device="cuda"),
                "tokens": torch.zeros(rows, dtype=torch.int32, device="cuda")}
    state = {"kind": case["kind"], "rows": rows, "x": _bf16((rows, case["in"]), generator),
             "matrix": _linear(case["out"], case["in"], generator),
             "out": torch.zeros((rows, case["out"]), dtype=torch.bfloat16, device="cuda")}
    if case["kind"] == "swiglu":
        state["up"] = _linear(case["out"], case["in"], generator)
        # activations after a norm through a projection that keeps their scale
        state["matrix"].weight_global_scale = state["up"].weight_global_scale = math.sqrt(case["in"]) * 0.15
    return state


# ---- one pass --------------------------------------------------------------------------------------------

def run(state):
    kind, rows = state["kind"], state.get("rows")
    if kind == "step":
        # The tokens come back to the host with every step.  They are the largest of the logits returned here;
        # beside them two logits of a random head can be closer than bf16 activations resolve.
        state["engine"].decode(state["slots"], state["tokens"], state["edits"])
        return state["views"]
    if kind == "projection":
        state["matrix"].forward_w4a16(state["x"], state["out"], rows)
        return state["out"]
    if kind == "swiglu":
        ops.swiglu_w4a16(state["matrix"], state["up"], state["x"], state["out"], rows)
        return state["out"]
    if kind == "attention":
        ops.gated_packed(state["query"], state["gate"], state["keys"], state["values"], state["tables"],
                         state["contexts"], state["widest"], state["output"], rows, 0, state["partitions"],
                         state["workspace"], state["page"], key_scales=state["scales"], value_scales=state["scales"])
        return state["output"]
    if kind == "delta":
        for layer in state["layers"]:
            ops.delta_decode_slots_packed(layer["codes"], layer["scales"], state["slots"], layer["q"], layer["k"],
                                          layer["v"], layer["alpha"], layer["beta"], layer["kq"], layer["out"],
                                          state["capacity"], rows)
        return [(layer["out"], layer["codes"], layer["scales"]) for layer in state["layers"]]
    ops.fp8_lm_head(state["weights"], state["row_scales"], state["x"], state["logits"], rows, state["in"], state["vocab"])
    ops.argmax(state["logits"], state["part_values"], state["part_indices"], state["tokens"], state["vocab"], rows)
    return {"logits": state["logits"], "tokens": state["tokens"]}


# ---- what a pass cannot do without -----------------------------------------------------------------------

def _matrix_bytes(out, width):
    return out * width // 2 + out * width // 16


def work(case):
    rows = case["rows"]
    if case["kind"] == "step":
        layers, heads = case["layers"], case["heads"]
        full = layers // 4
        weights = 3 * layers * INTERMEDIATE * HIDDEN
        weights += (layers - full) * HIDDEN * (2 * 16 * 128 + 2 * heads * 128 + 2 * heads + heads * 128)
        weights += full * HIDDEN * (2 * 24 * 256 + 2 * 4 * 256 + 24 * 256)
        tokens = _expected_tokens(case)
        state = (layers - full) * rows * heads * (128 * 128 + 512)
        nbytes = weights * 9 // 16 + VOCAB * (HIDDEN + 4) + rows * VOCAB * 4 + 2 * state + full * tokens * 2048
        flops = 2 * rows * (weights + VOCAB * HIDDEN) + full * tokens * 24 * 256 * 4 + 8 * (layers - full) * rows * heads * 128 * 128
        return {"bytes": nbytes, "flops": flops}
    if case["kind"] in ("projection", "swiglu"):
        matrices = 2 if case["kind"] == "swiglu" else 1
        return {"bytes": matrices * _matrix_bytes(case["out"], case["in"]) + 2 * rows * (case["in"] + case["out"]),
                "flops": 2 * matrices * rows * case["out"] * case["in"]}
    if case["kind"] == "attention":
        tokens = _expected_tokens(case)
        vectors = rows * 24 * 256 * 2 * (3 if case["gated"] else 2)
        return {"bytes": tokens * 2048 + vectors, "flops": tokens * 24 * 256 * 4}
    if case["kind"] == "delta":
        each = rows * case["heads"] * (2 * (128 * 128 + 512) + 2 * 512) + 2 * rows * 16 * 512
        return {"bytes": case["layers"] * each, "flops": 8 * case["layers"] * rows * case["heads"] * 128 * 128}
    return {"bytes": case["vocab"] * (case["in"] + 4) + rows * (2 * case["in"] + 4 * case["vocab"]),
            "flops": 2 * rows * case["vocab"] * case["in"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "step":
        # the same rows decoded one by one, in sixteens and all at once (other split and summation orders) give
        # logits 0.9 % apart after 64 layers: bf16 activations and int8 state codes round differently
        return {"rel": 0.03, "max": 0.6}
    if kind in ("projection", "swiglu", "attention"):
        # against float64: 1.7e-3 (half a bf16 step), worst element 4.7e-3
        return {"rel": 0.0066, "max": 0.02}
    if kind == "delta":
        # against float64: outputs 9e-8, 5e-6 of the state codes; a code that rounds the other way moves an
        # output of the next pass by up to half a percent of the outputs' RMS
        return {"rel": 5e-5, "max": 0.02, "differ": 1e-4}
    # the head in fp32 against float64: 1.9e-6, worst 9.4e-6
    return {"rel": 8e-6, "max": 4e-5}
