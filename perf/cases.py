"""The work that users of this package have it do, as measurable cases through its public entry points.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs, weights, workspace),
``run`` is one call, ``work`` what the call cannot do without and ``tolerance`` how far two correct implementations of
the same precision may lie apart.  Weights are uniform random trellis words (any bit string is a valid tile) with
+-1 input signs and output scales that keep activations near one; activations are N(0, 1), as after a norm.

Kinds:
  linear   ``Exl3Linear.forward_device``: one projection on device buffers, any row count, fp16 / bf16 / fp32
  group    ``Exl3Group.forward_device``: projections that share their input ([q|k|v], [gate|up])
  mlp      ``DenseMlp.forward_device``: [gate|up], SwiGLU, down
  moe      ``Exl3SwitchGlu.forward_device``: the grouped-expert block on given routes
  stack    ``Exl3Stack.forward``: the projections of a decode step as one object
  decoder  ``DenseDecoder``: set the token, replay the recorded step, read the arg-max
  host     ``Exl3Linear.forward``: one projection with numpy arrays in and out
"""
import math

import numpy as np
import torch

import mlxl3_b200 as ex
from mlxl3_b200.decoder import DecoderConfig, DenseDecoder, DenseMlp

DTYPES = {"f16": (torch.float16, ex.F16, 2), "bf16": (torch.bfloat16, ex.BF16, 2), "f32": (torch.float32, ex.F32, 4)}


def listed():
    return [
        # decode of one token: the o projection of a Llama-3-8B-shaped layer
        {"name": "linear-1row", "kind": "linear", "in": 4096, "out": 4096, "k": 4, "cb": 0, "rows": 1, "dtype": "f16", "bias": False,
         "exact": False},
        # a few tokens at once (small batch, draft tokens) of a small odd-sized layer with a bias, bf16, the MCG codebook
        {"name": "linear-3rows-bf16", "kind": "linear", "in": 2176, "out": 1408, "k": 5, "cb": 1, "rows": 3, "dtype": "bf16",
         "bias": True, "exact": False},
        # the same decode through the array interface: host rows in, host rows out
        {"name": "host-8rows", "kind": "host", "in": 4096, "out": 4096, "k": 4, "cb": 0, "rows": 8, "dtype": "f16", "bias": False,
         "exact": False},
        # speculative verify, 16 draft tokens: [gate|up] of a Qwen3-32B-shaped layer
        {"name": "group-16rows", "kind": "group", "in": 5120, "outs": "25600,25600", "k": 3, "cb": 0, "rows": 16, "dtype": "f16"},
        # batched decode: 64 sequences, fp32 activations, bit-exact weights
        {"name": "linear-64rows-f32", "kind": "linear", "in": 4096, "out": 14336, "k": 4, "cb": 0, "rows": 64, "dtype": "f32",
         "bias": False, "exact": True},
        # prefill of 512 tokens: the dense MLP block
        {"name": "mlp-512rows", "kind": "mlp", "hidden": 4096, "ffn": 14336, "k": 3, "cb": 0, "rows": 512},
        # prefill of a ragged long prompt: [q|k|v]
        {"name": "group-1999rows", "kind": "group", "in": 4096, "outs": "4096,1024,1024", "k": 6, "cb": 0, "rows": 1999, "dtype": "f16"},
        # one token through the expert block of a Qwen3-30B-A3B-shaped layer
        {"name": "moe-1token", "kind": "moe", "experts": 128, "top_k": 8, "in": 2048, "hidden": 768, "k": 3, "cb": 0, "tokens": 1},
        # a batch of 37 sequences through the same block
        {"name": "moe-37tokens", "kind": "moe", "experts": 128, "top_k": 8, "in": 2048, "hidden": 768, "k": 3, "cb": 0, "tokens": 37},
        # prefill of 256 tokens through the same block
        {"name": "moe-256tokens", "kind": "moe", "experts": 128, "top_k": 8, "in": 2048, "hidden": 768, "k": 3, "cb": 0, "tokens": 256},
        # the projections of eight Llama-3-8B-shaped blocks, one row, as one object
        {"name": "stack-8blocks", "kind": "stack", "blocks": 8, "hidden": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336, "k": 4,
         "cb": 0, "rows": 1},
        # one generated token of the whole Llama-3-8B-shaped model at a context of 2048
        {"name": "decoder-2048", "kind": "decoder", "layers": 32, "hidden": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336,
         "vocab": 128256, "k": 4, "cb": 0, "context": 2048},
    ]


def _log(rng, lo, hi, step=1):
    """A whole multiple of `step` between `lo` and `hi`, spread evenly over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "group", "mlp", "moe", "moe", "stack", "decoder", "host"])
    k, cb = rng.choice([2, 3, 3, 4, 4, 4, 5, 6, 8]), rng.choice([0, 0, 0, 0, 1, 2])
    if kind in ("linear", "host"):
        return {"kind": kind, "in": _log(rng, 512, 14336, 128), "out": _log(rng, 512, 25600, 128), "k": k, "cb": cb,
                "rows": _log(rng, 1, 2048 if kind == "linear" else 64), "dtype": rng.choice(["f16", "f16", "bf16", "f32"]),
                "bias": rng.random() < 0.25, "exact": rng.random() < 0.25}
    if kind == "group":
        if rng.random() < 0.5:
            q = _log(rng, 512, 8192, 128)
            outs = [q, max(128, q // rng.choice([1, 2, 4, 8]) // 128 * 128)]
            outs.append(outs[1])
        else:
            outs = [_log(rng, 512, 25600, 128)] * 2
        return {"kind": kind, "in": _log(rng, 512, 8192, 128), "outs": ",".join(map(str, outs)), "k": k, "cb": cb,
                "rows": _log(rng, 1, 2048), "dtype": rng.choice(["f16", "f16", "bf16", "f32"])}
    if kind == "mlp":
        return {"kind": kind, "hidden": _log(rng, 512, 5120, 128), "ffn": _log(rng, 1024, 25600, 128), "k": k, "cb": cb,
                "rows": _log(rng, 1, 1024)}
    if kind == "moe":
        experts = rng.choice([8, 32, 60, 64, 128])
        n_in, hidden = _log(rng, 512, 4096, 128), _log(rng, 256, 2048, 128)
        while experts * n_in * hidden > 128 * 2048 * 1024:
            n_in, hidden = max(512, n_in // 256 * 128), max(256, hidden // 256 * 128)
        return {"kind": kind, "experts": experts, "top_k": rng.choice([1, 2, 4, 6, 8]), "in": n_in, "hidden": hidden, "k": k,
                "cb": cb, "tokens": _log(rng, 1, 512)}
    kv_heads = rng.choice([2, 4, 8])
    shape = {"kind": kind, "hidden": _log(rng, 1024, 5120, 128), "heads": kv_heads * rng.choice([1, 2, 4, 8]), "kv_heads": kv_heads,
             "ffn": _log(rng, 2048, 16384, 128), "k": k, "cb": cb}
    if kind == "stack":
        return {**shape, "blocks": rng.randint(1, 8), "rows": rng.choice([1, 1, 1, 2])}
    return {**shape, "layers": rng.randint(1, 12), "vocab": _log(rng, 8192, 131072, 64), "context": _log(rng, 64, 4096)}


# ---- inputs ---------------------------------------------------------------------------------------------------------

class _Source:
    """Seeded random tensors, made on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, dtype=torch.float16):
        return torch.randn(shape, generator=self.gen, device="cuda", dtype=torch.float32).to(dtype)

    def words(self, *shape):
        """uint16 words on the host, uniform."""
        t = torch.randint(-32768, 32768, shape, generator=self.gen, device="cuda", dtype=torch.int16)
        return t.cpu().numpy().view(np.uint16)

    def signs(self, *shape, scale=1.0):
        t = torch.randint(0, 2, shape, generator=self.gen, device="cuda", dtype=torch.int16)
        return ((2 * t - 1).to(torch.float16) * scale).cpu().numpy()

    def linear(self, n_in, n_out, k, cb, bias=False, exact=False):
        return ex.Exl3Linear(self.words(n_in // 16, n_out // 16, 16 * k), self.signs(n_in), self.signs(n_out, scale=_svh(n_in)),
                             self.normal(n_out).cpu().numpy() if bias else None, k, cb, exact_weights=exact)


def _svh(n_in):
    return 1.0 / (1.2437 * math.sqrt(n_in))          # 1.2437: standard deviation of a decoded weight


def _outs(case):
    return [int(n) for n in case["outs"].split(",")]


class _View:
    """A framework buffer as a torch tensor, without a copy."""

    def __init__(self, buffer, shape, typestr):
        self.buffer = buffer
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (buffer.ptr, False), "version": 3}


def _tensor(buffer, shape, typestr="<f2"):
    return torch.as_tensor(_View(buffer, shape, typestr), device="cuda")


class _ModelWeights:
    """Weights of a decoder, projection by projection.  The trellises are runs of one block of random words, each from
    a place of its own; embedding and head are tied, as in small models."""

    def __init__(self, config, seed):
        self.config, self.source = config, _Source(seed)
        c = config
        self.most = max(c.hidden, c.heads * c.head_dim) * max(c.ffn, c.hidden) // 16 * c.k_bits
        self.block = self.source.words(2 * self.most)
        self.places = np.random.default_rng(seed)
        self.table = (self.source.normal(c.vocab, c.hidden) * (1.0 / math.sqrt(c.hidden))).cpu().numpy()

    def projection(self, layer, name):
        c = self.config
        q, kv = c.heads * c.head_dim, c.kv_heads * c.head_dim
        n_in, n_out = {"q": (c.hidden, q), "k": (c.hidden, kv), "v": (c.hidden, kv), "o": (q, c.hidden), "gate": (c.hidden, c.ffn),
                       "up": (c.hidden, c.ffn), "down": (c.ffn, c.hidden)}[name]
        count = n_in * n_out // 16 * c.k_bits
        at = int(self.places.integers(0, self.block.size - count))
        return (self.block[at:at + count].reshape(n_in // 16, n_out // 16, 16 * c.k_bits), self.source.signs(n_in),
                self.source.signs(n_out, scale=_svh(n_in)))

    def norm(self, layer, which):
        return (1.0 + 0.1 * self.source.normal(self.config.hidden)).cpu().numpy()

    def embed(self):
        return self.table

    def head(self):
        return self.table


def prepare(case, seed):
    ex.init(torch.cuda.current_device())
    ex.set_option("pdl", 1)                          # dependent launch, as the benchmark runs
    return {"linear": _prepare_linear, "host": _prepare_linear, "group": _prepare_group, "mlp": _prepare_mlp, "moe": _prepare_moe,
            "stack": _prepare_stack, "decoder": _prepare_decoder}[case["kind"]](case, seed)


def _prepare_linear(case, seed):
    source, rows = _Source(seed), case["rows"]
    kind, code, _ = DTYPES[case["dtype"]]
    layer = source.linear(case["in"], case["out"], case["k"], case["cb"], case["bias"], case["exact"])
    x = source.normal(rows, case["in"], dtype=kind)
    if case["kind"] == "host":
        x = x.view(torch.int16).cpu().numpy().view(np.uint16) if case["dtype"] == "bf16" else x.cpu().numpy()
        return {"kind": "host", "layer": layer, "x": x, "code": code}
    return {"kind": "linear", "layer": layer, "x": x, "code": code, "rows": rows, "y": torch.empty(rows, case["out"], dtype=kind, device="cuda"),
            "workspace": ex.new_workspace(layer.workspace_bytes(rows))}


def _prepare_group(case, seed):
    source, rows = _Source(seed), case["rows"]
    kind, code, _ = DTYPES[case["dtype"]]
    group = ex.Exl3Group([source.linear(case["in"], n, case["k"], case["cb"]) for n in _outs(case)])
    return {"kind": "group", "group": group, "x": source.normal(rows, case["in"], dtype=kind), "code": code, "rows": rows,
            "ys": [torch.empty(rows, n, dtype=kind, device="cuda") for n in _outs(case)],
            "workspace": ex.new_workspace(group.workspace_bytes(rows))}


def _prepare_mlp(case, seed):
    source, rows = _Source(seed), case["rows"]
    hidden, ffn = case["hidden"], case["ffn"]
    block = DenseMlp(*(source.linear(a, b, case["k"], case["cb"]) for a, b in ((hidden, ffn), (hidden, ffn), (ffn, hidden))))
    return {"kind": "mlp", "block": block, "x": source.normal(rows, hidden), "rows": rows,
            "y": torch.empty(rows, hidden, dtype=torch.float16, device="cuda")}


def _prepare_moe(case, seed):
    source, tokens = _Source(seed), case["tokens"]
    experts, n_in, hidden, k, top_k = case["experts"], case["in"], case["hidden"], case["k"], case["top_k"]
    block = ex.Exl3SwitchGlu(source.words(n_in // 16, experts * hidden // 8, 16 * k), source.signs(experts, 2, n_in),
                             source.signs(experts, 2, hidden, scale=_svh(n_in)), source.words(hidden // 16, experts * n_in // 16, 16 * k),
                             source.signs(experts, hidden), source.signs(experts, n_in, scale=_svh(hidden)), top_k, k, case["cb"])
    # routes as a softmax router gives them: some experts are asked for more often than others
    logits = source.normal(tokens, experts, dtype=torch.float32) + 0.5 * source.normal(1, experts, dtype=torch.float32)
    best = torch.topk(logits, top_k)
    return {"kind": "moe", "block": block, "x": source.normal(tokens, n_in), "tokens": tokens, "selected": best.indices.to(torch.int32),
            "scores": torch.softmax(best.values, 1).to(torch.float16), "y": torch.empty(tokens, n_in, dtype=torch.float16, device="cuda"),
            "workspace": ex.new_workspace(block.workspace_bytes(tokens))}


def _prepare_stack(case, seed):
    hidden, ffn, rows = case["hidden"], case["ffn"], case["rows"]
    config = DecoderConfig(layers=case["blocks"], hidden=hidden, heads=case["heads"], kv_heads=case["kv_heads"], ffn=ffn, vocab=64,
                           k_bits=case["k"], codebook=case["cb"])
    weights = _ModelWeights(config, seed)
    q, kv = 128 * case["heads"], 128 * case["kv_heads"]
    y = {n: torch.empty(rows, w, dtype=torch.float16, device="cuda")
         for n, w in (("q", q), ("k", kv), ("v", kv), ("o", hidden), ("gate", ffn), ("up", ffn), ("down", hidden))}
    x = weights.source.normal(rows, hidden)
    ops, source = [], x
    for block in range(case["blocks"]):
        one = {n: ex.Exl3Linear(*weights.projection(block, n), None, case["k"], case["cb"])
               for n in ("q", "k", "v", "o", "gate", "up", "down")}
        ops += [(ex.Exl3Group([one["q"], one["k"], one["v"]]), source.data_ptr(), [y[n].data_ptr() for n in "qkv"]),
                (one["o"], y["q"].data_ptr(), y["o"].data_ptr()),
                (ex.Exl3Group([one["gate"], one["up"]]), y["o"].data_ptr(), [y["gate"].data_ptr(), y["up"].data_ptr()]),
                (one["down"], y["gate"].data_ptr(), y["down"].data_ptr())]
        for n in ("q", "k", "v", "gate", "up"):
            one[n].close()
        source = y["down"]
    return {"kind": "stack", "stack": ex.Exl3Stack(ops, ex.F16, rows), "x": x, "y": y}


def _prepare_decoder(case, seed):
    context = case["context"]
    config = _config(case)
    weights = _ModelWeights(config, seed)
    model = DenseDecoder(config, weights)
    shape = (model.kv_heads, context, config.head_dim)
    rows = []
    for entry in model.layers:
        for name in ("k_cache", "v_cache"):
            cache = _tensor(entry[name], shape)
            cache[:, :context - 1] = weights.source.normal(model.kv_heads, context - 1, config.head_dim)
            rows.append(cache[:, context - 1])
    token = int(weights.places.integers(0, config.vocab))
    torch.cuda.synchronize()
    model.store_logits = True
    model.set_input(token, context - 1)
    model.record()
    # the cache rows that a step writes: of every layer, or of evenly spread ones where there are many
    step = -(-len(model.layers) // 24)
    rows = [r for i, r in enumerate(rows) if (i // 2) % step == 0]
    return {"kind": "decoder", "model": model, "token": token, "pos": context - 1, "rows": rows,
            "hidden": _tensor(model.buf[model.hidden_name], (config.hidden,)), "logits": _tensor(model.buf["logits"], (config.vocab,))}


def _config(case):
    return DecoderConfig(layers=case["layers"], hidden=case["hidden"], heads=case["heads"], kv_heads=case["kv_heads"], ffn=case["ffn"],
                         vocab=case["vocab"], k_bits=case["k"], codebook=case["cb"], max_ctx=case["context"])


# ---- one call -------------------------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "linear":
        s["layer"].forward_device(s["x"].data_ptr(), s["code"], s["rows"], s["y"].data_ptr(), s["workspace"])
        return s["y"]
    if kind == "host":
        y = s["layer"].forward(s["x"], s["code"])
        return torch.from_numpy(y.view(np.int16)).view(torch.bfloat16) if s["code"] == ex.BF16 else y
    if kind == "group":
        s["group"].forward_device(s["x"].data_ptr(), s["code"], s["rows"], [y.data_ptr() for y in s["ys"]], s["workspace"])
        return s["ys"]
    if kind == "mlp":
        s["block"].forward_device(s["x"].data_ptr(), s["rows"], s["y"].data_ptr())
        return s["y"]
    if kind == "moe":
        s["block"].forward_device(s["x"].data_ptr(), ex.F16, s["tokens"], s["selected"].data_ptr(), s["scores"].data_ptr(), ex.F16,
                                  s["y"].data_ptr(), s["workspace"])
        return s["y"]
    if kind == "stack":
        s["stack"].forward()
        return s["y"]                                # of the last block: the blocks share their buffers
    # a generation loop hands the token over, replays the step and reads the winner; the winner's index follows from the
    # logits (two logits may tie within the rounding of the layers below, so the index itself is not compared)
    model = s["model"]
    model.set_input(s["token"], s["pos"])
    model.step()
    value, _ = model.result()
    return {"best": value, "logits": s["logits"], "hidden": s["hidden"], "cache_rows": s["rows"]}


# ---- what a call cannot do without ----------------------------------------------------------------------------------

def _projection(n_in, n_out, k, rows, size=2):
    """Packed weights and scale vectors once, activations in and out once."""
    return n_in * n_out * k // 8 + 2 * (n_in + n_out) + rows * (n_in + n_out) * size, 2 * rows * n_in * n_out


def work(case):
    kind, k = case["kind"], case["k"]
    if kind in ("linear", "host"):
        parts = [_projection(case["in"], case["out"], k, case["rows"], DTYPES[case["dtype"]][2])]
    elif kind == "group":
        outs, size = _outs(case), DTYPES[case["dtype"]][2]
        parts = [_projection(case["in"], n, k, case["rows"], size) for n in outs]
        parts.append((-(len(outs) - 1) * case["rows"] * case["in"] * size, 0))                      # the input is read once
    elif kind == "mlp":
        h, f, rows = case["hidden"], case["ffn"], case["rows"]
        parts = [((3 * h * f * k) // 8 + 6 * (h + f) + 4 * rows * h, 6 * rows * h * f)]             # nothing between has to leave the chip
    elif kind == "moe":
        e, t, h, f = case["experts"], case["tokens"], case["in"], case["hidden"]
        touched = e * (1.0 - (1.0 - case["top_k"] / e) ** t)                                        # experts that some token asks for
        parts = [(touched * (3 * h * f * k / 8 + 2 * (3 * h + 3 * f)) + t * (4 * h + 6 * case["top_k"]), 6 * t * case["top_k"] * h * f)]
    else:
        h, f, rows = case["hidden"], case["ffn"], case.get("rows", 1)
        q, kv = 128 * case["heads"], 128 * case["kv_heads"]
        block = [_projection(a, b, k, rows) for a, b in ((h, q), (h, kv), (h, kv), (q, h), (h, f), (h, f), (f, h))]
        if kind == "decoder":
            block.append((4 * kv * case["context"], 4 * q * case["context"]))
        n = case["blocks"] if kind == "stack" else case["layers"]
        parts = [(n * sum(b for b, _ in block), n * sum(w for _, w in block))]
        if kind == "decoder":
            parts.append((2 * case["vocab"] * (h + 1), 2 * case["vocab"] * h))
    return {"bytes": sum(b for b, _ in parts), "flops": sum(w for _, w in parts)}


def tolerance(case):
    """Outputs are rounded to fp16 (2^-11) or bf16 (2^-8) after an fp16 rotation, whatever their type, so 32-bit rows
    carry fp16 results; blocks chain several such roundings and models chain blocks."""
    kind = case["kind"]
    if kind in ("linear", "host", "group"):
        return {"rel": 6e-3 if case["dtype"] == "bf16" else 2e-3}
    if kind in ("mlp", "moe"):
        return {"rel": 4e-3}
    return {"rel": 2e-2, "max": 0.25}
