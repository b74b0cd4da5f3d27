"""The work whose speed is measured: passes of the quantised KV cache as a serving engine makes them.

A case names one operation of the cache at one size:

  decode   one decode step: in each of `layers` layers, append the newest token and attend one query over the cache
  batch    one decode call over `batch` independent sequences of different lengths
  verify   one draft-verify step: in each layer, append `tokens` rows and attend them causally
  prefill  one prompt chunk of `tokens` rows over a prefix of `ctx` tokens: quantise-append, then causal attention
  append   the quantise-append of `tokens` rows alone

Shapes are the ones of this repository's workloads and tests: 24 query heads over 4 KV heads (others: 32 over 8, 16 over
2), head_dim 128 (the benchmark's) or 256 (the engine's own), fp16 or bf16 rows, caches written without variance balancing
(`iters` 0, the bit-exact regime) or with the engine's default of 16 iterations.  Keys and values are N(0, 1) with
channels {3, 17, 64, 101} of every 128 scaled by 20; page tables are shuffled.
"""
import math

import torch

import __graft_entry__ as entry

PAGE, TILE = 64, 128
OUTLIERS = (3, 17, 64, 101)


def _case(name, op, ctx, tokens=1, layers=1, head_dim=128, heads=(4, 24), dtype="fp16", iters=0, batch=0):
    return {"name": name, "op": op, "ctx": ctx, "tokens": tokens, "layers": layers, "head_dim": head_dim, "kv_heads": heads[0],
            "q_heads": heads[1], "dtype": dtype, "iters": iters, "batch": batch}


def listed():
    return [
        # the first tokens of an answer to a short question: every layer's calls are a few microseconds of latency
        _case("decode_1500", "decode", 1500, layers=16),
        # an ordinary long chat, all 16 attention layers of a step
        _case("decode_32768", "decode", 32768, layers=16),
        # the longest context the engine serves: KV of a layer is twice the L2
        _case("decode_378944", "decode", 378944, layers=2),
        # the engine's own geometry and default cache: head_dim 256, bf16 rows, balanced tiles, an odd length
        _case("decode_d256_30011", "decode", 30011, layers=16, head_dim=256, dtype="bf16", iters=16),
        # many users at once, 16K..131K tokens each
        _case("batch_32", "batch", 131072, batch=32),
        # speculative decoding: 3 drafts and the token before them
        _case("verify_4_131072", "verify", 131072, tokens=4, layers=4),
        # ... 7 drafts, a balanced bf16 cache of odd length
        _case("verify_8_100003", "verify", 100003, tokens=8, layers=4, dtype="bf16", iters=16),
        # ... 4 drafts in the engine's own geometry
        _case("verify_5_d256_20000", "verify", 20000, tokens=5, layers=8, head_dim=256, dtype="bf16", iters=16),
        # a chunk late in a very long prompt: the dense contraction
        _case("prefill_1024_262144", "prefill", 262144, tokens=1024),
        # a chunk of an ordinary prompt in the engine's own geometry
        _case("prefill_1024_d256_16384", "prefill", 16384, tokens=1024, head_dim=256, dtype="bf16", iters=16),
        # a short prompt of ragged length, nothing cached before it
        _case("prefill_777", "prefill", 0, tokens=777),
        # the append alone, as it runs beside the attention of another engine: balanced tiles
        _case("append_1024", "append", 4096, tokens=1024, layers=1, head_dim=256, dtype="bf16", iters=16),
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("decode", "decode", "batch", "verify", "verify", "prefill", "prefill", "append"))
    head_dim = 128 if op == "batch" else rng.choice((128, 128, 256))
    c = _case("", op, 0, head_dim=head_dim, heads=rng.choice(((4, 24), (4, 24), (4, 24), (8, 32), (2, 16))), dtype=rng.choice(("fp16", "bf16")),
              iters=0 if op == "batch" else rng.choice((0, 16)))
    del c["name"]
    if op == "batch":
        c.update(batch=rng.randint(2, 48), ctx=_between(rng, 4096, 131072))
    elif op == "append":
        c.update(ctx=TILE * rng.randint(0, 64), tokens=_between(rng, 1, 4096))
    elif op == "prefill":  # prefixes are whole chunks; at 256 dims they stay shorter
        longest = (256 if head_dim == 128 else 16) * 24 // max(24, c["q_heads"])
        c.update(ctx=1024 * (_between(rng, 1, longest + 1) - 1), tokens=_between(rng, 32, 1024))
    else:
        c.update(ctx=_between(rng, 300, 378000 if head_dim == 128 else 131072), tokens=1 if op == "decode" else rng.randint(2, 8))
        c.update(layers=max(1, min(8, 800000 * 128 // (c["ctx"] * head_dim))))
    return c


class _Gen:
    """Keys, values and queries of one seed."""

    def __init__(self, case, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        self.dim, self.dtype = case["head_dim"], torch.bfloat16 if case["dtype"] == "bf16" else torch.float16

    def rows(self, *shape):
        return torch.randn((*shape, self.dim), generator=self.g, device="cuda").to(self.dtype)

    def kv_rows(self, tokens, heads):
        x = torch.randn((tokens, heads, self.dim), generator=self.g, device="cuda")
        for s in range(0, self.dim, 128):
            for ch in OUTLIERS:
                x[:, :, s + ch] *= 20.0
        return x.to(self.dtype)

    def table(self, pages):
        return torch.randperm(pages, generator=self.g, device="cuda").to(torch.int32)


def _positions(begin, n):
    return torch.arange(begin, begin + n, dtype=torch.int32, device="cuda")


def _layer(case, gen, cached, room):
    """A cache of `cached` tokens with pages for `room` more."""
    pages = 2 * ((cached + room + TILE - 1) // TILE + 1)
    layer = entry.load_package().KvarnLayer(case["head_dim"], case["kv_heads"], case["q_heads"], pages, gen.table(pages), dtype=gen.dtype,
                                            sinkhorn_iters=case["iters"])
    for at in range(0, cached, 8192):
        n = min(8192, cached - at)
        layer.append(gen.kv_rows(n, case["kv_heads"]), gen.kv_rows(n, case["kv_heads"]), _positions(at, n))
    return layer


def _lengths(case):
    """Lengths of a batch's sequences: evenly spread from an eighth of the longest up to it, ragged."""
    n, longest = case["batch"], case["ctx"]
    return [max(1, longest // 8 + (longest - longest // 8) * (i + 1) // n - 37 * i % 128) for i in range(n)]


def prepare(case, seed):
    gen = _Gen(case, seed)
    op, ctx, tokens, kv, qh = case["op"], case["ctx"], case["tokens"], case["kv_heads"], case["q_heads"]
    state = {"op": op, "scale": 1.0 / math.sqrt(case["head_dim"])}
    if op == "batch":
        lengths = _lengths(case)
        layers = [_layer(case, gen, n, 0) for n in lengths]
        state.update(batch=entry.load_package().DecodeBatch(layers, lengths), q=gen.rows(len(lengths), qh),
                     pos=torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda"))
        return state
    state["layers"] = [_layer(case, gen, ctx, tokens) for _ in range(case["layers"])]
    state["k"] = [gen.kv_rows(tokens, kv) for _ in state["layers"]]
    state["v"] = [gen.kv_rows(tokens, kv) for _ in state["layers"]]
    state["q"] = [gen.rows(qh) if op == "decode" else gen.rows(tokens, qh) for _ in state["layers"]]
    state["pos"] = _positions(ctx, tokens)
    state["bound"] = ctx + tokens
    # the planes change too where the pass completes a tile
    state["planes"] = op in ("prefill", "append") or ctx // TILE != (ctx + tokens) // TILE
    return state


def run(state):
    op, scale = state["op"], state["scale"]
    if op == "batch":
        return state["batch"].attn_decode(state["q"], state["pos"], scale)
    outs = []
    for layer, q, k, v in zip(state["layers"], state["q"], state["k"], state["v"]):
        if op == "decode":
            outs.append(layer.append_decode(q, k, v, state["pos"], scale, state["bound"]))
        elif op == "verify":
            outs.append(layer.attn_verify(q, k, v, state["pos"], scale, state["bound"]))
        elif op == "prefill":
            outs.append(layer.attn_prefill(q, k, v, state["pos"], scale, state["bound"]))
        else:
            layer.append(k, v, state["pos"])
    result = {"out": outs, "stage": [layer.stage for layer in state["layers"]]}
    if state["planes"]:
        result["planes"] = [[layer.k_code, layer.k_scale, layer.v_code, layer.v_scale] for layer in state["layers"]]
    return result


def _attention_bytes(case, length):
    """Codes and axes of every sealed token, fp16 rows of the open tile, one page id per page."""
    d, kv = case["head_dim"], case["kv_heads"]
    sealed = length // TILE * TILE
    return sealed * kv * (d + 12 * (d // 128)) + (length - sealed) * kv * 4 * d + 4 * ((length + PAGE - 1) // PAGE)


def work(case):
    d, kv, qh, ctx, tokens = case["head_dim"], case["kv_heads"], case["q_heads"], case["ctx"], case["tokens"]
    if case["op"] == "batch":
        lengths = _lengths(case)
        return {"bytes": sum(_attention_bytes(case, n) for n in lengths) + 4 * len(lengths) * qh * d, "flops": 4 * qh * d * sum(lengths)}
    completed = (ctx + tokens) // TILE - ctx // TILE
    left = (ctx + tokens) % TILE  # rows of the open tile; a pass keeps the tile before it in the stage too
    staged = min(tokens, left + TILE if completed else left)
    append = 4 * tokens * kv * d + 4 * staged * kv * d + completed * TILE * kv * (d + 12 * (d // 128))
    if case["op"] == "append":
        return {"bytes": append, "flops": 2 * tokens * kv * d * int(math.log2(d))}
    attend = _attention_bytes(case, ctx + tokens) + 4 * tokens * qh * d
    return {"bytes": case["layers"] * (append + attend), "flops": case["layers"] * 4 * qh * d * (tokens * ctx + tokens * (tokens + 1) // 2)}


def tolerance(case):
    """About four times what was measured on B200.

    Balanced caches: the balancing keeps the best of its iterations, and sums in another order (or in 64 bits) choose another
    one of nearly equal ones.  The codes stay (2.9e-6 of the bytes differ; one byte of the smallest plane is 3e-5), but the
    fp16 axes are then rounded elsewhere: 1.2e-2 of the axes, up to 7.1e-3 of an attention output over such a cache
    (largest difference 0.14).  Unbalanced caches are bit-exact; their attention is compared with attention in 64 bits over
    the de-quantised cache, which at head_dim 256 differs by the rounding of the output alone, at 128 by the tile weights
    and operands kept in 16 bits.
    """
    if case["iters"]:
        return {"rel": 0.028, "max": 0.55, "differ": 1e-4}
    if case["op"] == "append":
        return "exact"
    bf16 = case["dtype"] == "bf16"
    if case["head_dim"] == 256:
        return {"rel": 7e-3, "max": 0.016} if bf16 else {"rel": 9e-4, "max": 2e-3}
    if case["op"] in ("decode", "batch"):
        return {"rel": 8e-3, "max": 0.023} if bf16 else {"rel": 1.7e-3, "max": 0.025}
    return {"rel": 8e-3, "max": 0.15} if bf16 else {"rel": 4e-3, "max": 0.15}
