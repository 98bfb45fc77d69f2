"""What this engine's speed is measured on: the dense Llama / Qwen2.5 decoder, from the smallest decode step to whole prompts.

A case is a dict. Its kinds:
  decode   one decode step of `rows` requests, the step recorded as a CUDA graph and replayed, as `LLMEngine` runs its
           decode steps: metadata packed and uploaded, graph replayed, positions committed
  portions one step of `prompts` prompt portions of up to `tokens` tokens behind `prefix` cached tokens, beside `rows`
           decoded tokens, through `StepRunner.run`; the logits of the last `want` tokens of each portion
  serve    `LLMEngine`: `prompts` requests of up to `tokens` tokens in, `new` sampled tokens each out
Context lengths of a step's requests and prompt lengths are spread evenly below the longest one, so most are odd and
ragged. Weights are random at the named model's sizes, N(0, 0.02) but for the embedding, N(0, 1): the layers then add to a
stream that is there, as in a trained model, and where the embedding is also the output matrix the sampled tokens are as
certain as a trained model's. The cache holds random keys and values of the size that such weights give.
"""
import math

import numpy as np
import torch

MODELS = {
    "llama-3.1-8b": dict(model_type="llama", hidden_size=4096, intermediate_size=14336, num_hidden_layers=32, num_attention_heads=32,
                         num_key_value_heads=8, head_dim=128, vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0,
                         tie_word_embeddings=False, max_position_embeddings=131072,
                         rope_scaling=dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                           original_max_position_embeddings=8192)),
    "qwen2.5-0.5b": dict(model_type="qwen2", hidden_size=896, intermediate_size=4864, num_hidden_layers=24, num_attention_heads=14,
                         num_key_value_heads=2, head_dim=64, vocab_size=151936, rms_norm_eps=1e-6, rope_theta=1e6,
                         tie_word_embeddings=True, max_position_embeddings=32768),
    "tiny-qwen2": dict(model_type="qwen2", hidden_size=96, intermediate_size=256, num_hidden_layers=3, num_attention_heads=3,
                       num_key_value_heads=1, head_dim=32, vocab_size=384, rms_norm_eps=1e-6, rope_theta=1e6,
                       tie_word_embeddings=True, max_position_embeddings=256),
}
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def _decode(model, rows, context, dtype="bfloat16", page=16):
    return {"kind": "decode", "model": model, "dtype": dtype, "rows": rows, "context": context, "page": page}


def _portions(model, prompts, tokens, prefix=0, rows=0, context=0, want=1, dtype="bfloat16", page=16):
    return {"kind": "portions", "model": model, "dtype": dtype, "prompts": prompts, "tokens": tokens, "prefix": prefix, "rows": rows,
            "context": context, "want": want, "page": page}


def _serve(model, prompts, tokens, new, dtype="bfloat16", page=16):
    return {"kind": "serve", "model": model, "dtype": dtype, "prompts": prompts, "tokens": tokens, "new": new, "page": page}


def listed():
    return [
        # one user's answer being written, at the longest context of the headline benchmark
        {"name": "8b decode 1 x 4096", **_decode("llama-3.1-8b", 1, 4096)},
        # the headline: eight requests, generating
        {"name": "8b decode 8 x 4096", **_decode("llama-3.1-8b", 8, 4096)},
        # a busy server
        {"name": "8b decode 64 x 4096", **_decode("llama-3.1-8b", 64, 4096)},
        # the headline prompt
        {"name": "8b prefill 2048", **_portions("llama-3.1-8b", 1, 2048)},
        # chunked prefill: a portion of a long prompt, beside requests that decode
        {"name": "8b chunk 500 of 12000 + 7", **_portions("llama-3.1-8b", 1, 500, prefix=12000, rows=7, context=3000)},
        # a small model answering one user: launches and latency
        {"name": "0.5b decode 1 x 300", **_decode("qwen2.5-0.5b", 1, 300)},
        # the continuous-batching stream's decode step
        {"name": "0.5b decode 32 x 1280", **_decode("qwen2.5-0.5b", 32, 1280)},
        # the stream's prompts, several in one step
        {"name": "0.5b prefill 4 x 700", **_portions("qwen2.5-0.5b", 4, 700)},
        # requests from prompt to last token through the engine, sampled
        {"name": "0.5b serve 8 x 200 + 24", **_serve("qwen2.5-0.5b", 8, 200, 24)},
        # the true 32-bit path: decoding, scoring a text (logits of every token), and the smallest calls
        {"name": "0.5b f32 decode 4 x 500", **_decode("qwen2.5-0.5b", 4, 500, dtype="float32")},
        {"name": "0.5b f32 score 2 x 200", **_portions("qwen2.5-0.5b", 2, 200, want=200, dtype="float32")},
        {"name": "tiny f32 serve 4 x 40 + 12", **_serve("tiny-qwen2", 4, 40, 12, dtype="float32", page=8)},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "portions", "portions", "serve"))
    if kind == "serve":
        if rng.random() < 0.3:
            return _serve("tiny-qwen2", _log(rng, 1, 4), _log(rng, 8, 150), _log(rng, 4, 24), dtype="float32", page=rng.choice((4, 8, 16)))
        return _serve("qwen2.5-0.5b", _log(rng, 1, 8), _log(rng, 16, 200), _log(rng, 4, 24), page=rng.choice((16, 32)))
    model, dtype = rng.choice((("llama-3.1-8b", "bfloat16"), ("qwen2.5-0.5b", "bfloat16"), ("qwen2.5-0.5b", "float32")))
    page = rng.choice((16, 16, 32))
    if dtype == "float32":
        if kind == "decode":
            return _decode(model, _log(rng, 1, 8), _log(rng, 16, 1000), dtype=dtype, page=page)
        prompts = _log(rng, 1, 4)
        tokens = _log(rng, 8, 400 // prompts)
        return _portions(model, prompts, tokens, want=rng.choice((1, tokens)), dtype=dtype, page=page)
    if kind == "decode":
        return _decode(model, _log(rng, 1, 64), _log(rng, 64, 4096), page=page)
    prompts = _log(rng, 1, 4)
    prefix = rng.choice((0, 0, _log(rng, 100, 12000)))
    tokens = _log(rng, 16, (512 if prefix else 2048) // prompts)
    rows = rng.choice((0, _log(rng, 1, 32)))
    return _portions(model, prompts, tokens, prefix=prefix // prompts, rows=rows, context=_log(rng, 64, 3000) if rows else 0, page=page)


def spread(longest, n):
    """n lengths from `longest` down to half of it."""
    return [longest - (longest // 2) * i // max(1, n - 1) for i in range(n)]


def plan(case):
    """[(tokens already in the cache, tokens of this step)] of the step's requests: portions first, then decoded tokens."""
    out = []
    if case["kind"] != "decode":
        out += [(case.get("prefix", 0), n) for n in spread(case["tokens"], case["prompts"])]
    if case.get("rows"):
        out += [(n - 1, 1) for n in spread(case["context"], case["rows"])]
    return out


# ---- inputs, from the seed alone

def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(seed * 1000 + stream)


def weights(case, seed):
    """Tensors by their checkpoint names; matrices in the case's type, norm weights and biases in float32."""
    c, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
    D, F, V, hd = c["hidden_size"], c["intermediate_size"], c["vocab_size"], c["head_dim"]
    gen = _generator(seed, 0)
    q, kv = c["num_attention_heads"] * hd, c["num_key_value_heads"] * hd

    def matrix(n, k, std=0.02):
        return torch.empty(n, k, dtype=dtype, device="cuda").normal_(0.0, std, generator=gen)

    def vector(n, mean):
        return torch.empty(n, dtype=torch.float32, device="cuda").normal_(mean, 0.02, generator=gen)

    out = {"model.embed_tokens.weight": matrix(V, D, 1.0)}
    for i in range(c["num_hidden_layers"]):
        p = "model.layers.%d." % i
        for name, n in (("q", q), ("k", kv), ("v", kv)):
            out[p + "self_attn.%s_proj.weight" % name] = matrix(n, D)
            if c["model_type"] == "qwen2":
                out[p + "self_attn.%s_proj.bias" % name] = vector(n, 0.0)
        out[p + "self_attn.o_proj.weight"] = matrix(D, q)
        out[p + "mlp.gate_proj.weight"] = matrix(F, D)
        out[p + "mlp.up_proj.weight"] = matrix(F, D)
        out[p + "mlp.down_proj.weight"] = matrix(D, F)
        out[p + "input_layernorm.weight"] = vector(D, 1.0)
        out[p + "post_attention_layernorm.weight"] = vector(D, 1.0)
    out["model.norm.weight"] = vector(D, 1.0)
    if not c["tie_word_embeddings"]:
        out["lm_head.weight"] = matrix(V, D)
    return out


def token_ids(case, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, MODELS[case["model"]]["vocab_size"], n).tolist() for _, n in plan(case)]


def cached(case, seed, layer):
    """What the cache holds of one layer before the step: (all requests' pages in order, [key, value], heads, page, size)."""
    c, page = MODELS[case["model"]], case["page"]
    pages = sum(-(-start // page) for start, _ in plan(case))
    t = torch.empty(pages, 2, c["num_key_value_heads"], page, c["head_dim"], dtype=DTYPES[case["dtype"]], device="cuda")
    return t.normal_(0.0, 0.02 * math.sqrt(c["hidden_size"]), generator=_generator(seed, 1 + layer))


def prepare(case, seed):
    from fusezap_core_b200 import DecoderModel, EngineConfig, LLMEngine, SamplingParams
    from fusezap_core_b200.cache import CacheManager
    from fusezap_core_b200.config import describe
    from fusezap_core_b200.engine import Portion, StepRunner
    from fusezap_core_b200.kernels import cuda_ops

    typed, spec = describe(MODELS[case["model"]])
    model = DecoderModel(spec, typed)
    model.ops = cuda_ops(case["dtype"], "cuda:0")
    requests, page = plan(case), case["page"]
    longest = max(s + n for s, n in requests) + case.get("new", 0)
    max_len = -(-longest // page) * page
    model.bind(weights(case, seed), model.ops, case["dtype"], "cuda:0", max_len)
    ids = token_ids(case, seed)
    pages = sum(-(-(s + n + case.get("new", 0)) // page) for s, n in requests)
    state = {"case": case, "model": model}
    if case["kind"] == "serve":
        engine = LLMEngine(model, EngineConfig(dtype=case["dtype"], max_model_len=max_len, num_blocks=pages, block_size=page,
                                               max_num_seqs=case["prompts"], max_prefill_tokens=sum(n for _, n in requests)))
        state.update(engine=engine, prompts=ids, params=[SamplingParams(max_tokens=case["new"], temperature=0.8, top_p=0.95, seed=i,
                                                                        ignore_eos=True) for i in range(len(ids))])
        return state
    cache = CacheManager(model.cache_needs(), model.state_needs(), page, pages, len(requests), max_len, model.ops.dtype, "cuda:0")
    runner = StepRunner(model, cache, max_rows=sum(n for _, n in requests), max_segments=len(requests))
    for r, (start, _) in enumerate(requests):
        cache.ensure(r, max(start, 1))
        cache.commit(r, start)
    held = [p for r, (start, _) in enumerate(requests) for p in cache.table(0, r)[:-(-start // page)]]
    if held:
        at = torch.tensor(held, device="cuda")
        for layer in range(spec_layers(case)):
            cache.groups[0].pool[layer].index_copy_(0, at, cached(case, seed, layer))
    want = case.get("want", 1)
    portions = [Portion(r, ids[r], list(range(max(0, n - want), n))) for r, (_, n) in enumerate(requests)]
    state.update(runner=runner, portions=portions, starts=[s for s, _ in requests])
    if case["kind"] == "decode":
        runner.run(portions)
        _rewind(state)
        runner.prepare(portions)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = runner.forward()
        state.update(graph=graph, logits=logits)
    return state


def spec_layers(case):
    return MODELS[case["model"]]["num_hidden_layers"]


def _rewind(state):
    """The requests stand before this step's tokens again."""
    for r, start in enumerate(state["starts"]):
        state["runner"].cache.commit(r, start)


def run(state):
    if state["case"]["kind"] == "serve":
        engine = state["engine"]
        tokens = engine.generate(state["prompts"], state["params"])
        # the logits that the last token of every request was sampled from
        logits = engine.runner.ws.get("logits", (len(tokens), engine.model.spec.vocab_size), torch.float32)
        return {"tokens": torch.tensor(tokens), "logits": logits}
    runner, portions = state["runner"], state["portions"]
    _rewind(state)
    if state["case"]["kind"] == "portions":
        return runner.run(portions)
    starts = runner.prepare(portions)
    state["graph"].replay()
    runner.commit(portions, starts)
    return state["logits"]


def work(case):
    c = MODELS[case["model"]]
    D, F, V, L, hd = c["hidden_size"], c["intermediate_size"], c["vocab_size"], c["num_hidden_layers"], c["head_dim"]
    Hq, Hkv, size = c["num_attention_heads"], c["num_key_value_heads"], DTYPES[case["dtype"]].itemsize
    body = L * (D * (2 * Hq + 2 * Hkv) * hd + 3 * D * F)
    steps = [plan(case)] + [[(s + n + i, 1) for s, n in plan(case)] for i in range(case.get("new", 1) - 1)]
    total_bytes = total_flops = 0
    for step in steps:
        wanted = sum(min(n, case.get("want", 1)) for _, n in step)
        tokens = sum(n for _, n in step)
        pairs = sum(n * s + n * (n + 1) // 2 for s, n in step)
        total_bytes += size * (body + V * D + tokens * D + sum(s + 2 * n for s, n in step) * 2 * Hkv * hd * L) + 4 * wanted * V
        total_flops += 2 * (tokens * body + wanted * V * D) + 4 * pairs * Hq * hd * L
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # bfloat16: roundings of h, the attention output, the gated product and the cache in every layer. float32: sums of
    # up to 4,864 terms in every layer. Measured against 64 bits: 0.017 at the 8B sizes (0.024 between two such results),
    # 0.0044 at the 0.5B sizes, 2.1e-6 in float32. Tokens are certain (see the top), so they are the same.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 0.03, "max": 0.2, "differ": 0.0} if case["model"].startswith("llama") else {"rel": 0.016, "max": 0.1, "differ": 0.0}


# ---- the same in 64 bits, by plain torch

def _frequencies(c):
    """Per pair of dimensions, in float32, which is how the architecture defines them."""
    d = c["head_dim"]
    inv = (1.0 / (np.float32(c["rope_theta"]) ** (np.arange(0, d, 2).astype(np.float32) / np.float32(d)))).astype(np.float32)
    s = c.get("rope_scaling")
    if s:
        old, wl = s["original_max_position_embeddings"], 2 * math.pi / inv
        smooth = (old / wl - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])
        blend = (1 - smooth) * inv / s["factor"] + smooth * inv
        inv = np.where(wl > old / s["low_freq_factor"], inv / s["factor"], np.where(wl < old / s["high_freq_factor"], inv, blend)).astype(np.float32)
    return inv


def _forward(case, w, requests, ids, past, want):
    """Logits of the last `want` tokens of each request. past: layer -> its cached pages, as `cached` lays them out, or None."""
    c, page = MODELS[case["model"]], case["page"]
    Hq, Hkv, hd, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    inv = _frequencies(c)
    angles = np.concatenate([np.arange(s, s + n, dtype=np.float32)[:, None] * inv[None] for s, n in requests]).astype(np.float64)
    cos, sin = (torch.from_numpy(f(angles)).cuda()[:, None] for f in (np.cos, np.sin))

    def norm(x, weight):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight.double()

    def linear(x, name):
        y = x @ w[name + ".weight"].double().T
        return y + w[name + ".bias"].double() if name + ".bias" in w else y

    def turned(x):
        a, b = x.chunk(2, -1)
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    x = w["model.embed_tokens.weight"][torch.tensor([t for r in ids for t in r], device="cuda")].double()
    for i in range(c["num_hidden_layers"]):
        p = "model.layers.%d." % i
        h = norm(x, w[p + "input_layernorm.weight"])
        q, k, v = (linear(h, p + "self_attn.%s_proj" % n).view(len(x), -1, hd) for n in "qkv")
        q, k = turned(q), turned(k)
        held = past(i) if past else None
        outs, at, first = [], 0, 0
        for s, n in requests:
            kk, vv = k[at: at + n], v[at: at + n]
            if s:
                pages = -(-s // page)
                old = held[first: first + pages].double().permute(1, 0, 3, 2, 4).reshape(2, pages * page, Hkv, hd)[:, :s]
                kk, vv, first = torch.cat((old[0], kk)), torch.cat((old[1], vv)), first + pages
            qq = q[at: at + n].view(n, Hkv, Hq // Hkv, hd)
            out = torch.empty_like(qq)
            for g in range(Hkv):
                scores = torch.einsum("nhd,md->hnm", qq[:, g], kk[:, g]) / math.sqrt(hd)
                if n > 1:
                    scores = scores.masked_fill(torch.arange(s + n, device="cuda")[None] > torch.arange(s, s + n, device="cuda")[:, None], -math.inf)
                out[:, g] = torch.einsum("hnm,md->nhd", scores.softmax(-1), vv[:, g])
            outs.append(out.reshape(n, Hq * hd))
            at += n
        x = x + linear(torch.cat(outs), p + "self_attn.o_proj")
        h = norm(x, w[p + "post_attention_layernorm.weight"])
        x = x + linear(torch.nn.functional.silu(linear(h, p + "mlp.gate_proj")) * linear(h, p + "mlp.up_proj"), p + "mlp.down_proj")
    last, at = [], 0
    for _, n in requests:
        last += range(at + max(0, n - want), at + n)
        at += n
    head = w.get("lm_head.weight", w["model.embed_tokens.weight"])
    h = norm(x[last], w["model.norm.weight"])
    return torch.cat([h @ rows.double().T for rows in head.split(16384)], -1)


def exact(case, seed):
    w, requests, ids = weights(case, seed), plan(case), token_ids(case, seed)
    with torch.no_grad():
        if case["kind"] != "serve":
            return _forward(case, w, requests, ids, lambda layer: cached(case, seed, layer), case.get("want", 1))
        logits = None
        for _ in range(case["new"]):      # a token that is certain is the one with the largest logit
            logits = _forward(case, w, [(0, len(r)) for r in ids], ids, None, 1)
            ids = [r + [int(t)] for r, t in zip(ids, logits.argmax(-1))]
        return {"tokens": None, "logits": logits}
