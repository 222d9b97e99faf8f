"""What the speed of this framework is judged by: generation through the continuous-batching engine, and its sampler.

``listed()`` holds the cases, ``draw(rng)`` gives more of the same ranges.  Everything but the sampler case goes through
``LLMEngine.add_request`` / ``step`` / ``core.release``, the calls of the server and of ``generate``.

Models are the named shapes of ``onnx_genai_b200.models.config``: Qwen2.5-0.5B with int4 projections (the batch-1 and
small-batch serving configuration), Qwen2.5-7B in bf16 (the headline configuration) and Qwen3-30B-A3B (experts).  The
small one has all its layers; the other two have fewer, so that states are made quickly -- every layer is the same work.

Weights are random, but embeddings and LM head agree on a follower for every token (the token itself where they are
tied), as far above the other logits as it is in a trained model that is sure of itself.  Greedy tokens, and drawn ones at top-p
0.9, therefore do not depend on the last bits of the logits, and two correct implementations produce the same text.

``cached`` cases are the later turns of conversations: the prompts' whole pages lie in the prefix cache, a pass computes
the rest of each prompt (at most 16 tokens) and then decodes.  The others prefill their prompts (no prefix cache).
"""
import math
import random
import types

import torch

from onnx_genai_b200 import ops
from onnx_genai_b200.engine.llm_engine import EngineConfig, LLMEngine
from onnx_genai_b200.models.config import preset
from onnx_genai_b200.models.decoder import DecoderWeights, LayerWeights

SMALL, DENSE, EXPERTS = "qwen2.5-0.5b", "qwen2.5-7b", "qwen3-30b-a3b"
LAYERS = {SMALL: 24, DENSE: 8, EXPERTS: 4}
EMBED_STD = {SMALL: 2.0, DENSE: 2.0, EXPERTS: 1.0}   # against what the layers add: the follower stays in view


def _gen(name, model, seqs, low, high, new, cached, kv="bf16", budget=2304, temperature=0.0, top_p=1.0):
    """``seqs`` requests with prompts of ``low`` to ``high`` tokens, ``new`` tokens each; ``budget``: tokens a step may hold."""
    return {"name": name, "kind": "generate", "model": model, "seqs": seqs, "low": low, "high": high, "new": new, "cached": cached,
            "kv": kv, "budget": budget, "temperature": temperature, "top_p": top_p}


def listed():
    return [
        # one user of the small int4 model: latency per token, the reference's own headline
        _gen("int4_one", SMALL, 1, 512, 512, 32, True),
        # a small server of the same model at its usual batch
        _gen("int4_batch", SMALL, 64, 100, 700, 16, True),
        # prompts of that model: int4 products with many rows
        _gen("int4_prompts", SMALL, 6, 30, 1001, 1, False, budget=4096),
        # one user of the large model
        _gen("dense_one", DENSE, 1, 777, 777, 16, True),
        # a handful of users with 8-bit pages
        _gen("dense_few_int8_pages", DENSE, 16, 300, 2300, 16, True, kv="int8"),
        # long contexts with e4m3 pages
        _gen("dense_long_e4m3_pages", DENSE, 8, 6000, 12000, 16, True, kv="fp8", budget=8192),
        # the headline's decode: 256 conversations, drawn tokens
        _gen("dense_batch", DENSE, 256, 128, 1100, 16, True, temperature=0.7, top_p=0.9),
        # time to first token of a short question, and of long documents
        _gen("dense_short_prompt", DENSE, 1, 77, 77, 1, False),
        _gen("dense_long_prompts", DENSE, 4, 1500, 2048, 1, False, budget=8192),
        # serving: requests arrive together, prompts are cut to the step's budget while others decode
        _gen("dense_serving", DENSE, 40, 128, 1000, 12, False, temperature=0.7, top_p=0.9),
        # experts: decode, where few rows meet each expert, and prompts
        _gen("experts_decode", EXPERTS, 32, 60, 900, 16, True),
        # the sampler alone, as a caller with its own loop uses it: flat and sure rows, top-k, top-p and min-p
        {"name": "sample", "kind": "sample", "rows": 256, "vocab": 152064},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("small", "small_prompts", "dense", "dense", "dense_prompts", "serving", "experts", "experts_prompts", "sample"))
    sampled = rng.random() < 0.5
    how = {"temperature": 0.7, "top_p": 0.9} if sampled else {}
    kv = rng.choice(("bf16", "bf16", "fp8", "int8"))
    if kind == "sample":
        return _nameless({"kind": "sample", "rows": _log(rng, 1, 256), "vocab": rng.choice((32000, 151936, 152064))})
    if kind == "small":
        return _nameless(_gen("", SMALL, _log(rng, 1, 64), 16, _log(rng, 32, 1000), rng.randint(4, 24), True, **how))
    if kind == "small_prompts":
        return _nameless(_gen("", SMALL, _log(rng, 1, 8), 9, _log(rng, 20, 1000), 1, False, budget=4096, **how))
    if kind == "dense":
        seqs = _log(rng, 1, 256)
        high = _log(rng, 64, min(12000, 262144 // seqs))
        return _nameless(_gen("", DENSE, seqs, high // 4, high, rng.randint(4, 16), True, kv=kv, budget=4096, **how))
    if kind == "dense_prompts":
        return _nameless(_gen("", DENSE, _log(rng, 1, 4), 5, _log(rng, 16, 2048), 1, False, kv=kv, budget=8192, **how))
    if kind == "serving":
        return _nameless(_gen("", DENSE, rng.randint(8, 40), 32, _log(rng, 64, 1000), rng.randint(4, 12), False, kv=kv, **how))
    if kind == "experts":
        return _nameless(_gen("", EXPERTS, _log(rng, 1, 64), 16, _log(rng, 64, 1000), rng.randint(4, 16), True, **how))
    return _nameless(_gen("", EXPERTS, _log(rng, 1, 4), 7, _log(rng, 16, 1500), 1, False, budget=8192, **how))


def _nameless(case):
    return {k: v for k, v in case.items() if k != "name"}


def _lengths(case):
    """Prompt lengths: spread over the range, in an order of no pattern, the same for every seed; one request alone has the longest."""
    n, low, high = case["seqs"], min(case["low"], case["high"]), case["high"]
    if n == 1:
        return [high]
    lens = [low + (high - low) * i // (n - 1) for i in range(n)]
    random.Random(n).shuffle(lens)
    return lens


def _config(case):
    top = max(_lengths(case)) + case["new"]
    cfg = preset(case["model"])
    return cfg.replace(num_layers=LAYERS[case["model"]], max_position=max(cfg.max_position, top))


# ------------------------------------------------------------------------------------------
# weights
# ------------------------------------------------------------------------------------------
def _plain_weights(cfg, seed):
    """The model's matrices as a checkpoint has them, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)

    def normal(*shape, std=0.02):
        return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)

    def matrix(n, k):
        if cfg.weight_format != "int4":
            return normal(n, k)
        codes = torch.randint(1, 16, (2, n, k // 32, 16), dtype=torch.uint8, device="cuda", generator=g)   # 1 to 15 stand for -7 to 7
        codes = codes[0] | codes[1] << 4
        scales = torch.empty(n, k // 32, device="cuda").uniform_(0.002, 0.0065, generator=g).bfloat16()
        return codes, scales

    a = EMBED_STD[cfg.name]
    embed = normal(cfg.vocab, cfg.hidden, std=a)
    follower = torch.arange(cfg.vocab, device="cuda")
    head = embed
    if not cfg.tie_embeddings:
        follower = torch.randperm(cfg.vocab, device="cuda", generator=g)
        head = torch.empty_like(embed)
        head[follower] = embed
    layers = []
    for _ in range(cfg.num_layers):
        l = {"q": matrix(cfg.q_size, cfg.hidden), "k": matrix(cfg.kv_size, cfg.hidden), "v": matrix(cfg.kv_size, cfg.hidden),
             "o": matrix(cfg.hidden, cfg.q_size)}
        if cfg.qkv_bias:
            l["bias"] = normal(cfg.q_size + 2 * cfg.kv_size)
        if cfg.moe.num_experts:
            e, i = cfg.moe.num_experts, cfg.moe.expert_intermediate
            l["router"] = normal(e, cfg.hidden)
            l["gate"], l["up"], l["down"] = normal(e, i, cfg.hidden), normal(e, i, cfg.hidden), normal(e, cfg.hidden, i)
        else:
            l["gate"], l["up"] = matrix(cfg.intermediate, cfg.hidden), matrix(cfg.intermediate, cfg.hidden)
            l["down"] = matrix(cfg.hidden, cfg.intermediate)
        layers.append(l)
    # the other logits have a deviation of about 1
    norm = torch.full((cfg.hidden,), 1.0 / (a * math.sqrt(cfg.hidden)), dtype=torch.bfloat16, device="cuda")
    return {"embed": embed, "head": head, "follower": follower, "norm": norm, "layers": layers}


def _bound_weights(cfg, plain):
    """The same as the engine takes them."""
    ones = torch.ones(cfg.hidden, dtype=torch.bfloat16, device="cuda")
    half = 128
    layers = []
    for l in plain["layers"]:
        if cfg.weight_format == "int4":
            cuts = [0, cfg.q_size, cfg.q_size + cfg.kv_size, cfg.q_size + 2 * cfg.kv_size]

            def lin(key, bias=None):
                codes, scales = l[key]
                return types.SimpleNamespace(q=codes, scales=scales, zp=None, bias=bias, k=codes.shape[1] * 32, block=32)

            quant = {"qkv": [lin(key, l["bias"][cuts[i]:cuts[i + 1]]) for i, key in enumerate("qkv")]}
            quant.update({key: lin(key) for key in ("o", "gate", "up", "down")})
            layers.append(LayerWeights(ln1=ones, qkv_w=None, qkv_b=None, o_w=None, ln2=ones, quant=quant))
            continue
        lw = LayerWeights(ln1=ones, qkv_w=torch.cat([l["q"], l["k"], l["v"]]), qkv_b=l.get("bias"), o_w=l["o"], ln2=ones)
        if cfg.moe.num_experts:
            e, i = cfg.moe.num_experts, cfg.moe.expert_intermediate
            lw.router_w = l["router"]
            lw.expert_gate_up = torch.stack([l["gate"].view(e, i // half, half, -1), l["up"].view(e, i // half, half, -1)], 2).reshape(e, 2 * i, -1)
            lw.expert_down = l["down"]
        else:
            lw.gate_up_w, lw.down_w = ops.pack_gate_up(l["gate"], l["up"], half), l["down"]
        layers.append(lw)
    return DecoderWeights(embed=plain["embed"], layers=layers, final_norm=plain["norm"], lm_head=plain["head"], swiglu_half=half)


def _prompts(case, cfg, seed):
    g = torch.Generator().manual_seed(seed * 31 + 5)
    return [torch.randint(0, cfg.vocab, (n,), generator=g, dtype=torch.int32).numpy() for n in _lengths(case)]


# ------------------------------------------------------------------------------------------
# the path
# ------------------------------------------------------------------------------------------
def _logit_rows(case, seed):
    """Half the rows flat, half sure of a few tokens; every combination of filters a request may carry."""
    g = torch.Generator(device="cuda").manual_seed(seed * 13 + 3)
    r, v = case["rows"], case["vocab"]
    logits = torch.randn(r, v, device="cuda", generator=g) * 2.0
    best = torch.randint(0, v, (r, 8), device="cuda", generator=g)
    lift = torch.rand(r, 8, device="cuda", generator=g) * 8.0 + 6.0
    lift[::2] = 0.0
    logits.scatter_add_(1, best, lift)
    rows = torch.arange(r, device="cuda")
    return (logits.bfloat16(), torch.full((r,), 0.7, device="cuda"), torch.where(rows % 4 == 3, 50, 0).int(),
            torch.where(rows % 8 == 6, 1.0, 0.9).float(), torch.where(rows % 16 == 5, 0.05, 0.0).float(),
            torch.rand(r, device="cuda", generator=g))


def prepare(case, seed):
    if case["kind"] == "sample":
        rows = _logit_rows(case, seed)
        return {"case": case, "rows": rows, "work": torch.empty(case["rows"] * case["vocab"], dtype=torch.int32, device="cuda")}
    cfg = _config(case)
    prompts = _prompts(case, cfg, seed)
    top = max(len(p) for p in prompts) + case["new"]
    pages = sum((len(p) + case["new"]) // ops.PAGE + 2 for p in prompts)
    eng = LLMEngine(EngineConfig(model=cfg, num_pages=2 * pages + 64, max_seqs=case["seqs"], max_tokens_per_step=max(case["budget"], 2 * case["seqs"]),
                                 max_seq_len=top + ops.PAGE, prefill_chunk=case["budget"], enable_prefix_cache=case["cached"],
                                 kv_dtype=case["kv"], cuda_graphs=True), weights=_bound_weights(cfg, _plain_weights(cfg, seed)))
    state = {"case": case, "eng": eng, "prompts": prompts}
    if case["cached"]:      # the conversations' earlier turns
        run(state)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return {"tokens": ops.sample(*state["rows"], work=state["work"])}
    eng, new = state["eng"], case["new"]
    ids = [eng.add_request(p, new, temperature=case["temperature"], top_p=case["top_p"], seed=11 + i, ignore_eos=True)
           for i, p in enumerate(state["prompts"])]
    at = {sid: i for i, sid in enumerate(ids)}
    tokens = torch.zeros(len(ids), new, dtype=torch.int32)
    count = [0] * len(ids)
    logits = None
    left = len(ids)
    while left:
        events = eng.step().events
        done = []
        for row, (sid, tok, fin) in enumerate(events):     # an event for every row of the step's logits, in their order
            i = at[sid]
            tokens[i, count[i]] = tok
            count[i] += 1
            if fin is not None:
                done.append((row, i))
        if done:                                           # the logits behind every request's last token
            left -= len(done)
            if len(done) == len(ids) and all(r == i for r, i in done):
                logits = eng.model.logits[: len(ids)]
                break
            if logits is None:
                logits = torch.empty(len(ids), eng.model.logits.shape[1], dtype=eng.model.logits.dtype, device="cuda")
            for row, i in done:
                logits[i].copy_(eng.model.logits[row])
    for sid in ids:
        eng.core.release(sid)
    few = _compared(case)
    return {"tokens": tokens, "first": logits[:few], "others": logits[few:]}


def _compared(case):
    """How many requests exact() works out."""
    total = n = 0
    for k in _lengths(case):
        total += k + case["new"]
        if n and total > 6000:
            break
        n += 1
    return n


# ------------------------------------------------------------------------------------------
# what it has to do, and what it should give
# ------------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 2 * case["rows"] * case["vocab"], "flops": 4 * case["rows"] * case["vocab"]}
    cfg, lens, new = _config(case), _lengths(case), case["new"]
    cached = [(n - 1) // ops.PAGE * ops.PAGE if case["cached"] else 0 for n in lens]
    rows = sum(n - c for n, c in zip(lens, cached))             # prompt rows computed
    budget = max(case["budget"], 2 * case["seqs"])
    steps = -(-rows // budget) + new - 1
    per = 2.0 if cfg.weight_format != "int4" else 0.5 + 2.0 / 32
    attn = cfg.hidden * (2 * cfg.q_size + 2 * cfg.kv_size)
    e, k, i = cfg.moe.num_experts, cfg.moe.top_k, cfg.moe.expert_intermediate or cfg.intermediate
    mlp = 3 * cfg.hidden * i
    kv_row = cfg.num_layers * 2 * cfg.kv_size * (2 if case["kv"] == "bf16" else 1)
    head = 2 * cfg.vocab * cfg.hidden
    touched = (lambda t: mlp * e * (1 - (1 - k / e) ** t)) if e else (lambda t: mlp)
    prompt_steps = steps - (new - 1)
    data = prompt_steps * (cfg.num_layers * (attn + touched(rows / prompt_steps)) * per + head)
    data += (new - 1) * (cfg.num_layers * (attn + touched(len(lens))) * per + head)
    data += kv_row * sum(n + sum(n + j for j in range(1, new)) for n in lens)
    active = cfg.num_layers * (attn + mlp * (k if e else 1))
    tokens = rows + len(lens) * (new - 1)
    flops = 2.0 * active * tokens + head * len(lens) * new
    pairs = sum((n * (n + 1) - c * (c + 1)) / 2 + sum(n + j for j in range(1, new)) for n, c in zip(lens, cached))
    flops += 4.0 * cfg.num_layers * cfg.q_size * pairs
    return {"bytes": data, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.01}    # a draw that falls on the edge between two tokens
    # bf16 activations between the products of all layers; 8-bit pages and experts chosen by near-equal scores add to that
    return {"rel": 0.03, "max": 0.3, "differ": 0.002}


def exact(case, seed):
    """The logits of the first requests, in 64 bits throughout (pages, weights' products and sums)."""
    if case["kind"] == "sample":
        return None
    cfg = _config(case)
    plain = _plain_weights(cfg, seed)
    new, few = case["new"], _compared(case)
    wide = torch.float64
    seqs = []
    for p in _prompts(case, cfg, seed)[:few]:
        ids = torch.from_numpy(p).long().cuda().tolist()
        for _ in range(new - 1):
            ids.append(int(plain["follower"][ids[-1]]))
        seqs.append(ids)
    cuts = [0]
    for s in seqs:
        cuts.append(cuts[-1] + len(s))
    ids = torch.tensor([t for s in seqs for t in s], device="cuda")
    where = torch.cat([torch.arange(len(s), device="cuda") for s in seqs]).to(wide)
    d = cfg.head_dim
    ang = where[:, None] * (cfg.rope_theta ** (-torch.arange(0, d, 2, device="cuda", dtype=wide) / d))[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]

    def full(m):
        if not isinstance(m, tuple):
            return m.to(wide)
        codes, scales = m
        c = torch.stack([codes & 15, codes >> 4], -1).reshape(codes.shape[0], -1, 32).to(wide) - 8.0
        return (c * scales.to(wide)[:, :, None]).reshape(codes.shape[0], -1)

    def norm(x):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.rms_eps)

    def turned(x):
        a, b = x[..., : d // 2], x[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def mlp(x, gate, up, down):
        return (torch.nn.functional.silu(x @ full(gate).t()) * (x @ full(up).t())) @ full(down).t()

    x = plain["embed"][ids].to(wide)
    for l in plain["layers"]:
        h = norm(x)
        q, k, v = (h @ full(l[key]).t() for key in "qkv")
        if cfg.qkv_bias:
            bias = l["bias"].to(wide)
            q, k, v = q + bias[: cfg.q_size], k + bias[cfg.q_size: cfg.q_size + cfg.kv_size], v + bias[cfg.q_size + cfg.kv_size:]
        q, k, v = turned(q.view(-1, cfg.num_heads, d)), turned(k.view(-1, cfg.num_kv_heads, d)), v.view(-1, cfg.num_kv_heads, d)
        o = torch.empty_like(q)
        group = cfg.num_heads // cfg.num_kv_heads
        for lo, hi in zip(cuts, cuts[1:]):
            for a in range(lo, hi, 1024):
                b = min(hi, a + 1024)
                seen = torch.arange(lo, b, device="cuda")[None, :] <= torch.arange(a, b, device="cuda")[:, None]
                for n in range(cfg.num_kv_heads):
                    s = torch.einsum("qgd,kd->gqk", q[a:b, n * group:(n + 1) * group], k[lo:b, n]) / math.sqrt(d)
                    w = torch.softmax(s.masked_fill(~seen, float("-inf")), -1)
                    o[a:b, n * group:(n + 1) * group] = torch.einsum("gqk,kd->qgd", w, v[lo:b, n])
        x = x + o.reshape(-1, cfg.q_size) @ full(l["o"]).t()
        h = norm(x)
        if cfg.moe.num_experts:
            probs = torch.softmax(h @ full(l["router"]).t(), -1)
            best, which = torch.topk(probs, cfg.moe.top_k, -1)
            if cfg.moe.renormalize:
                best = best / best.sum(-1, keepdim=True)
            for e in range(cfg.moe.num_experts):
                rows, slot = (which == e).nonzero(as_tuple=True)
                if rows.numel():
                    x[rows] += best[rows, slot, None] * mlp(h[rows], l["gate"][e], l["up"][e], l["down"][e])
        else:
            x = x + mlp(h, l["gate"], l["up"], l["down"])
    last = torch.tensor([c - 1 for c in cuts[1:]], device="cuda")
    logits = (norm(x[last]) * plain["norm"].to(wide)) @ plain["head"].to(wide).t()
    follower = plain["follower"][ids[last]]
    if not bool((logits.argmax(-1) == follower).all()):
        raise RuntimeError("a token's follower is not its likeliest successor: the text of a pass is then not certain")
    return {"tokens": None, "first": logits, "others": None}
