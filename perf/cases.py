"""What a user of this framework has it do, as measurable cases: requests served by a decoder (bf16 and block-scaled fp8), and the
operations that the other model designs spend their time in (attention over long prompts, latent attention, experts, packed
k-quant weights, sampling, recurrent layers), each over its range from a single row to a full token budget.

`prepare` makes a case's inputs from the seed, `run` is one pass through the public entry points, `exact` the same result in 64
bits by plain torch. Lengths inside a batch are ragged and follow from the case alone, so every seed has the same work."""
import math
import random

import torch

DEV = "cuda"
PAGE = 128
BUDGET = 4096                 # tokens of one engine step
VOCAB = 32000
BF16 = torch.bfloat16
# layer sizes: a 1B, an 8B and a 70B decoder
SIZES = {
    "1b": dict(width=2048, heads=16, kv=4, ffn=8192),
    "8b": dict(width=4096, heads=32, kv=8, ffn=14336),
    "70b": dict(width=8192, heads=64, kv=8, ffn=28672),
}


def listed():
    return [
        # one user's chat on a small model: a short prompt, then a token at a time; nothing but latency counts
        dict(name="chat bf16", kind="serve", size="1b", layers=8, fp8=False, seqs=1, prompt=40, steps=12),
        # continuous batching: prompts enter in chunks under the token budget while earlier requests decode beside them
        dict(name="batch bf16", kind="serve", size="8b", layers=8, fp8=False, seqs=48, prompt=1024, steps=8),
        # the same for layers of a 70B checkpoint in block-scaled fp8
        dict(name="batch fp8", kind="serve", size="70b", layers=2, fp8=True, seqs=32, prompt=512, steps=8),
        # chunks of long documents: new rows attend over what earlier chunks left in the cache
        dict(name="long prompts", kind="attention", heads=32, kv=8, seqs=2, rows=2048, prefix=14000, window=0),
        # latent attention (DeepSeek-V2-Lite's heads): prompts ...
        dict(name="latent prompts", kind="latent", heads=16, seqs=3, rows=1500, prefix=700),
        # ... and a decode step of a few long conversations
        dict(name="latent decode", kind="latent", heads=16, seqs=12, rows=1, prefix=4000),
        # mixture of experts: a prompt step, and a decode step of a few users
        dict(name="experts prompts", kind="experts", width=2048, ffn=1408, rows=3001, scoring="softmax"),
        dict(name="experts decode", kind="experts", width=2048, ffn=1408, rows=5, scoring="sigmoid"),
        # a feed-forward kept packed (Q4_K, Q6_K) at decode size
        dict(name="packed weights", kind="packed", size="8b", rows=4),
        # a step's sampling: every request has its own temperature, top-k and top-p
        dict(name="sampling", kind="sample", rows=64, vocab=128256),
        # recurrent layers: two prompts through the delta rule, and decode rows beside a prompt through gated linear attention
        dict(name="delta prompts", kind="delta", heads=32, decode=0, chunks=2, rows=2000, per_head=False),
        dict(name="gated mixed", kind="gated", heads=16, decode=48, chunks=1, rows=1000),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["serve", "serve", "attention", "latent", "latent", "experts", "packed", "sample", "delta", "gated"])
    if kind == "serve":
        fp8 = rng.random() < 0.4
        return dict(kind=kind, size="70b" if fp8 else rng.choice(["1b", "8b"]), layers=2 if fp8 else rng.choice([4, 8]), fp8=fp8, seqs=_log(rng, 1, 32 if fp8 else 48),
                    prompt=_log(rng, 16, 512 if fp8 else 1024), steps=rng.randint(2, 12 if not fp8 else 8))
    if kind == "attention":
        heads, kv = rng.choice([(32, 8), (16, 4), (64, 8)])
        return dict(kind=kind, heads=heads, kv=kv, seqs=rng.randint(1, 4), rows=_log(rng, 64, 1024 if heads == 64 else 2048), prefix=_log(rng, 500, 7000 if heads == 64 else 14000),
                    window=rng.choice([0, 0, 1024]))
    if kind == "latent":
        if rng.random() < 0.5:
            return dict(kind=kind, heads=16, seqs=_log(rng, 1, 96), rows=1, prefix=_log(rng, 200, 4000))
        return dict(kind=kind, heads=16, seqs=rng.randint(1, 3), rows=_log(rng, 100, 1500), prefix=_log(rng, 1, 700))
    if kind == "experts":
        return dict(kind=kind, width=2048, ffn=1408, rows=_log(rng, 1, 4000) if rng.random() < 0.5 else _log(rng, 1, 128), scoring=rng.choice(["softmax", "sigmoid"]))
    if kind == "packed":
        return dict(kind=kind, size=rng.choice(["1b", "8b"]), rows=_log(rng, 1, 128) if rng.random() < 0.7 else _log(rng, 129, 1024))
    if kind == "sample":
        return dict(kind=kind, rows=_log(rng, 1, 256), vocab=rng.choice([128256, 128256, 32000]))
    decode = rng.choice([0, _log(rng, 1, 64)])
    chunks = rng.randint(1, 4) if decode == 0 else rng.choice([0, 0, 1])
    rows = _log(rng, 50, 4000 // max(chunks, 2))
    if kind == "delta":
        return dict(kind=kind, heads=rng.choice([16, 32]), decode=decode, chunks=chunks, rows=rows, per_head=rng.random() < 0.5)
    return dict(kind=kind, heads=rng.choice([16, 32]), decode=decode, chunks=chunks, rows=rows)


# ------------------------------------------------------------------------------------------------------
# shared by prepare and exact
# ------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * std).to(dtype)


def _lengths(case, n, lo, hi, salt=""):
    """n lengths between lo and hi that follow from the case's sizes."""
    r = random.Random(salt + repr(sorted((k, v) for k, v in case.items() if k != "name")))
    return [r.randint(lo, hi) for _ in range(n)]


def _int32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _paged(ctx, seed):
    """Block tables of sequences whose pages lie scattered over the cache. Returns (pages, tables [n, blocks], lists)."""
    per = [-(-c // PAGE) for c in ctx]
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(seed)).tolist()
    tables, at = torch.zeros(len(ctx), max(per), dtype=torch.int32), 0
    for i, n in enumerate(per):
        tables[i, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
    return sum(per), tables


def _cached(cache, table, n):
    """Rows 0 .. n - 1 of one sequence, from a cache [pages, page, columns]."""
    return cache[table[:-(-n // PAGE)].long()].flatten(0, 1)[:n]


# ------------------------------------------------------------------------------------------------------
# serve: requests through the engine, logits of every position that would be sampled
# ------------------------------------------------------------------------------------------------------


def _serve_steps(case):
    """[[(request, first token, tokens, wanted)], [requests that end]] of every engine step, and the prompts' lengths."""
    S, extra = case["seqs"], case["steps"]
    prompts = _lengths(case, S, max(1, case["prompt"] // 8), case["prompt"]) if S > 1 else [case["prompt"]]
    done, steps = [0] * S, []
    while any(done[i] < prompts[i] + extra for i in range(S)):
        entries, ends, room = [], [], BUDGET
        for i in range(S):
            if prompts[i] <= done[i] < prompts[i] + extra:
                entries.append((i, done[i], 1, True))
                room -= 1
        for i in range(S):
            n = min(prompts[i] - done[i], room)
            if n > 0:
                entries.append((i, done[i], n, done[i] + n == prompts[i]))
                room -= n
        for i, _, n, _ in entries:
            done[i] += n
            if done[i] == prompts[i] + extra:
                ends.append(i)
        steps.append((entries, ends))
    return steps, prompts


def _serve_config(case):
    from mojo_b200.models.config import ModelConfig

    s = SIZES[case["size"]]
    return ModelConfig(hidden_size=s["width"], num_layers=case["layers"], num_heads=s["heads"], num_kv_heads=s["kv"], head_dim=128, intermediate_size=s["ffn"],
                       vocab_size=VOCAB, max_position_embeddings=4096, quantization="fp8_block" if case["fp8"] else None)


def _quant_blocks(w):
    """e4m3 with one scale per 128 x 128 block, as checkpoints hold it."""
    n, k = w.shape
    b = w.float().view(n // 128, 128, k // 128, 128)
    s = b.abs().amax(dim=(1, 3)) / 448.0
    return (b / s[:, None, :, None]).view(n, k).to(torch.float8_e4m3fn), s


def _serve_weights(case, seed):
    """(name, tensors) of a checkpoint in the order they are made: the embedding, every layer, the final norm, the head. What a layer adds
    to the residual shrinks with the depth, as in trained decoders; otherwise a few layers of random weights magnify every rounding."""
    s, g = SIZES[case["size"]], _gen(seed)
    W, F, H, G = s["width"], s["ffn"], s["heads"], s["kv"]
    norm = lambda: 1.0 + _randn(g, W, std=0.1)  # noqa: E731
    yield "embed", _randn(g, VOCAB, W)
    for i in range(case["layers"]):
        shapes = dict(wq=(H * 128, W), wk=(G * 128, W), wv=(G * 128, W), wo=(W, H * 128), w_gate=(F, W), w_up=(F, W), w_down=(W, F))
        w = {n: _randn(g, *z, std=(z[1] * (2 * case["layers"] if n in ("wo", "w_down") else 1)) ** -0.5) for n, z in shapes.items()}
        w.update(attn_norm=norm(), mlp_norm=norm())
        if case["fp8"]:
            pairs = {n: _quant_blocks(w[n]) for n in shapes}
            w.update({n: p[0] for n, p in pairs.items()})
            w["scales"] = {n: p[1] for n, p in pairs.items()}
        yield i, w
    yield "final_norm", norm()
    yield "lm_head", _randn(g, VOCAB, W, std=0.02)


def _serve_tokens(case, prompts, seed):
    g = torch.Generator().manual_seed(seed + 7)
    return [torch.randint(0, VOCAB, (n + case["steps"],), generator=g).tolist() for n in prompts]


def _prepare_serve(case, seed):
    from mojo_b200.engine import EngineConfig, LLMEngine
    from mojo_b200.models.llama import LlamaModel

    steps, prompts = _serve_steps(case)
    cfg = _serve_config(case)
    model = LlamaModel(cfg, DEV, BF16)
    for name, w in _serve_weights(case, seed):
        model.load_layer(name, w) if isinstance(name, int) else model.load_tensor(name, w)
    pages = sum(-(-(n + case["steps"]) // PAGE) for n in prompts) + 2
    engine = LLMEngine(EngineConfig(model=cfg, device="cuda:0", dtype=BF16, page_size=PAGE, num_pages=pages, max_num_seqs=case["seqs"], max_num_batched_tokens=BUDGET,
                                    max_model_len=2048, capture_graphs_at_start=False), model=model)
    tokens = _serve_tokens(case, prompts, seed)
    plan = [([(i, tokens[i][at:at + n], [n - 1] if want else []) for i, at, n, want in entries], ends) for entries, ends in steps]
    state = dict(kind="serve", engine=engine, plan=plan)
    run(state)      # a server warms up: the graphs of these steps' shapes are captured
    return state


def _run_serve(s):
    outs = [s["engine"].run_tokens(entries, ends) for entries, ends in s["plan"]]
    return [o for o in outs if o is not None]


def _rms(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _exact_serve(case, seed):
    steps, prompts = _serve_steps(case)
    tokens = _serve_tokens(case, prompts, seed)
    s = SIZES[case["size"]]
    H, G = s["heads"], s["kv"]
    lens = [len(t) for t in tokens]
    ids = torch.tensor([t for ts in tokens for t in ts], device=DEV)
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens]).double()
    angle = pos[:, None] * (500000.0 ** (-torch.arange(0, 128, 2, device=DEV).double() / 128))[None]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rope(z):
        a, b = z[..., :64], z[..., 64:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

    def product(x, w, name):
        if not case["fp8"]:
            return x @ w[name].double().T
        b = x.view(x.shape[0], -1, 128)        # activations enter as e4m3 with a scale per 128 columns
        scale = b.abs().amax(-1, keepdim=True).clamp_min(1e-12) / 448.0
        xq = ((b / scale).float().to(torch.float8_e4m3fn).double() * scale).view(x.shape)
        full = w["scales"][name].double().repeat_interleave(128, 0).repeat_interleave(128, 1)
        return xq @ (w[name].double() * full).T

    def attend(q, k, v):
        out = []
        for qs, ks, vs in zip(q.split(lens), k.split(lens), v.split(lens)):
            n = qs.shape[0]
            sc = torch.einsum("qgpd,kgd->gpqk", qs.view(n, G, H // G, 128), ks) / math.sqrt(128)
            sc.masked_fill_(torch.ones(n, n, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
            out.append(torch.einsum("gpqk,kgd->qgpd", torch.softmax(sc, -1), vs).reshape(n, H * 128))
        return torch.cat(out)

    for name, w in _serve_weights(case, seed):
        if name == "embed":
            x = w[ids].double()
        elif name == "final_norm":
            x = _rms(x, w)
        elif name == "lm_head":
            head = w.double()
        else:
            h = _rms(x, w["attn_norm"])
            T = h.shape[0]
            q, k = rope(product(h, w, "wq").view(T, H, 128)), rope(product(h, w, "wk").view(T, G, 128))
            x = x + product(attend(q, k, product(h, w, "wv").view(T, G, 128)), w, "wo")
            h = _rms(x, w["mlp_norm"])
            x = x + product(torch.nn.functional.silu(product(h, w, "w_gate")) * product(h, w, "w_up"), w, "w_down")
    first = [sum(lens[:i]) for i in range(len(lens))]
    outs = []
    for entries, _ in steps:
        # the engine's order: decode rows, then chunks; wanted rows come in the order of the entries, which is the same
        rows = [first[i] + at + n - 1 for i, at, n, want in entries if want]
        if rows:
            outs.append(x[torch.tensor(rows, device=DEV)] @ head.T)
    return outs


def _work_serve(case):
    steps, _ = _serve_steps(case)
    s = SIZES[case["size"]]
    W, F, H, G, L = s["width"], s["ffn"], s["heads"], s["kv"], case["layers"]
    params = W * (2 * H + 2 * G) * 128 + 3 * W * F
    nbytes = flops = 0.0
    for entries, _ in steps:
        rows, wanted = sum(n for _, _, n, _ in entries), sum(e[3] for e in entries)
        pairs = sum(n * at + n * (n + 1) / 2 for _, at, n, _ in entries)
        flops += L * (2.0 * rows * params + 4.0 * pairs * H * 128) + 2.0 * wanted * W * VOCAB
        nbytes += L * (params * (1 if case["fp8"] else 2) + sum(at + n for _, at, n, _ in entries) * G * 128 * 4) + (W * VOCAB * 2 + wanted * VOCAB * 2 if wanted else 0) + rows * W * 2
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------------------
# attention: chunks of prompts over a paged cache
# ------------------------------------------------------------------------------------------------------


def _chunks(case):
    """(rows, context) of every sequence."""
    if case["rows"] == 1:
        return [(1, c) for c in _lengths(case, case["seqs"], max(1, case["prefix"] // 4), case["prefix"])]
    rows = _lengths(case, case["seqs"], max(1, case["rows"] // 2), case["rows"])
    return [(n, n + p) for n, p in zip(rows, _lengths(case, case["seqs"], case["prefix"] // 4, case["prefix"], "p"))]


def _meta(case, seed):
    from mojo_b200 import ops

    lens = _chunks(case)
    pages, tables = _paged([c for _, c in lens], seed)
    cu = [0]
    for n, _ in lens:
        cu.append(cu[-1] + n)
    ctx = [c for _, c in lens]
    nd = len(lens) if case["rows"] == 1 else 0
    work = None
    if not nd:
        work = torch.from_numpy(ops.prefill_work_items(cu, ctx, 0)).to(DEV)
    meta = ops.AttnMeta(_int32(cu), _int32(ctx), tables.to(DEV), nd, max(n for n, _ in lens), max(ctx), work=work, n_items=0 if work is None else work.shape[0])
    return meta, pages


def _attention_inputs(case, seed, pages, rows):
    g = _gen(seed)
    kc, vc = (_randn(g, pages, case["kv"], PAGE, 128) for _ in range(2))
    return _randn(g, rows, case["heads"] * 128), kc, vc


def _prepare_attention(case, seed):
    from mojo_b200 import ops

    meta, pages = _meta(case, seed)
    q, kc, vc = _attention_inputs(case, seed, pages, sum(n for n, _ in _chunks(case)))
    return dict(kind="attention", q=q, kc=kc, vc=vc, meta=meta, mods=ops.ScoreMods(window=case["window"]))


def _run_attention(s):
    from mojo_b200 import ops

    return ops.paged_attention(s["q"], s["kc"], s["vc"], s["meta"], 128 ** -0.5, 128, mods=s["mods"])


def _seen(n, c, window):
    at, key = torch.arange(c - n, c, device=DEV)[:, None], torch.arange(c, device=DEV)[None]
    return (key <= at) & (key > at - window) if window else key <= at


def _exact_attention(case, seed):
    lens = _chunks(case)
    pages, tables = _paged([c for _, c in lens], seed)
    q, kc, vc = _attention_inputs(case, seed, pages, sum(n for n, _ in lens))
    H, per, out, at = case["heads"], case["heads"] // case["kv"], torch.empty(q.shape, dtype=torch.float64, device=DEV), 0
    for (n, c), table in zip(lens, tables.to(DEV)):
        hidden = ~_seen(n, c, case["window"])
        for h in range(H):
            k, v = (_cached(z[:, h // per], table, c).double() for z in (kc, vc))
            sc = (q[at:at + n, h * 128:(h + 1) * 128].double() @ k.T / math.sqrt(128)).masked_fill_(hidden, float("-inf"))
            out[at:at + n, h * 128:(h + 1) * 128] = torch.softmax(sc, -1) @ v
        at += n
    return out


def _pairs(case):
    w = case.get("window", 0)
    return sum(sum(min(p, w) if w else p for p in range(c - n + 1, c + 1)) for n, c in _chunks(case))


def _work_attention(case):
    keys = sum(min(c, n + case["window"]) if case["window"] else c for n, c in _chunks(case))
    return {"bytes": keys * case["kv"] * 512.0 + sum(n for n, _ in _chunks(case)) * case["heads"] * 512.0, "flops": 4.0 * 128 * case["heads"] * _pairs(case)}


# ------------------------------------------------------------------------------------------------------
# latent attention: the cached vector of a token is all that its heads see
# ------------------------------------------------------------------------------------------------------


def _latent_inputs(case, seed, pages):
    g, rows, H = _gen(seed), sum(n for n, _ in _chunks(case)), case["heads"]
    # queries are columns of one projection; latents are normed, the rotated part beside them is not
    return _randn(g, rows, H * 576 + 576, std=0.8), _randn(g, pages, PAGE, 576)


def _prepare_latent(case, seed):
    meta, pages = _meta(case, seed)
    qa, cache = _latent_inputs(case, seed, pages)
    H = case["heads"]
    return dict(kind="latent", q=qa[:, :H * 512].unflatten(1, (H, 512)), r=qa[:, H * 512:H * 576].unflatten(1, (H, 64)), cache=cache, meta=meta)


def _run_latent(s):
    from mojo_b200 import ops

    return ops.mla_attend(s["q"], s["r"], s["cache"], s["meta"], 192 ** -0.5)


def _exact_latent(case, seed):
    lens, H = _chunks(case), case["heads"]
    pages, tables = _paged([c for _, c in lens], seed)
    qa, cache = _latent_inputs(case, seed, pages)
    q = torch.cat([qa[:, :H * 512].unflatten(1, (H, 512)), qa[:, H * 512:H * 576].unflatten(1, (H, 64))], dim=2)
    out, at = torch.empty(q.shape[0], H, 512, dtype=torch.float64, device=DEV), 0
    for (n, c), table in zip(lens, tables.to(DEV)):
        kv, hidden = _cached(cache, table, c).double(), ~_seen(n, c, 0)
        for h in range(H):
            sc = (q[at:at + n, h].double() @ kv.T / math.sqrt(192)).masked_fill_(hidden, float("-inf"))
            out[at:at + n, h] = torch.softmax(sc, -1) @ kv[:, :512]
        at += n
    return out


def _work_latent(case):
    lens, H = _chunks(case), case["heads"]
    return {"bytes": sum(c for _, c in lens) * 1152.0 + sum(n for n, _ in lens) * H * (576 + 512) * 2.0, "flops": 2.0 * H * (576 + 512) * _pairs(case)}


# ------------------------------------------------------------------------------------------------------
# experts: routing, the chosen experts' products, their weighted sum into the residual and the next norm
# ------------------------------------------------------------------------------------------------------

EXPERTS, TOP = 64, 6


def _expert_inputs(case, seed):
    g, W, F, T = _gen(seed), case["width"], case["ffn"], case["rows"]
    return dict(h=_randn(g, T, W), x=_randn(g, T, W, dtype=torch.float32), norm=1.0 + _randn(g, W, std=0.1, dtype=torch.float32), router=_randn(g, EXPERTS, W, std=0.03),
                w_gu=_randn(g, EXPERTS, 2 * F, W, std=0.02), w_down=_randn(g, EXPERTS, W, F, std=0.02))


def _prepare_experts(case, seed):
    from mojo_b200 import ops

    d = _expert_inputs(case, seed)
    d["p"] = ops.MoeWeights(d.pop("router"), d.pop("w_gu"), d.pop("w_down"), EXPERTS, TOP, scoring=case["scoring"], norm_top=case["scoring"] == "sigmoid")
    return dict(kind="experts", **d)


def _run_experts(s):
    from mojo_b200 import ops

    done = ops.Finished(None, experts=ops.moe_experts(s["h"], s["p"]))
    return ops.residual_norm(s["x"], s["norm"], 1e-5, BF16, done, store=False)


def _exact_experts(case, seed):
    d = _expert_inputs(case, seed)
    h, T, W = d["h"].double(), case["rows"], case["width"]
    logits = h @ d["router"].double().T
    scores = torch.softmax(logits, -1) if case["scoring"] == "softmax" else torch.sigmoid(logits)
    weights, ids = scores.gather(1, logits.topk(TOP, dim=-1).indices), logits.topk(TOP, dim=-1).indices
    if case["scoring"] == "sigmoid":
        weights = weights / weights.sum(-1, keepdim=True)
    x = d["x"].double()
    for e in range(EXPERTS):
        tok, j = torch.where(ids == e)
        if tok.numel():
            gu = (h[tok] @ d["w_gu"][e].double().T).view(len(tok), -1, 2, 16)      # gate and up rows interleaved in blocks of 16
            act = (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).reshape(len(tok), -1)
            x.index_add_(0, tok, (act @ d["w_down"][e].double().T) * weights[tok, j][:, None])
    return _rms(x, d["norm"])


def _work_experts(case):
    T, W, F = case["rows"], case["width"], case["ffn"]
    used = EXPERTS * (1 - (1 - TOP / EXPERTS) ** T)
    return {"bytes": used * 3 * W * F * 2.0 + T * W * 8.0 + EXPERTS * W * 2.0, "flops": 2.0 * T * TOP * 3 * W * F + 2.0 * T * W * EXPERTS}


# ------------------------------------------------------------------------------------------------------
# packed: a gated feed-forward whose weights stay in k-quant blocks
# ------------------------------------------------------------------------------------------------------

Q4_K, Q6_K = 12, 14


def _packed_inputs(case, seed):
    s, g = SIZES[case["size"]], _gen(seed)
    W, F = s["width"], s["ffn"]

    def half(n, lo, hi):
        return (torch.rand(n, generator=g, device=DEV) * (hi - lo) + lo).to(torch.float16).view(torch.uint8).view(n, 2)

    def raw(n, size):
        return torch.randint(0, 256, (n, size), generator=g, device=DEV, dtype=torch.uint8)

    n4, n6 = 2 * F * W // 256, F * W // 256
    b4, b6 = raw(n4, 144), raw(n6, 210)
    b4[:, 0:2], b4[:, 2:4] = half(n4, 0.5e-4, 1.5e-4), half(n4, 3.7e-4, 11e-4)
    b6[:, 208:210] = half(n6, 1e-5, 2e-5)
    return _randn(g, case["rows"], W), b4, b6


def _prepare_packed(case, seed):
    x, b4, b6 = _packed_inputs(case, seed)
    s = SIZES[case["size"]]
    return dict(kind="packed", x=x, gate_up=b4.view(-1), down=b6.view(-1), ffn=s["ffn"], width=s["width"])


def _run_packed(s):
    from mojo_b200 import ops

    act = ops.swiglu(ops.linear_gguf(s["x"], s["gate_up"], ops.GGML_Q4_K, 2 * s["ffn"]))
    return ops.linear_gguf(act, s["down"], ops.GGML_Q6_K, s["width"])


def _unpack4(b):
    d, dmin = (b[:, i:i + 2].contiguous().view(torch.float16).double() for i in (0, 2))
    sc, q = b[:, 4:16].int(), b[:, 16:].int().view(-1, 4, 32)
    low, high = sc[:, 0:4], sc[:, 4:8]
    scale = torch.cat([low & 63, (sc[:, 8:12] & 15) | ((low >> 6) << 4)], dim=1).double()
    least = torch.cat([high & 63, (sc[:, 8:12] >> 4) | ((high >> 6) << 4)], dim=1).double()
    q = torch.stack([q & 15, q >> 4], dim=2).view(-1, 8, 32).double()
    return ((d * scale)[:, :, None] * q - (dmin * least)[:, :, None]).view(-1)


def _unpack6(b):
    low, high = b[:, :128].int().view(-1, 2, 1, 64), b[:, 128:192].int().view(-1, 2, 1, 32)
    low = torch.cat([low & 15, low >> 4], dim=2).view(-1, 2, 4, 32)
    high = torch.cat([(high >> (2 * i)) & 3 for i in range(4)], dim=2)
    scale = b[:, 192:208].contiguous().view(torch.int8).double().view(-1, 2, 4, 2, 1)
    d = b[:, 208:210].contiguous().view(torch.float16).double().view(-1, 1, 1, 1, 1)
    return (d * scale * ((low | (high << 4)) - 32).view(-1, 2, 4, 2, 16).double()).view(-1)


def _exact_packed(case, seed):
    x, b4, b6 = _packed_inputs(case, seed)
    s = SIZES[case["size"]]
    gu = x.double() @ _unpack4(b4).view(-1, s["width"]).T
    return (torch.nn.functional.silu(gu[:, :s["ffn"]]) * gu[:, s["ffn"]:]) @ _unpack6(b6).view(-1, s["ffn"]).T


def _work_packed(case):
    s, M = SIZES[case["size"]], case["rows"]
    W, F = s["width"], s["ffn"]
    return {"bytes": W * F / 256.0 * (2 * 144 + 210) + M * W * 4.0, "flops": 6.0 * M * W * F}


# ------------------------------------------------------------------------------------------------------
# sample: token ids drawn from a step's logits
# ------------------------------------------------------------------------------------------------------


def _prepare_sample(case, seed):
    g, n = _gen(seed), case["rows"]
    r = random.Random(repr(sorted(case.items(), key=str)))
    kinds = [r.choice([(0.7, 0, 0.9), (1.0, 50, 1.0), (0.8, 40, 0.95), (0.6, 20, 0.95), (1.0, 0, 0.95), (0.0, 0, 1.0)]) for _ in range(n)]
    return dict(kind="sample", logits=_randn(g, n, case["vocab"], std=2.5), temperature=torch.tensor([k[0] for k in kinds], device=DEV),
                top_k=_int32([k[1] for k in kinds]), top_p=torch.tensor([k[2] for k in kinds], device=DEV), seed=seed)


def _run_sample(s):
    from mojo_b200 import ops

    return ops.sample(s["logits"], s["temperature"], s["top_k"], s["top_p"], s["seed"], 3)


# ------------------------------------------------------------------------------------------------------
# recurrent layers: one decode row for each live sequence, and chunks that begin new ones
# ------------------------------------------------------------------------------------------------------

TAPS = 4


def _recurrent_lens(case):
    return [1] * case["decode"] + _lengths(case, case["chunks"], max(1, case["rows"] // 2), case["rows"])


def _seq_rows(case):
    from mojo_b200 import ops

    lens, nd, at, rows = _recurrent_lens(case), case["decode"], 0, []
    for n in lens:
        rows.append([at, at + n])
        at += n
    owner = [i for i, n in enumerate(lens) for _ in range(n)]
    banks = [[2 * i if i < nd else -1, 2 * i + 1] for i in range(len(lens))]
    return ops.SeqRows(_int32(owner), _int32(rows), _int32(banks), nd, nd, len(lens) - nd)


def _delta_inputs(case, seed):
    g, n, H, T = _gen(seed), len(_recurrent_lens(case)), case["heads"], sum(_recurrent_lens(case))
    C, dk = 3 * H * 128, H if case["per_head"] else H * 128
    return dict(proj=_randn(g, T, C + H), decay=_randn(g, T, dk), gate=_randn(g, T, H * 128), conv_w=_randn(g, TAPS, C, std=0.3, dtype=torch.float32),
                rate=-torch.exp(_randn(g, H, std=0.5, dtype=torch.float32)), dt_bias=_randn(g, dk, std=0.5, dtype=torch.float32) - 3.0,
                norm=1.0 + _randn(g, 128, std=0.1, dtype=torch.float32), bank=_randn(g, 2 * n, TAPS - 1, C), state=_randn(g, n, H, 128, 128, std=0.3, dtype=torch.float32))


def _prepare_delta(case, seed):
    from mojo_b200 import ops

    d = _delta_inputs(case, seed)
    p = ops.DeltaParams(d.pop("conv_w"), d.pop("rate"), d.pop("dt_bias"), d.pop("norm"), gate_silu=case["per_head"])
    return dict(kind="delta", p=p, seq=_seq_rows(case), heads=case["heads"], **d)


def _run_delta(s):
    from mojo_b200 import ops

    H = s["heads"]
    out = ops.delta_rule(s["proj"], s["decay"], s["gate"], s["p"], s["bank"], s["state"], s["seq"], 3 * H * 128, H, H, 128, 128, H * 128, 1e-5)
    return out, s["state"], s["bank"]


def _head_out(o, norm):
    return o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-5) * norm.double()


def _exact_delta(case, seed):
    d, lens, nd, H = _delta_inputs(case, seed), _recurrent_lens(case), case["decode"], case["heads"]
    C, T = 3 * H * 128, sum(lens)
    u, state, bank, outs, at = d["proj"][:, :C].double(), d["state"].double(), d["bank"].double(), [], 0
    beta = torch.sigmoid(d["proj"][:, C:].double()).view(T, H, 1)
    step = torch.nn.functional.softplus(d["decay"].double() + d["dt_bias"].double()).view(T, H, -1)
    decay = torch.exp(d["rate"].double()[None, :, None] * step).expand(T, H, 128)
    gate = d["gate"].double()
    gate = (torch.nn.functional.silu(gate) if case["per_head"] else torch.sigmoid(gate)).view(T, H, 128)
    new_state, new_bank = state.clone(), bank.clone()
    groups = ([(0, nd, 1)] if nd else []) + [(nd + i, nd + i + 1, n) for i, n in enumerate(lens[nd:])]
    for lo, hi, n in groups:      # all decode rows at once, every chunk by itself
        S = hi - lo
        cur = u[at:at + S * n].view(S, n, C)
        past = bank[2 * lo:2 * hi:2] if lo < nd else torch.zeros(S, TAPS - 1, C, dtype=torch.float64, device=DEV)
        line = torch.cat([past, cur], dim=1)
        conv = torch.nn.functional.silu(sum(line[:, t:t + n] * d["conv_w"][t].double() for t in range(TAPS)))
        new_bank[2 * lo + 1:2 * hi:2] = line[:, -(TAPS - 1):]
        q, k, v = conv.view(S, n, 3, H, 128).unbind(2)
        q, k = (z * torch.rsqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q = q * 128 ** -0.5
        g, b = decay[at:at + S * n].view(S, n, H, 128), beta[at:at + S * n].view(S, n, H, 1)
        M, out = state[lo:hi].clone() if lo < nd else torch.zeros(S, H, 128, 128, dtype=torch.float64, device=DEV), []
        for t in range(n):
            M = M * g[:, t, :, :, None]
            miss = (v[:, t] - torch.einsum("shk,shkv->shv", k[:, t], M)) * b[:, t]
            M = M + k[:, t, :, :, None] * miss[:, :, None]
            out.append(torch.einsum("shk,shkv->shv", q[:, t], M))
        new_state[lo:hi] = M
        outs.append(torch.stack(out, 1).view(S * n, H, 128))
        at += S * n
    return (_head_out(torch.cat(outs), d["norm"]) * gate).view(T, H * 128), new_state, new_bank


def _gated_inputs(case, seed):
    g, n, H, T = _gen(seed), len(_recurrent_lens(case)), case["heads"], sum(_recurrent_lens(case))
    return dict(proj=_randn(g, T, 4 * H * 128), z=_randn(g, T, H * 128, dtype=torch.float32), bias=_randn(g, H * 128, dtype=torch.float32) + 2.0,
                norm=1.0 + _randn(g, 128, std=0.1, dtype=torch.float32), state=_randn(g, n, H, 128, 128, std=3.0, dtype=torch.float32))


def _prepare_gated(case, seed):
    from mojo_b200 import ops

    d = _gated_inputs(case, seed)
    p = ops.GatedLinearParams(d.pop("bias"), d.pop("norm"), 16.0)
    return dict(kind="gated", p=p, seq=_seq_rows(case), heads=case["heads"], out=torch.empty(d["proj"].shape[0], case["heads"] * 128, dtype=BF16, device=DEV), **d)


def _run_gated(s):
    from mojo_b200 import ops

    return ops.gated_linear(s["proj"], s["z"], s["p"], s["state"], s["seq"], s["heads"], 128, 128, 1e-5, s["out"]), s["state"]


def _exact_gated(case, seed):
    d, lens, nd, H = _gated_inputs(case, seed), _recurrent_lens(case), case["decode"], case["heads"]
    T, state, outs, at = sum(lens), d["state"].double(), [], 0
    q, k, v, gate = d["proj"].double().view(T, 4, H, 128).unbind(1)
    a = torch.exp(torch.nn.functional.logsigmoid(d["z"].double() + d["bias"].double()) / 16.0).view(T, H, 128)
    new_state = state.clone()
    for lo, hi, n in ([(0, nd, 1)] if nd else []) + [(nd + i, nd + i + 1, n) for i, n in enumerate(lens[nd:])]:
        S = hi - lo
        M, out = state[lo:hi].clone() if lo < nd else torch.zeros(S, H, 128, 128, dtype=torch.float64, device=DEV), []
        qs, ks, vs, az = (z[at:at + S * n].view(S, n, H, 128) for z in (q, k, v, a))
        for t in range(n):
            M = M * az[:, t, :, :, None] + ks[:, t, :, :, None] * vs[:, t, :, None]
            out.append(torch.einsum("shk,shkv->shv", qs[:, t] * 128 ** -0.5, M))
        new_state[lo:hi] = M
        outs.append(torch.stack(out, 1).view(S * n, H, 128))
        at += S * n
    return (_head_out(torch.cat(outs), d["norm"]) * torch.nn.functional.silu(gate)).view(T, H * 128), new_state


def _work_recurrent(case, steps, row_bytes):
    T, H, n = sum(_recurrent_lens(case)), case["heads"], len(_recurrent_lens(case))
    return {"bytes": T * row_bytes * H * 128 + (n + case["decode"]) * H * 65536.0, "flops": 2.0 * steps * T * H * 128 * 128}


# ------------------------------------------------------------------------------------------------------

_PREPARE = dict(serve=_prepare_serve, attention=_prepare_attention, latent=_prepare_latent, experts=_prepare_experts, packed=_prepare_packed, sample=_prepare_sample,
                delta=_prepare_delta, gated=_prepare_gated)
_RUN = dict(serve=_run_serve, attention=_run_attention, latent=_run_latent, experts=_run_experts, packed=_run_packed, sample=_run_sample, delta=_run_delta, gated=_run_gated)
_EXACT = dict(serve=_exact_serve, attention=_exact_attention, latent=_exact_latent, experts=_exact_experts, packed=_exact_packed, delta=_exact_delta, gated=_exact_gated)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    make = _EXACT.get(case["kind"])      # sampled ids are whole numbers: nothing to be off by
    return None if make is None else make(case, seed)


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 2.0 * case["rows"] * case["vocab"], "flops": 4.0 * case["rows"] * case["vocab"]}
    if kind == "delta":       # q, k, v and the gate in, the result out; four multiply-adds per element of the state and row
        return _work_recurrent(case, 4, 10 if case["per_head"] else 12)
    if kind == "gated":
        return _work_recurrent(case, 3, 14)
    return dict(serve=_work_serve, attention=_work_attention, latent=_work_latent, experts=_work_experts, packed=_work_packed)[kind](case)


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    return {"rel": dict(serve=0.03 if case.get("fp8") else 0.02, attention=0.009, latent=0.008, experts=0.007, packed=0.018, delta=0.007, gated=0.007)[case["kind"]]}
