"""The framework's work, case by case: sizes, inputs, one pass, what it cannot do without, and its values in 64 bits.

A case is one call, or the short run of calls of one block, as the model runners make it: attention over the paged cache
and over prompts, whole decoder layers of a denoising step and of a prompt, the LM head with its sampler, the recurrences
and the latent attention of the causal designs, an expert feed-forward, and a whole fp32 prompt of a causal model.
Random weights of the sizes the benchmark names (width 2048 or 4096, heads of 128, vocabulary 32768 or 151936).
"""
import importlib
import math
import random

import torch

pkg = importlib.import_module("mineru-diffusion_b200")
ops = pkg.ops
hybrid = importlib.import_module("mineru-diffusion_b200.hybrid")
PAGE, HEAD, BF, F32, F64 = 256, 128, torch.bfloat16, torch.float32, torch.float64
DEV = "cuda"
EPS = 1e-6


def listed():
    return [
        # one request's block of masked tokens against its prefix: the smallest call, one per layer and step
        {"name": "block_attn_1", "kind": "block_attn", "bs": 1, "block": 32, "ctx": 1600, "hq": 16, "hkv": 8},
        # 64 requests in flight with prefixes between half of 8192 and 8192: the largest decode batch
        {"name": "block_attn_64", "kind": "block_attn", "bs": 64, "block": 32, "ctx": 8192, "hq": 16, "hkv": 8},
        # prompts: staircase attention of four long documents
        {"name": "prompt_attn_4x4096", "kind": "prompt_attn", "bs": 4, "len": 4096, "even": True, "hq": 16, "hkv": 8},
        # two layers of a denoising step of one request, replayed from a graph as the runner does
        {"name": "layers_denoise_1", "kind": "denoise", "bs": 1, "block": 32, "ctx": 1600},
        # two layers of one page image's prompt: 1024 visual rows and 32 ids
        {"name": "layers_prompt_1056", "kind": "prompt", "bs": 1, "len": 1056, "even": True},
        # LM head and sampler of one request's step
        {"name": "lm_head_32", "kind": "lm_head", "m": 32, "vocab": 151936, "hidden": 2048},
        # the gated delta rule over four prompts, with the decays it is given as projections
        {"name": "delta_4x2048", "kind": "delta", "bs": 4, "len": 2048, "even": True, "heads": 16},
        # the mLSTM over four prompts
        {"name": "mlstm_4x2048", "kind": "mlstm", "bs": 4, "len": 2048, "even": True, "heads": 8},
        # Mamba-2's recurrence over four prompts: 64 heads of 128 x 64, eight key heads
        {"name": "mamba_4x2048", "kind": "mamba", "bs": 4, "len": 2048, "even": True, "heads": 64},
        # latent attention of a decoding step of 32 requests
        {"name": "latent_32", "kind": "latent", "bs": 32, "ctx": 4096, "heads": 16},
        # an expert feed-forward of a prompt portion: six of 64 experts for each token
        {"name": "experts_2048", "kind": "experts", "m": 2048, "width": 2048, "ff": 1024},
        # a prompt through a whole causal model (delta rule, mLSTM, latent attention) in true fp32
        {"name": "causal_fp32_500", "kind": "causal", "len": 500, "width": 1024},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["block_attn", "prompt_attn", "denoise", "prompt", "lm_head", "delta", "mlstm", "mamba", "latent", "experts", "causal"])
    c = {"kind": kind}
    if kind in ("block_attn", "denoise"):
        c.update(bs=log(1, 64), block=rng.choice([8, 16, 32, 32, 64]), ctx=log(200, 8192 if kind == "block_attn" else 4096))
        if kind == "block_attn":
            c.update(zip(("hq", "hkv"), rng.choice([(16, 8), (16, 8), (32, 8), (8, 4)])))
        else:
            c["bs"] = min(c["bs"], 2048 // c["block"])
    elif kind in ("prompt_attn", "prompt", "delta", "mlstm", "mamba"):
        c.update(bs=rng.randint(1, 4), len=log(65, 4096 if kind == "prompt_attn" else 2048), even=False)
        if kind == "prompt_attn":
            c.update(zip(("hq", "hkv"), rng.choice([(16, 8), (16, 16), (8, 4)])))
        elif kind != "prompt":
            c["heads"] = {"delta": rng.randint(4, 16), "mlstm": rng.randint(2, 8), "mamba": 8 * rng.randint(1, 8)}[kind]
    elif kind == "lm_head":
        c.update(m=8 * log(1, 128), vocab=rng.choice([32768, 151936]), hidden=2048)
    elif kind == "latent":
        c.update(bs=log(1, 64), ctx=log(200, 8192), heads=rng.choice([16, 16, 32]))
    elif kind == "experts":
        c.update(m=log(1, 4096), width=2048, ff=rng.choice([512, 1024]))
    else:
        c.update(len=log(16, 500), width=rng.choice([512, 1024]))
    return c


# ----------------------------------------------------------------------------- sizes that follow from a case
def rng_of(case):
    return random.Random(str(sorted((k, v) for k, v in case.items() if k != "name")))


def lengths(case):
    """Rows of every prompt: all alike, or between half of the longest and the longest."""
    r, n = rng_of(case), case["len"]
    return [n] * case["bs"] if case["even"] else [n] + [r.randint(max(1, n // 2), n) for _ in range(case["bs"] - 1)]


def contexts(case):
    """Tokens each request attends to."""
    r, n = rng_of(case), case["ctx"]
    return [n + case.get("block", 0)] + [r.randint(max(1, n // 2), n) + case.get("block", 0) for _ in range(case["bs"] - 1)]


def offsets(counts):
    cu = [0]
    for n in counts:
        cu.append(cu[-1] + n)
    return cu


def int32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def paged(ctx, g):
    """Shuffled page list for requests of the given contexts: (page table, number of pages)."""
    need = [(n + PAGE - 1) // PAGE for n in ctx]
    perm = torch.randperm(sum(need), generator=torch.Generator().manual_seed(g.initial_seed()))
    table = torch.full((len(ctx), max(need)), -1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = perm[at:at + n].int()
        at += n
    return table.to(DEV), at


def randn(g, *shape, scale=1.0, dtype=BF):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def layers_config(layers):
    return pkg.DecoderConfig(vocab_size=1024, hidden_size=2048, intermediate_size=6144, num_hidden_layers=layers, num_attention_heads=16,
                             num_key_value_heads=8, head_dim=HEAD, max_position_embeddings=16384)


# ----------------------------------------------------------------------------- inputs
def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return dict(globals()["prepare_" + case["kind"]](case, g, seed), kind=case["kind"])


def prepare_block_attn(case, g, seed):
    bs, block, hq, hkv, ctx = case["bs"], case["block"], case["hq"], case["hkv"], contexts(case)
    table, pages = paged(ctx, g)
    q = randn(g, bs, block, hq, HEAD)
    kc, vc = randn(g, pages, PAGE, hkv, HEAD), randn(g, pages, PAGE, hkv, HEAD)
    ns = ops.default_nsplit(bs, block, hq, hkv, max(ctx))
    ws = torch.empty(max(16, ops.attn_workspace_bytes(bs, block, hq, ns)), dtype=torch.uint8, device=DEV)
    return dict(q=q, kc=kc, vc=vc, ctx=int32(ctx), table=table, max_ctx=max(ctx), ws=ws, out=torch.empty_like(q))


def prepare_prompt_attn(case, g, seed):
    n = lengths(case)
    m = sum(n)
    q, k, v = randn(g, m, case["hq"], HEAD), randn(g, m, case["hkv"], HEAD), randn(g, m, case["hkv"], HEAD)
    return dict(q=q, k=k, v=v, cu=int32(offsets(n)), longest=max(n), out=torch.empty_like(q))


def decoder(ctx_or_len, max_tokens, max_seqs, block, g, seed):
    """Two decoder layers with their cache, and the slots of the given rows."""
    cfg = layers_config(2)
    table, pages = paged(ctx_or_len, g)
    cache = randn(g, 2, 2, pages, PAGE, 8, HEAD)
    w = pkg.DecoderWeights.random_init(cfg, seed, DEV)
    return pkg.DecoderEngine(cfg, w, cache, max_tokens, max_seqs, block), w, table


def slots_of(table, spans):
    t = table.tolist()
    return int32([t[r][p // PAGE] * PAGE + p % PAGE for r, (lo, hi) in enumerate(spans) for p in range(lo, hi)])


def prepare_denoise(case, g, seed):
    bs, block, ctx = case["bs"], case["block"], contexts(case)
    m = bs * block
    engine, w, table = decoder(ctx, m, bs, block, g, seed)
    spans = [(n - block, n) for n in ctx]
    pos = torch.tensor([p for lo, hi in spans for p in range(lo, hi)], dtype=torch.int64, device=DEV)
    c = pkg.Context(slot_mapping=slots_of(table, spans), context_lens=int32(ctx), block_tables=table, block_size=block)
    engine.embeds[:m].copy_(randn(g, m, 2048, scale=0.5))
    nsplit = engine.attn_nsplit(bs, max(ctx))
    rows = engine.forward(m, pos, c, nsplit=nsplit)       # sets kernel attributes outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rows = engine.forward(m, pos, c, nsplit=nsplit)
    return dict(graph=graph, rows=rows, engine=engine, w=w, pos=pos, ctx=c, cu=offsets([block] * bs), lens=ctx)


def prepare_prompt(case, g, seed):
    n = lengths(case)
    m = sum(n)
    engine, w, table = decoder(n, m, case["bs"], 32, g, seed)
    cu = int32(offsets(n))
    pos = torch.cat([torch.arange(x, dtype=torch.int64) for x in n]).to(DEV)
    c = pkg.Context(is_prefill=True, cu_seqlens_q=cu, cu_seqlens_k=cu, slot_mapping=slots_of(table, [(0, x) for x in n]), block_tables=table,
                    block_size=32)
    engine.embeds[:m].copy_(randn(g, m, 2048, scale=0.5))
    return dict(engine=engine, w=w, pos=pos, ctx=c, m=m, longest=max(n), cu=offsets(n), lens=n)


def prepare_lm_head(case, g, seed):
    m, v, h = case["m"], case["vocab"], case["hidden"]
    return dict(x=randn(g, m, h), w=randn(g, v, h, scale=0.02), temps=torch.full((m // 8,), 1.0, device=DEV), seed=seed,
                ws=torch.empty(ops.lmhead_workspace_bytes(m, v), dtype=torch.uint8, device=DEV),
                x0=torch.empty(m, dtype=torch.int32, device=DEV), conf=torch.empty(m, device=DEV))


def portions(counts):
    cu, bs = offsets(counts), len(counts)
    return (int32([i for i, n in enumerate(counts) for _ in range(n)]), int32(cu), int32([0] * bs), int32(list(range(bs))))


def prepare_delta(case, g, seed):
    n, h = lengths(case), case["heads"]
    m, unit = sum(n), torch.nn.functional.normalize
    q = unit(torch.randn(m, h, HEAD, generator=g, device=DEV), dim=-1) * HEAD ** -0.5
    k = unit(torch.randn(m, h, HEAD, generator=g, device=DEV), dim=-1)
    v = randn(g, m, h, HEAD, dtype=F32)
    beta = torch.sigmoid(randn(g, m, h, dtype=F32))
    return dict(q=q, k=k, v=v, beta=beta, raw=randn(g, m, h * HEAD, dtype=F32), a_log=randn(g, h, dtype=F32) - 2.0, dt=randn(g, h * HEAD, dtype=F32),
                p=portions(n), lens=n, dec=torch.empty(m, h, HEAD, device=DEV), scalars=torch.empty(m, h, 4, device=DEV),
                state=torch.zeros(len(n), h, HEAD, HEAD, device=DEV), out=torch.empty(m, h, HEAD, device=DEV))


def prepare_mlstm(case, g, seed):
    n, h, vd = lengths(case), case["heads"], 256
    m, cap = sum(n), 15.0
    li = cap * torch.tanh(randn(g, m, h, dtype=F32) / cap)
    lf = torch.nn.functional.logsigmoid(cap * torch.tanh((randn(g, m, h, dtype=F32) + 3.0) / cap))
    return dict(q=randn(g, m, h, HEAD).float() * HEAD ** -0.5, k=randn(g, m, h, HEAD).float(), v=randn(g, m, h, vd).float(), li=li, lf=lf,
                p=portions(n), lens=n, state=torch.zeros(len(n), h, vd + 1, HEAD, device=DEV),
                mst=torch.zeros(len(n), h, ops.scan_blocks(vd), device=DEV), out=torch.empty(m, h, vd, device=DEV), den=torch.empty(m, h, device=DEV))


def prepare_mamba(case, g, seed):
    n, h, kvh, vd = lengths(case), case["heads"], 8, 64
    m, silu = sum(n), torch.nn.functional.silu
    step = torch.nn.functional.softplus(randn(g, m, h, dtype=F32))
    return dict(q=silu(randn(g, m, kvh * HEAD, dtype=F32)).to(BF), k=silu(randn(g, m, kvh * HEAD, dtype=F32)).to(BF),
                v=silu(randn(g, m, h * vd, dtype=F32)).to(BF), step=step, log_decay=-step * torch.exp(randn(g, h, dtype=F32) - 2.0),
                skip=1.0 + 0.3 * randn(g, h, dtype=F32), p=portions(n), lens=n, kvh=kvh, longest=max(n),
                state=torch.zeros(len(n), h, vd, HEAD, device=DEV), out=torch.empty(m, h, vd, device=DEV))


def prepare_latent(case, g, seed):
    bs, heads, width, ctx = case["bs"], case["heads"], 512, contexts(case)
    table, pages = paged(ctx, g)
    ns = hybrid.key_parts(bs * -(-heads // 16), max(ctx))
    return dict(q=randn(g, bs, heads * width), cache=randn(g, pages * PAGE, width), table=table, row_seq=int32(list(range(bs))),
                row_pos=int32([n - 1 for n in ctx]), heads=heads, scale=width ** -0.5, nsplit=ns, lens=ctx, out=torch.empty(bs, heads * width, dtype=BF, device=DEV),
                ws=torch.empty(max(16, ops.latent_attn_workspace_bytes(bs, heads, width, ns)), dtype=torch.uint8, device=DEV))


EXPERTS, TOP = 64, 6


def prepare_experts(case, g, seed):
    m, w, ff = case["m"], case["width"], case["ff"]
    tiles = ops.moe_max_tiles(m, TOP, EXPERTS)
    rows, new = tiles * 128, lambda *s, dtype: torch.empty(*s, dtype=dtype, device=DEV)
    return dict(h=randn(g, m, w), z=randn(g, m, EXPERTS, dtype=F32), up=randn(g, EXPERTS, ff, w, scale=w ** -0.5), down=randn(g, EXPERTS, w, ff, scale=ff ** -0.5),
                norm=1.0 + 0.1 * randn(g, w, dtype=F32), residual=randn(g, m, w, dtype=F32), tiles=tiles, ids=new(m, TOP, dtype=torch.int32),
                weights=new(m, TOP, dtype=F32), slot=new(m, TOP, dtype=torch.int32), row_token=new(rows, dtype=torch.int32),
                tile_expert=new(tiles, dtype=torch.int32), num_tiles=new(4, dtype=torch.int32), xs=new(rows, w, dtype=BF),
                act=new(rows, ff, dtype=BF), ys=new(rows, w, dtype=BF), y=new(m, w, dtype=BF))


def causal_config(width):
    heads, dense = width // 128, {"kind": "dense", "ff": 3 * width}
    return {"architecture": "Zikunex", "vocab": 2048, "width": width, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "layers": [
        {"type": "channel_delta", "mixer": dict(heads=heads, kv_heads=heads, dim=128, vdim=128, conv=4), "mlp": dense},
        {"type": "latent_attention", "mixer": dict(heads=heads, dim=128, vdim=128, q_rank=384, kv_rank=256, scale=128 ** -0.5), "mlp": dense},
        {"type": "mlstm", "mixer": dict(heads=heads // 2, dim=128, vdim=256, gate_cap=15.0), "mlp": dense}]}


def prepare_causal(case, g, seed):
    n = case["len"]
    cfg = pkg.HybridConfig.from_json(causal_config(case["width"]))
    tensors = hybrid.random_tensors(cfg, seed, DEV)
    weights = hybrid.HybridWeights.build(cfg, dict(tensors), DEV, F32)
    config = pkg.Config(max_num_seqs=16, max_model_len=512, max_num_batched_tokens=512, num_kvcache_blocks=2, decoder_config=cfg, dtype="float32",
                        enforce_eager=True, num_state_slots=1)
    seq = pkg.CausalSequence(torch.randint(0, 2048, (n,), generator=torch.Generator().manual_seed(seed)).tolist())
    seq.block_table, seq.state_slot, seq.num_cached_tokens = [0, 1], 0, 0
    return dict(runner=pkg.CausalModelRunner(config, weights=weights), seq=seq, n=n, tensors=tensors, want=[(0, p) for p in wanted(n)])


def wanted(n):
    """The last 16 positions of a prompt, whose logits a caller asks for."""
    return list(range(n - 16, n))


# ----------------------------------------------------------------------------- one pass
def run(s):
    return globals()["run_" + s["kind"]](s)


def run_block_attn(s):
    return ops.block_attn_with_kvcache(s["q"], s["kc"], s["vc"], s["ctx"], s["table"], max_ctx=s["max_ctx"], workspace=s["ws"], out=s["out"])


def run_prompt_attn(s):
    return ops.sparse_attn_varlen(s["q"], s["k"], s["v"], s["cu"], s["cu"], 32, max_seqlen=s["longest"], out=s["out"])


def run_denoise(s):
    s["graph"].replay()
    return s["rows"]


def run_prompt(s):
    return s["engine"].forward(s["m"], s["pos"], s["ctx"], max_seqlen=s["longest"])


def run_lm_head(s):
    return ops.lm_head_sample(s["x"], s["w"], s["temps"], 8, seed=s["seed"], step=3, workspace=s["ws"], x0=s["x0"], conf=s["conf"])


def run_delta(s):
    m, h = s["beta"].shape
    ops.channel_decay(s["raw"], s["a_log"], s["dt"], s["q"], s["k"], s["beta"], s["p"], s["dec"], s["scalars"], HEAD)
    ops.scan(ops.SCAN_DELTA, BF, len(s["lens"]), h, h, HEAD, HEAD, s["q"], s["k"], s["v"], s["beta"], None, s["state"], s["p"], g=s["dec"],
             scalars=s["scalars"], out=s["out"])
    return s["out"], s["state"]


def run_mlstm(s):
    h = s["li"].shape[1]
    ops.scan(ops.SCAN_MLSTM, BF, len(s["lens"]), h, h, HEAD, 256, s["q"], s["k"], s["v"], s["li"], s["lf"], s["state"], s["p"], mstate=s["mst"],
             out=s["out"], den=s["den"])
    return s["out"], s["den"], s["state"], s["mst"]


def run_mamba(s):
    ops.chunk_scan(len(s["lens"]), s["step"].shape[1], s["kvh"], HEAD, 64, s["q"], s["k"], s["v"], s["log_decay"], s["step"], s["state"], s["p"],
                   s["longest"], s["out"], skip=s["skip"])
    return s["out"], s["state"]


def run_latent(s):
    ops.latent_attn(s["q"], s["cache"], s["table"], s["row_seq"], s["row_pos"], s["heads"], s["scale"], s["out"], s["nsplit"], s["ws"])
    return s["out"]


def run_experts(s):
    m, w = s["h"].shape
    ops.moe_route(ops.Rows(s["z"]), m, EXPERTS, TOP, 8, 4, s["ids"], s["weights"])
    ops.moe_plan(s["ids"], EXPERTS, s["tiles"], s["slot"], s["row_token"], s["tile_expert"], s["num_tiles"])
    ops.moe_gather(s["h"], s["xs"], s["row_token"], s["num_tiles"], s["tiles"])
    ops.gemm_experts(s["xs"], s["up"], s["act"], s["tile_expert"], s["num_tiles"], m, act=ops.ACT_RELU2)
    ops.gemm_experts(s["act"], s["down"], s["ys"], s["tile_expert"], s["num_tiles"], m)
    ops.residual_norm(s["residual"], w, 1e-5, BF, weight=s["norm"], out=s["y"], moe=(s["ys"], s["slot"], s["weights"]))
    return s["y"], s["residual"]


def run_causal(s):
    return s["runner"].execute([s["seq"]], [s["n"]], s["want"])[0]


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    k = case["kind"]
    if k == "block_attn":
        keys, hq, hkv, b = sum(contexts(case)), case["hq"], case["hkv"], case["block"]
        return {"bytes": 2 * (2 * keys * hkv + 2 * case["bs"] * b * hq) * HEAD, "flops": 4 * keys * b * hq * HEAD}
    if k == "prompt_attn":
        n, hq, hkv = lengths(case), case["hq"], case["hkv"]
        return {"bytes": 2 * sum(n) * 2 * (hq + hkv) * HEAD, "flops": 4 * hq * HEAD * pairs(n)}
    if k in ("denoise", "prompt"):
        n = contexts(case) if k == "denoise" else lengths(case)
        m = case["bs"] * case["block"] if k == "denoise" else sum(n)
        p = case["block"] * sum(n) if k == "denoise" else pairs(n)
        weights = 2 * (4096 * 2048 + 2048 * 2048 + 3 * 6144 * 2048)
        kv = 2 * 2 * sum(n) * 8 * HEAD * 2
        return {"bytes": 2 * weights + kv + 2 * m * 2048 * 2, "flops": 2 * m * weights + 2 * 4 * 16 * HEAD * p}
    if k == "lm_head":
        m, v, h = case["m"], case["vocab"], case["hidden"]
        return {"bytes": 2 * (m + v) * h + 8 * m, "flops": 2 * m * v * h}
    if k in ("delta", "mlstm", "mamba"):
        m, h = sum(lengths(case)), case["heads"]
        vd = {"delta": 128, "mlstm": 256, "mamba": 64}[k]
        state = case["bs"] * h * (vd + (k == "mlstm")) * HEAD * 4
        io = {"delta": h * 4 * (3 * HEAD + 2 * vd + 1), "mlstm": h * 4 * (2 * HEAD + 2 * vd + 3), "mamba": 2 * 2 * 8 * HEAD + h * (6 * vd + 8)}[k]
        return {"bytes": m * io + state, "flops": m * h * vd * HEAD * {"delta": 8, "mlstm": 6, "mamba": 4}[k]}
    if k == "latent":
        keys, heads = sum(contexts(case)), case["heads"]
        return {"bytes": 2 * (keys + 2 * case["bs"] * heads) * 512, "flops": 4 * keys * heads * 512}
    if k == "experts":
        m, w, ff = case["m"], case["width"], case["ff"]
        touched = min(EXPERTS, m * TOP)
        return {"bytes": touched * 2 * w * ff * 2 + m * (w * (2 + 8 + 2) + EXPERTS * 4), "flops": 4 * m * TOP * w * ff}
    n, w = case["len"], case["width"]
    h = w // 128
    per = 3 * 6 * w * w + w * (4 * w + 256 + h) + 256 * w + (384 + 256) * w + 384 * w + 512 * w + w * w + w * (5 * w + w)
    return {"bytes": 4 * per + 4 * 2048 * w + 16 * 2048 * 4, "flops": 2 * n * per + 16 * 2 * 2048 * w + n * h * 128 * 128 * 14 + 2 * h * 128 * n * n}


def pairs(n):
    """(query, key) pairs of staircases of 32 over sequences of the given lengths, from the sequence's end."""
    total = 0
    for t in n:
        pad = -t % 32
        total += sum(min(t, ((i + pad) // 32 + 1) * 32 - pad) for i in range(t))
    return total


def tolerance(case):
    """About four times the distance from `exact` that was measured (attention 0.0023 - 0.0027, two bf16 layers 0.0065, recurrences
    2e-7 - 2e-6, experts 0.002, fp32 model 2.6e-6)."""
    return {
        "block_attn": {"rel": 0.01}, "prompt_attn": {"rel": 0.012}, "denoise": {"rel": 0.025}, "prompt": {"rel": 0.025},
        "lm_head": {"rel": 1e-3, "differ": 0.005}, "delta": {"rel": 1e-5}, "mlstm": {"rel": 1e-5}, "mamba": {"rel": 1e-5},
        "latent": {"rel": 0.008}, "experts": {"rel": 0.008}, "causal": {"rel": 1.5e-5},
    }[case["kind"]]


# ----------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    with torch.no_grad():
        return globals()["exact_" + case["kind"]](case, prepare(case, seed))


def paged_rows(cache, table, i, n):
    """The first n cached rows of request i."""
    pages = table[i, :(n + PAGE - 1) // PAGE].long()
    return cache[pages].flatten(0, 1)[:n].to(F64)


def attend(q, k, v, scale, mask=None):
    """q [t, hq, d], k and v [n, hkv, d]."""
    out, rep = torch.empty_like(q), q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // rep].T * scale
        if mask is not None:
            s.masked_fill_(~mask, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h // rep]
    return out


def stairs(t, size=32):
    i = torch.arange(t, device=DEV)
    pad = -t % size
    last = torch.clamp(((i + pad) // size + 1) * size - pad, max=t)
    return i[None, :] < last[:, None]


def exact_block_attn(case, s):
    out = torch.empty(s["q"].shape, dtype=F64, device=DEV)
    for i, n in enumerate(contexts(case)):
        out[i] = attend(s["q"][i].to(F64), paged_rows(s["kc"], s["table"], i, n), paged_rows(s["vc"], s["table"], i, n), HEAD ** -0.5)
    return out


def exact_prompt_attn(case, s):
    out, cu = torch.empty(s["q"].shape, dtype=F64, device=DEV), offsets(lengths(case))
    for a, b in zip(cu, cu[1:]):
        out[a:b] = attend(*(s[x][a:b].to(F64) for x in "qkv"), HEAD ** -0.5, stairs(b - a))
    return out


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def exact_layers(s, is_prompt):
    eng, pos, cu, ctx = s["engine"], s["pos"], s["cu"], s["ctx"]
    m = cu[-1]
    eps = eng.cfg.rms_norm_eps
    inv = 1.0 / (eng.cfg.rope_theta ** (torch.arange(0, HEAD, 2, dtype=F64, device=DEV) / HEAD))
    ang = pos.reshape(-1).to(F64)[:, None] * inv
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def rope(x):
        a, b = x[..., :64], x[..., 64:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    x = eng.embeds[:m].to(F64)
    for li, w in enumerate(s["w"].layers):
        h = rms(x, eps) * w.input_ln.to(F64)
        z = (h @ w.qkv.to(F64).T).view(m, 32, HEAD)
        q, k, v = rope(rms(z[:, :16], eps) * w.q_norm.to(F64)), rope(rms(z[:, 16:24], eps) * w.k_norm.to(F64)), z[:, 24:]
        o = torch.empty_like(q)
        for i, (a, b) in enumerate(zip(cu, cu[1:])):
            if is_prompt:
                o[a:b] = attend(q[a:b], k[a:b], v[a:b], HEAD ** -0.5, stairs(b - a))
            else:
                n = s["lens"][i]
                kk, vv = (paged_rows(eng.kv_cache[j, li], ctx.block_tables, i, n) for j in range(2))
                kk[n - (b - a):], vv[n - (b - a):] = k[a:b], v[a:b]
                o[a:b] = attend(q[a:b], kk, vv, HEAD ** -0.5)
        x = x + o.flatten(1) @ w.o.to(F64).T
        h = rms(x, eps) * w.post_ln.to(F64)
        gate, up = (h @ w.gate_up.to(F64).T).chunk(2, -1)
        x = x + (torch.nn.functional.silu(gate) * up) @ w.down.to(F64).T
    return rms(x, eps) * s["w"].final_ln.to(F64)


def exact_denoise(case, s):
    return exact_layers(s, False)


def exact_prompt(case, s):
    return exact_layers(s, True)


def exact_lm_head(case, s):
    return None          # the choice depends on the library's own noise


def exact_delta_scan(q, k, v, g, beta, lens):
    """Every sequence token by token, all sequences at once: [m, heads, ...] in, outputs and states [v, k] out."""
    cu, bs, h, d, vd = offsets(lens), len(lens), q.shape[1], q.shape[2], v.shape[2]
    S = torch.zeros(bs, h, d, vd, dtype=F64, device=DEV)
    out = torch.empty(v.shape, dtype=F64, device=DEV)
    order = sorted(range(bs), key=lambda i: -lens[i])
    at = torch.tensor([cu[i] for i in order], device=DEV)
    for t in range(max(lens)):
        n = sum(lens[i] > t for i in order)
        r = at[:n] + t
        T = S[:n] * g[r][..., None]
        u = beta[r][..., None] * (v[r] - torch.einsum("bhdv,bhd->bhv", T, k[r]))
        T += k[r][..., None] * u[:, :, None]
        S[:n] = T
        out[r] = torch.einsum("bhdv,bhd->bhv", T, q[r])
    back = torch.empty_like(S)
    back[torch.tensor(order, device=DEV)] = S
    return out, back.transpose(2, 3)


def exact_delta(case, s):
    h = case["heads"]
    d = {k: s[k].to(F64) for k in ("q", "k", "v", "beta", "raw", "a_log", "dt")}
    g = torch.exp(-torch.exp(d["a_log"])[None, :, None] * torch.nn.functional.softplus(d["raw"] + d["dt"]).view(-1, h, HEAD))
    return exact_delta_scan(d["q"], d["k"], d["v"], g, d["beta"], s["lens"])


def exact_mlstm_scan(q, k, v, li, lf, lens):
    """Numerator, denominator, state [v | normaliser, k] and running maximum of every sequence."""
    cu, bs, h, d, vd = offsets(lens), len(lens), q.shape[1], q.shape[2], v.shape[2]
    out, den = torch.empty(v.shape, dtype=F64, device=DEV), torch.empty(q.shape[:2], dtype=F64, device=DEV)
    order = sorted(range(bs), key=lambda i: -lens[i])
    at = torch.tensor([cu[i] for i in order], device=DEV)
    S, m = torch.zeros(bs, h, d, vd + 1, dtype=F64, device=DEV), torch.zeros(bs, h, dtype=F64, device=DEV)
    v1 = torch.cat([v, torch.ones_like(v[..., :1])], -1)
    for t in range(max(lens)):
        n = sum(lens[i] > t for i in order)
        r = at[:n] + t
        new = torch.maximum(lf[r] + m[:n], li[r])
        S[:n] = torch.exp(lf[r] + m[:n] - new)[..., None, None] * S[:n] + (torch.exp(li[r] - new)[..., None] * k[r])[..., None] * v1[r][:, :, None]
        m[:n] = new
        num = torch.einsum("bhdv,bhd->bhv", S[:n], q[r])
        out[r], den[r] = num[..., :vd], torch.maximum(num[..., vd].abs(), torch.exp(-new)) + 1e-6
    back, top = torch.empty_like(S), torch.empty_like(m)
    back[torch.tensor(order, device=DEV)], top[torch.tensor(order, device=DEV)] = S, m
    return out, den, back.transpose(2, 3), top


def exact_mlstm(case, s):
    out, den, state, top = exact_mlstm_scan(*(s[k].to(F64) for k in ("q", "k", "v", "li", "lf")), s["lens"])
    return out, den, state, top[..., None].expand(s["mst"].shape)


def exact_mamba(case, s):
    lens, h = s["lens"], case["heads"]
    cu, rep = offsets(lens), h // s["kvh"]
    m = cu[-1]
    q, k = (s[x].to(F64).view(m, s["kvh"], HEAD).repeat_interleave(rep, 1) for x in "qk")
    v, step, g = s["v"].to(F64).view(m, h, 64), s["step"].to(F64), torch.exp(s["log_decay"].to(F64))
    out, S = torch.empty(m, h, 64, dtype=F64, device=DEV), torch.zeros(len(lens), h, 64, HEAD, dtype=F64, device=DEV)
    order = sorted(range(len(lens)), key=lambda i: -lens[i])
    at = torch.tensor([cu[i] for i in order], device=DEV)
    for t in range(max(lens)):
        n = sum(lens[i] > t for i in order)
        r = at[:n] + t
        S[:n] = g[r][..., None, None] * S[:n] + (step[r][..., None] * v[r])[..., None] * k[r][:, :, None]
        out[r] = torch.einsum("bhvd,bhd->bhv", S[:n], q[r]) + s["skip"].to(F64)[None, :, None] * v[r]
    back = torch.empty_like(S)
    back[torch.tensor(order, device=DEV)] = S
    return out, back


def exact_latent(case, s):
    out = torch.empty(case["bs"], case["heads"], 512, dtype=F64, device=DEV)
    cache = s["cache"].view(-1, PAGE, 512)
    for i, n in enumerate(s["lens"]):
        c = paged_rows(cache, s["table"], i, n)
        p = torch.softmax(s["q"][i].view(-1, 512).to(F64) @ c.T * s["scale"], -1)
        out[i] = p @ c
    return out.flatten(1)


def exact_experts(case, s):
    m, z = case["m"], torch.softmax(s["z"].to(F64), -1)
    kept = z.view(m, 8, 8).max(-1).values.topk(4, -1).indices
    allowed = torch.zeros(m, 8, dtype=torch.bool, device=DEV).scatter_(1, kept, True).repeat_interleave(8, 1)
    ids = z.masked_fill(~allowed, -1.0).topk(TOP, -1).indices
    w = z.gather(1, ids)
    w = w / (w.sum(-1, keepdim=True) + 1e-20)
    res, h = s["residual"].to(F64), s["h"].to(F64)
    for e in range(EXPERTS):
        rows, slot = (ids == e).nonzero(as_tuple=True)
        if len(rows):
            a = torch.relu(h[rows] @ s["up"][e].to(F64).T) ** 2
            res[rows] += w[rows, slot][:, None] * (a @ s["down"][e].to(F64).T)
    return rms(res, 1e-5) * s["norm"].to(F64), res


def exact_causal(case, s):
    w, cfg, n = {k: v.to(F64) for k, v in s["tensors"].items()}, causal_config(case["width"]), case["len"]
    x = w["embed"][torch.tensor(s["seq"].token_ids, device=DEV)]
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)      # noqa: E731
    for i, layer in enumerate(cfg["layers"]):
        mx, get = layer["mixer"], lambda name: w[f"l{i}.mix.{name}"]           # noqa: E731,B023
        h, H = rms(x, 1e-5) * w[f"l{i}.norm1"], mx["heads"]
        if layer["type"] == "channel_delta":
            def conv(name):
                z, taps = h @ get(name).T, get(name + ".conv")                 # noqa: B023
                z = torch.cat([torch.zeros(3, z.shape[1], dtype=F64, device=DEV), z])
                return torch.nn.functional.silu(sum(z[j:j + n] * taps[:, j] for j in range(4))).view(n, H, 128)     # noqa: B023
            q, k, v = unit(conv("q")) * 128 ** -0.5, unit(conv("k")), conv("v")
            a = (h @ get("a1").T) @ get("a2").T + get("dt_bias")
            g = torch.exp(-torch.exp(get("A_log"))[None, :, None] * torch.nn.functional.softplus(a).view(n, H, 128))
            o = exact_delta_scan(q, k, v, g, torch.sigmoid(h @ get("b").T), [n])[0]
            o = rms(o, 1e-5) * get("norm") * torch.sigmoid((h @ get("g1").T) @ get("g2").T).view(n, H, 128)
            y = o.flatten(1) @ get("o").T
        elif layer["type"] == "latent_attention":
            q = ((rms(h @ get("dq").T, 1e-5) * get("dq.norm")) @ get("uq").T).view(n, H, 128)
            c = rms(h @ get("dkv").T, 1e-5) * get("dkv.norm")
            mask = torch.ones(n, n, dtype=torch.bool, device=DEV).tril()
            y = attend(q, (c @ get("uk").T).view(n, H, 128), (c @ get("uv").T).view(n, H, 128), mx["scale"], mask).flatten(1) @ get("o").T
        else:
            cap = mx["gate_cap"]
            q, k, v = (h @ get("q").T).view(n, H, 128) * 128 ** -0.5, (h @ get("k").T).view(n, H, 128), (h @ get("v").T).view(n, H, 256)
            li = cap * torch.tanh((h @ get("i").T + get("i.b")) / cap)
            lf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ get("f").T + get("f.b")) / cap))
            num, den, _, _ = exact_mlstm_scan(q, k, v, li, lf, [n])
            o = rms(num / den[..., None], 1e-5).flatten(1)
            y = (o * get("norm") * torch.sigmoid(h @ get("g").T)) @ get("o").T
        x = x + y
        h = rms(x, 1e-5) * w[f"l{i}.norm2"]
        x = x + torch.relu(h @ w[f"l{i}.mlp.up"].T) ** 2 @ w[f"l{i}.mlp.down"].T
    x = (rms(x, 1e-5) * w["final.norm"])[wanted(n)]
    return x @ w["head"].T
