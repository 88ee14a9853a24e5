"""Kernel forms at the edges of their tiles and dispatch rules: pairs of query tiles, shares of latent tiles, pairs of expert
tiles."""
import importlib

import pytest
import torch

pkg = importlib.import_module("mineru-diffusion_b200")
ops = pkg.ops
pytestmark = pytest.mark.gpu
DEV, BF, F64 = "cuda", torch.bfloat16, torch.float64


def gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm().clamp_min(1e-30))


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# One, two and three query tiles per sequence (tiles of 128 / group tokens), a tile alone in its pair before and after whole
# pairs, few tiles (one per unit) and more units than SMs.  P and the output are bf16: 2^-9 relative each.
@pytest.mark.parametrize("hq,hkv", [(16, 8), (6, 2), (16, 2), (4, 4)])
@pytest.mark.parametrize("lens", [[64], [1, 65, 129, 190], [700, 33, 64, 1000, 5, 321] * 4])
def test_prompt_attention_pairs(hq, hkv, lens):
    _prompts(hq, hkv, lens)


# Several waves of CTAs in which a unit of one tile and one tile of keys comes behind a whole pair, behind its like, and in front of
# a pair: the warps of the tile that is not there have to see every unit's queries arrive.
def test_prompt_attention_tiles_alone_behind_pairs():
    _prompts(2, 1, [128] * 150 + [40] * 460 + [100] * 150 + [7] * 150)


# More tiles than SMs: prompts of one length, in pairs and alone in several rounds; an odd last tile; sequences that differ, sorted by
# their time; more items than are sorted, and more sequences, which go as they come.
@pytest.mark.parametrize("hq,hkv,lens", [(16, 8, [256] * 8), (16, 8, [1500]), (16, 8, [1500, 1500]), (8, 8, [600] * 7), (8, 8, [129, 700, 3, 250] * 5),
                                         (2, 2, list(range(130, 430))), (1, 1, [5, 300] + [1, 17] * 520)])
def test_prompt_attention_dealt_out(hq, hkv, lens):
    _prompts(hq, hkv, lens)


# Portions behind cached tokens, the queries being the last rows of each sequence: pairs, tiles alone beside them, rows of one token
# with many keys beside a prompt, in one round and in several.  P and the output are bf16: 2^-9 relative each.
@pytest.mark.parametrize("hq,hkv", [(16, 8), (8, 8)])
@pytest.mark.parametrize("portions,cached", [([512] * 3, [700, 0, 1500]), ([300, 1, 65, 700, 130, 1] * 3, [0, 2000, 511, 100, 900, 3] * 3), ([600], [1333]),
                                             ([256] + [1] * 40, [0] + [1000] * 40)])
def test_causal_attention_behind_cached_tokens(hq, hkv, portions, cached):
    ends, cu_q, cu_k, g = [a + b for a, b in zip(portions, cached)], [0], [0], gen(len(portions))
    for n, t in zip(portions, ends):
        cu_q.append(cu_q[-1] + n)
        cu_k.append(cu_k[-1] + t)
    q, k, v = (torch.randn(m, h, 128, generator=g, device=DEV).to(BF) for m, h in ((cu_q[-1], hq), (cu_k[-1], hkv), (cu_k[-1], hkv)))
    out = torch.zeros_like(q)
    ops.causal_attn_varlen(q, k, v, i32(cu_q), i32(cu_k), len(portions), max(portions), 0.1, out)
    assert pkg._lib.device_status() == 0
    for i, (n, t) in enumerate(zip(portions, ends)):
        kk, vv = (x[cu_k[i]:cu_k[i + 1]].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
        s = torch.einsum("ihd,jhd->hij", q[cu_q[i]:cu_q[i + 1]].double(), kk) * 0.1
        seen = torch.arange(t, device=DEV)[None] <= torch.arange(t - n, t, device=DEV)[:, None]
        ref = torch.einsum("hij,jhd->ihd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), vv)
        assert rel(out[cu_q[i]:cu_q[i + 1]], ref) < 8e-3, i


def _prompts(hq, hkv, lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    m, g = cu[-1], gen(hq + len(lens))
    q, k, v = (torch.randn(m, h, 128, generator=g, device=DEV).to(BF) for h in (hq, hkv, hkv))
    out = torch.zeros_like(q)
    ops.sparse_attn_varlen(q, k, v, i32(cu), i32(cu), 32, max_seqlen=max(lens), out=out)
    assert pkg._lib.device_status() == 0
    for a, b in zip(cu, cu[1:]):
        t = b - a
        i = torch.arange(t, device=DEV)
        pad = -t % 32
        seen = i[None] < torch.clamp(((i + pad) // 32 + 1) * 32 - pad, max=t)[:, None]
        kk, vv = (x[a:b].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
        s = torch.einsum("ihd,jhd->hij", q[a:b].double(), kk) * 128 ** -0.5
        ref = torch.einsum("hij,jhd->ihd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), vv)
        assert rel(out[a:b], ref) < 8e-3, (a, b)


# Rows that end inside, on and behind a tile of 64 keys and a page, a padding row, one and two groups of heads, whole rows and
# parts; whatever lies in the cache behind a context must not matter.  bf16 output: 2^-9.
@pytest.mark.parametrize("width,heads", [(128, 3), (256, 16), (384, 20), (512, 16), (512, 33)])
@pytest.mark.parametrize("nsplit", [1, 2, 5])
def test_latent_attention_shares(width, heads, nsplit):
    ctx = [1, 64, 65, 0, 256, 257, 1000, 700, 3, 511]
    need = [(n + 255) // 256 for n in ctx]
    perm, g = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).tolist(), gen(width + heads)
    table = torch.full((len(ctx), max(need)), -1, dtype=torch.int32)
    cache = torch.full((sum(need) * 256, width), float("nan"), dtype=BF, device=DEV)
    at = 0
    for i, n in enumerate(ctx):
        for p in range(need[i]):
            page = perm[at]
            at += 1
            table[i, p] = page
            rows = min(256, n - 256 * p)
            cache[page * 256:page * 256 + rows] = torch.randn(rows, width, generator=g, device=DEV).to(BF)
    m = len(ctx)
    q = torch.randn(m, heads * width, generator=g, device=DEV).to(BF)
    out = torch.full((m, heads * width), 7.0, dtype=BF, device=DEV)
    ws = torch.full((max(16, ops.latent_attn_workspace_bytes(m, heads, width, nsplit)),), 255, dtype=torch.uint8, device=DEV)
    ops.latent_attn(q, cache, table.to(DEV), i32(list(range(m))), i32([n - 1 for n in ctx]), heads, 0.11, out, nsplit, ws)
    assert pkg._lib.device_status() == 0
    for i, n in enumerate(ctx):
        if n == 0:
            assert float((out[i].float() - 7).abs().max()) == 0
            continue
        c = cache.view(-1, 256, width)[table[i, :need[i]].long().to(DEV)].flatten(0, 1)[:n].double()
        p = torch.softmax(q[i].view(heads, width).double() @ c.T * 0.11, -1)
        assert rel(out[i].view(heads, width), p @ c) < 4e-3, i


# Around the rule for pairs (160 rows per expert; option 2 takes them from there on, whatever they gain), experts of one, two, three and
# no tiles, output columns that do not fill the last tile, and more ids than the plan has in flight.
@pytest.mark.parametrize("pairs", [1, 2])
@pytest.mark.parametrize("E,top,m,kind", [(4, 2, 300, "spread"), (4, 2, 400, "spread"), (8, 3, 900, "skewed"), (5, 1, 900, "one"), (64, 6, 2600, "spread")])
@pytest.mark.parametrize("n", [264, 512])
def test_expert_tiles_in_pairs(E, top, m, kind, n, pairs):
    k, g = 128, gen(E + m)
    ids = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(i))[:top] for i in range(m)])
    if kind == "one":
        ids[:] = 3
    elif kind == "skewed":
        ids[: m - 7] = torch.tensor([1, 5, 6])
    tiles = ops.moe_max_tiles(m, top, E)
    slot, row_token = torch.full((m, top), -9, dtype=torch.int32, device=DEV), torch.full((tiles * 128,), -9, dtype=torch.int32, device=DEV)
    tile_expert, num = torch.full((tiles,), -9, dtype=torch.int32, device=DEV), torch.full((1,), 1, dtype=torch.int32, device=DEV)
    x, w = torch.randn(m, k, generator=g, device=DEV).to(BF), (torch.randn(E, n, k, generator=g, device=DEV) * k ** -0.5).to(BF)
    xs, y = torch.zeros(tiles * 128, k, dtype=BF, device=DEV), torch.full((tiles * 128 + 1, n), 9.0, dtype=BF, device=DEV)
    ops.moe_plan(ids.int().to(DEV), E, tiles, slot, row_token, tile_expert, num)
    ops.moe_gather(x, xs, row_token, num, tiles)
    ops.set_option(ops.OPT_GEMM_PAIR, pairs)
    try:
        ops.gemm_experts(xs, w, y[:-1], tile_expert, num, m)
    finally:
        ops.set_option(ops.OPT_GEMM_PAIR, 1)
    assert pkg._lib.device_status() == 0
    s = slot.cpu().long()
    assert len(set(s.flatten().tolist())) == m * top and (tile_expert.cpu()[s // 128] == ids).all()
    assert float((y[int(num) * 128:].float() - 9).abs().max()) == 0          # rows of no tile stay as they were
    got = y[s.to(DEV)]
    for e in range(E):
        rows, at = (ids == e).nonzero(as_tuple=True)
        if len(rows):
            ref = x[rows.to(DEV)].double() @ w[e].double().T
            assert rel(got[rows.to(DEV), at.to(DEV)], ref) < 4e-3, e


def _window_case(H, KH, D, portions, starts, window, sink, edit=None):
    """Outputs of ops.window_attn for portions behind cached tokens, pages in any order and rubbish behind every context, and of
    the same attention in 64 bits; ``edit(values, start)`` may change a sequence's values [tokens, KH, D]."""
    bs, g, dp = len(portions), gen(H + D + window), (D + 63) // 64 * 64
    ctx = [a + b for a, b in zip(portions, starts)]
    need = [(n + 255) // 256 for n in ctx]
    perm, at = torch.randperm(sum(need), generator=torch.Generator().manual_seed(3)).tolist(), 0
    table = torch.full((bs, max(need)), -1, dtype=torch.int32)
    kc, vc = (torch.full((sum(need) * 256, KH, dp), float("nan"), dtype=BF, device=DEV) for _ in range(2))
    scale, qs, refs = 1.5 * D ** -0.5, [], []
    for i, n in enumerate(ctx):
        table[i, :need[i]] = torch.tensor(perm[at:at + need[i]])
        at += need[i]
        q, k, v = (torch.randn(t, h, D, generator=g, device=DEV).to(BF) for t, h in ((portions[i], H), (n, KH), (n, KH)))
        if edit is not None:
            edit(v, starts[i])
        slots = (table[i, :need[i]].long()[:, None] * 256 + torch.arange(256)).flatten()[:n].to(DEV)
        for c, x in ((kc, k), (vc, v)):
            c[slots] = 0
            c[slots, :, :D] = x
        qs.append(torch.zeros(portions[i], H, dp, dtype=BF, device=DEV))
        qs[-1][..., :D] = q
        p, j = torch.arange(starts[i], n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
        seen = (j <= p) & (j > p - window) if window else j <= p
        kk, vv = (x.double().repeat_interleave(H // KH, 1) for x in (k, v))
        s = (torch.einsum("ihd,jhd->hij", q.double(), kk) * scale).masked_fill(~seen, float("-inf"))
        if sink:
            s = torch.cat([s, torch.zeros_like(s[..., :1])], -1)
        w = torch.softmax(s, -1)[..., :n]
        # a value that is not seen does not count, whatever it is
        ref = torch.einsum("hij,jhd->ihd", w, torch.nan_to_num(vv, posinf=0, neginf=0))
        for t in (~torch.isfinite(v)).any(-1).any(-1).nonzero().flatten().tolist():
            ref[seen[:, t]] = float("nan")
        refs.append(ref)
    cu = [0]
    for n in portions:
        cu.append(cu[-1] + n)
    rows = (i32([i for i, n in enumerate(portions) for _ in range(n)]), i32(cu), i32(starts), i32(list(range(bs))))
    out = torch.full((cu[-1], (H * D + 7) // 8 * 8), 7.0, dtype=BF, device=DEV)
    ops.window_attn(torch.cat(qs), kc, vc, table.to(DEV), rows, i32([p for s, n in zip(starts, portions) for p in range(s, s + n)]), max(portions), D,
                    window, sink, scale, out)
    assert pkg._lib.device_status() == 0
    return [out[a:b, :H * D].view(b - a, H, D) for a, b in zip(cu, cu[1:])], refs


# A value of a token behind a query tile reaches no row of that tile, whatever it is: not through a key tile that the two query tiles of
# a pair share either (weights of zero times infinity).  160 tiles of 64 rows: pairs; the tiles meet inside a key tile.
@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("start", [0, 37])
def test_window_pairs_keep_the_future_out(window, start):
    def poison(v, first):
        v[first + 64 + 5] = float("inf")

    got, ref = _window_case(8, 4, 128, [256] * 10, [start] * 10, window, True, poison)
    for o, r in zip(got, ref):
        assert rel(o[:64], r[:64]) < 8e-3
        hit = torch.isnan(r).flatten(1).any(1)
        assert not bool(torch.isfinite(o[hit]).all(-1).any())


# Pairs of window attention in several rounds: one and two channel halves, channels that do not fill them, ragged portions behind cached
# tokens, windows narrower than a tile, of a tile and one, and none; rubbish behind every context.
@pytest.mark.parametrize("H,KH,D", [(8, 4, 128), (8, 4, 64), (6, 6, 96), (12, 4, 40)])
@pytest.mark.parametrize("window", [0, 50, 129])
@pytest.mark.parametrize("portions,starts", [([300, 20, 700, 65, 128] * 4, [0, 1000, 37, 255, 600] * 4), ([256] * 12, [100] * 12)])
def test_window_pairs(H, KH, D, window, portions, starts):
    got, ref = _window_case(H, KH, D, portions, starts, window, True)
    for i, (o, r) in enumerate(zip(got, ref)):
        assert rel(o, r) < 8e-3, i


# Ids per thread of the plan: one, up to 4, 12 and 24 in registers, more in two walks; some pairs go nowhere.  Gathered rows of one piece, of
# a warp's eight rounds of pieces, and of one more.  Whole numbers and copies: exact.
@pytest.mark.parametrize("m,top,experts", [(1, 1, 3), (512, 2, 64), (513, 2, 40), (1024, 4, 64), (1366, 3, 7), (2048, 6, 64), (2049, 6, 64), (4096, 6, 160),
                                           (4097, 6, 64)])
def test_expert_plan_and_gather(m, top, experts):
    ids = torch.rand(m, experts, generator=gen(m), device=DEV).topk(top, dim=1).indices.int()
    ids[::97] = -1
    tiles = ops.moe_max_tiles(m, top, experts)
    slot, row_token = torch.full((m, top), -9, dtype=torch.int32, device=DEV), torch.full((tiles * 128,), -9, dtype=torch.int32, device=DEV)
    tile_expert, num = torch.full((tiles,), -9, dtype=torch.int32, device=DEV), i32([0] * 4)
    ops.moe_plan(ids, experts, tiles, slot, row_token, tile_expert, num)
    counts = torch.bincount(ids[ids >= 0].long(), minlength=experts)
    per = ((counts + 127) // 128).tolist()
    used = sum(per)
    assert int(num[0]) == used <= tiles and tile_expert[:used].tolist() == [e for e, n in enumerate(per) for _ in range(n)]
    assert bool((slot[ids < 0] == -1).all()) and bool((slot[ids >= 0] >= 0).all())
    flat, pairs = slot[ids >= 0].long(), (ids >= 0).nonzero()
    assert len(flat.unique()) == len(flat)                                           # a row of its own for every pair
    assert torch.equal(tile_expert[flat // 128], ids[ids >= 0]) and torch.equal(row_token[flat].long(), pairs[:, 0])
    empty = torch.ones(used * 128, dtype=torch.bool, device=DEV)
    empty[flat] = False
    assert bool((row_token[:used * 128][empty] == -1).all())
    for width in (8, 2048, 2056):
        x = torch.randn(m, width + 8, generator=gen(1), device=DEV).to(BF)[:, :width]
        xs = torch.full((tiles * 128, width), 3.0, dtype=BF, device=DEV)
        ops.moe_gather(x, xs, row_token, num, tiles)
        assert torch.equal(xs[flat], x[pairs[:, 0]]) and bool((xs[:used * 128][empty] == 3).all())


# Several keys at a time (four, two, one by width): contexts that end inside a round of the four warps.  fp32 sums of up to 70 weights.
@pytest.mark.parametrize("width", [256, 384, 1024])
def test_fp32_latent_rows(width):
    pos = [0, 1, 3, 4, 5, 11, 15, 16, 17, 31, 32, 63, 69]
    q, cache = torch.randn(len(pos), 2, width, generator=gen(1), device=DEV) * 3, torch.randn(256, width, generator=gen(2), device=DEV)
    out, ws = torch.zeros(len(pos), 2 * width, device=DEV), torch.empty(16, dtype=torch.uint8, device=DEV)
    ops.latent_attn(q.view(len(pos), -1), cache, i32([[0]]), i32([0] * len(pos)), i32(pos), 2, width ** -0.5, out, 1, ws)
    for i, p in enumerate(pos):
        a = torch.softmax(q[i].double() @ cache[:p + 1].double().T * width ** -0.5, -1)
        assert rel(out[i].view(2, width), a @ cache[:p + 1].double()) < 2e-6, p


# One, two and four heads per reading of a key (by the number of rows and heads; three leave a group short): a row's bits are the same in
# each, its error that of fp32 sums.  The row alone takes one head at a time.
@pytest.mark.parametrize("m,heads,width", [(460, 4, 256), (460, 5, 96), (460, 6, 512), (160, 3, 256), (150, 3, 200)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_latent_rows_of_several_heads(m, heads, width, dtype):
    if dtype == BF and width in (256, 512):
        pytest.skip("a width of the tensor-core form")
    q = (torch.randn(m, heads * width, generator=gen(1), device=DEV) * 3).to(dtype)
    cache = torch.randn(512, width, generator=gen(2), device=DEV).to(dtype)
    pos, table = i32([-1 if r == 7 else r for r in range(m)]), i32([[1, 0]])
    out, ws = torch.full((m, heads * width), 5.0, dtype=dtype, device=DEV), torch.empty(16, dtype=torch.uint8, device=DEV)
    ops.latent_attn(q, cache, table, i32([0] * m), pos, heads, width ** -0.5, out, 1, ws)
    rows = torch.cat([cache[256:], cache[:256]]).double()
    for r in (0, 1, 17, 255, m - 1):
        r, one = min(r, m - 1), torch.zeros(1, heads * width, dtype=dtype, device=DEV)
        ops.latent_attn(q[r:r + 1], cache, table, i32([0]), pos[r:r + 1].contiguous(), heads, width ** -0.5, one, 1, ws)
        assert torch.equal(one[0], out[r]), r
        a = torch.softmax(q[r].view(heads, width).double() @ rows[:r + 1].T * width ** -0.5, -1)
        assert rel(out[r].view(heads, width), a @ rows[:r + 1]) < (2e-6 if dtype == torch.float32 else 4e-3), r
    assert bool((out[7] == 5).all())


# More experts than there are half warps, with one id per thread, up to four, and more: the same plan and gather.
@pytest.mark.parametrize("m,top,experts", [(1, 8, 65), (100, 8, 160), (300, 8, 256), (700, 8, 256), (520, 4, 1030), (683, 6, 64), (684, 6, 64)])
def test_expert_plan_of_many_experts(m, top, experts):
    test_expert_plan_and_gather(m, top, experts)
