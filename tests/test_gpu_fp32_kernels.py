"""The fp32 products and the scans in blocks of 16 tokens at the edges of their tiles, blocks and dispatch rules."""
import importlib

import pytest
import torch

from oracle import hybrid_oracle as orc

pkg = importlib.import_module("mineru-diffusion_b200")
ops = pkg.ops
pytestmark = pytest.mark.gpu
DEV, F32, F64 = "cuda", torch.float32, torch.float64


def gen(seed):
    return torch.Generator().manual_seed(seed)


def rel(got, ref):
    got, ref = got.double().cpu(), ref.double().cpu()
    return float((got - ref).norm() / ref.norm().clamp_min(1e-30))


# tiles of 16 x 32, 64 x 64 and 128 x 128, with rows, columns and k that fill none of them.  An fp32 sum of k products is off by
# at most k * 2^-24 and, with errors of either sign, by about sqrt(k) * 2^-24 = 2.7e-6 at k = 2000.
@pytest.mark.parametrize("m,n,k", [(1, 4, 16), (15, 36, 48), (17, 132, 144), (63, 1028, 272), (65, 1000, 528), (129, 4100, 80), (500, 1024, 2000),
                                   (1030, 2300, 112), (2050, 2052, 176)])
@pytest.mark.parametrize("act", [ops.ACT_NONE, ops.ACT_RELU2, ops.ACT_RELU_GLU, ops.ACT_SILU])
def test_fp32_product_tiles(m, n, k, act):
    x, w = torch.randn(m, k + 8, generator=gen(1)), torch.randn(2 * n if act == ops.ACT_RELU_GLU else n, k, generator=gen(2)) * k ** -0.5
    y = torch.full((m + 1, n + 4), 7.0, device=DEV)
    ops.gemm(x.to(DEV)[:, :k], w.to(DEV), y[:m, :n], act=act, act_from=4 if act == ops.ACT_SILU else 0)
    z = x[:, :k].to(DEV, F64) @ w.to(DEV, F64).T
    if act == ops.ACT_RELU2:
        z = torch.relu(z) ** 2
    elif act == ops.ACT_RELU_GLU:
        z = torch.relu(z[:, :n]) * z[:, n:]
    elif act == ops.ACT_SILU:
        z[:, 4:] = torch.nn.functional.silu(z[:, 4:])
    assert rel(y[:m, :n], z) < 3e-6
    assert float((y[:m, n:] - 7).abs().max()) == 0 and float((y[m] - 7).abs().max()) == 0
    assert pkg._lib.device_status() == 0


# The tile goes by the number of rows, the order of a row's sums does not: the same bits alone and beside any other rows.
@pytest.mark.parametrize("n,k", [(36, 16), (3072, 112), (1024, 176), (1024, 1024), (260, 2000)])
@pytest.mark.parametrize("act", [ops.ACT_NONE, ops.ACT_RELU_GLU])
def test_fp32_product_of_a_row_does_not_depend_on_the_others(n, k, act):
    x, w = torch.randn(4100, k, generator=gen(3)).to(DEV), torch.randn(2 * n if act == ops.ACT_RELU_GLU else n, k, generator=gen(4)).to(DEV)
    whole = ops.gemm(x, w, torch.zeros(4100, n, device=DEV), act=act)
    for m in (1, 16, 33, 64, 100, 500, 1000, 2050):
        assert torch.equal(ops.gemm(x[:m], w, torch.zeros(m, n, device=DEV), act=act), whole[:m]), m


def _portions(counts, starts, slots):
    cu = torch.tensor([0] + list(counts)).cumsum(0)
    row_seq = torch.cat([torch.full((n,), i) for i, n in enumerate(counts)])
    return tuple(torch.as_tensor(x).to(torch.int32).to(DEV) for x in (row_seq, cu, starts, slots))


def mlstm_parts(q, k, v, li, lf):
    S, n, m = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64), torch.zeros(q.shape[1:], dtype=F64), torch.zeros(q.shape[1], dtype=F64)
    num, den = [], []
    for t in range(len(q)):
        new = torch.maximum(lf[t] + m, li[t])
        a, b, m = torch.exp(lf[t] + m - new), torch.exp(li[t] - new), new
        S = a[:, None, None] * S + b[:, None, None] * k[t][:, :, None] * v[t][:, None]
        n = a[:, None] * n + b[:, None] * k[t]
        num.append(torch.einsum("hdv,hd->hv", S, q[t]))
        den.append(torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)
    return torch.stack(num), torch.stack(den)


# token counts around a block, two portions one behind the other, a padding entry; columns that fill 16, 32 and 64 wide CTAs or
# do not; one and several heads per key head; enough heads for the wide CTAs.  2e-6: thrice what the token by token form shows.
# Portions this short go token by token; a padding entry of 2000 rows lifts the average to where blocks are taken (not with the 80 and
# 160 sequence heads of two cases, whose CTAs would not run all at once; the last cases are as wide as fits).
@pytest.mark.parametrize("padding", [20, 2000])
@pytest.mark.parametrize("mode", [ops.SCAN_DELTA, ops.SCAN_MLSTM, ops.SCAN_DECAY])
@pytest.mark.parametrize("H,KH,D,DV,bs", [(2, 1, 64, 24, 3), (3, 3, 128, 33, 3), (8, 4, 128, 80, 3), (20, 20, 128, 128, 3), (40, 40, 64, 70, 3),
                                          (8, 8, 64, 80, 3), (16, 16, 128, 128, 3), (18, 18, 64, 100, 3)])
def test_scan_in_blocks(mode, H, KH, D, DV, bs, padding):
    if mode == ops.SCAN_MLSTM:
        KH = H
    first, second, slots = [47, 16, 1], [17, 33, 31], [2, 0, 3]
    rep, cols, nb = H // KH, DV + (mode == ops.SCAN_MLSTM), ops.scan_blocks(DV)
    state = torch.full((5, H, cols, D), 5.0, device=DEV)            # a slot is never cleared
    mst = torch.full((5, H, nb), 5.0, device=DEV)
    total = [a + b for a, b in zip(first, second)]
    g = gen(H + D)
    k = torch.nn.functional.normalize(torch.randn(sum(total), KH, D, generator=g), dim=-1)
    q = torch.randn(sum(total), KH, D, generator=g) * D ** -0.5
    v = torch.randn(sum(total), H, DV, generator=g)
    decay = torch.exp(-torch.exp(torch.randn(sum(total), H, D, generator=g) - 1))
    decay[::7, :, ::5] = 0.0                                        # a decay may forget everything
    beta = torch.rand(sum(total), H, generator=g)
    li, lf = torch.randn(sum(total), H, generator=g) * 4, torch.nn.functional.logsigmoid(torch.randn(sum(total), H, generator=g) * 3 + 1)
    skip = torch.randn(H, generator=g)
    base = [0] + torch.tensor(total).cumsum(0).tolist()
    got_o, got_d = torch.zeros(sum(total), H, DV), torch.ones(sum(total), H)
    for part, counts in enumerate((first, second)):
        rows = torch.cat([torch.arange(base[i] + (first[i] if part else 0), base[i] + (first[i] if part else 0) + n) for i, n in enumerate(counts)])
        pad = torch.cat([rows, rows[torch.arange(padding) % len(rows)]])      # the padding entry: nothing is read or written for it
        m = len(pad)
        p = _portions(counts + [padding], [first[i] if part else 0 for i in range(3)] + [0], slots + [-1])
        at = lambda t: t[pad].contiguous().to(DEV)                   # noqa: E731,B023
        o, den = torch.full((m, H, DV), 9.0, device=DEV), torch.full((m, H), 9.0, device=DEV)
        if mode == ops.SCAN_DELTA:
            kk, qq = (t[pad].double().repeat_interleave(rep, 1) for t in (k, q))
            before = decay[pad].double() * kk.roll(1, 0)             # (read for the second token of a pair only)
            sc = torch.stack([(kk * qq).sum(-1), (before * kk).sum(-1), (before * qq).sum(-1), beta[pad].double()], -1).float().to(DEV)
            ops.scan(mode, F32, 4, H, KH, D, DV, at(q), at(k), at(v), None, None, state, p, g=at(decay), scalars=sc, out=o)
        elif mode == ops.SCAN_MLSTM:
            ops.scan(mode, F32, 4, H, KH, D, DV, at(q), at(k), at(v), at(li), at(lf), state, p, mstate=mst, out=o, den=den)
        else:
            ops.scan(mode, F32, 4, H, KH, D, DV, at(q), at(k), at(v), at(decay[..., 1]), at(beta), state, p, out=o, skip=skip.to(DEV))
        assert float((o[-padding:] - 9).abs().max()) == 0
        got_o[rows], got_d[rows] = o[:-padding].cpu(), den[:-padding].cpu()
    assert pkg._lib.device_status() == 0
    assert float((state[[1, 4]] - 5).abs().max()) == 0
    for i in range(3):
        r = slice(base[i], base[i + 1])
        qq, kk, vv = (t[r].double().repeat_interleave(rep, 1) if t is not v else t[r].double() for t in (q, k, v))
        if mode == ops.SCAN_DELTA:
            ref = orc.delta_scan(qq, kk, vv, decay[r].double(), beta[r].double())
            assert rel(got_o[r], ref) < 2e-6, i
        elif mode == ops.SCAN_MLSTM:
            # numerator and denominator by themselves: their quotient is as ill-conditioned as |n . q| is small
            num, den = mlstm_parts(qq, kk, vv, li[r].double(), lf[r].double())
            assert rel(got_o[r], num) < 2e-6 and rel(got_d[r], den) < 2e-6, i
        else:
            S, ref = torch.zeros(H, DV, D, dtype=F64), []
            for t in range(len(qq)):
                S = decay[r][t, :, 1].double()[:, None, None] * S + beta[r][t].double()[:, None, None] * vv[t][:, :, None] * kk[t][:, None]
                ref.append(torch.einsum("hvd,hd->hv", S, qq[t]) + skip.double()[:, None] * vv[t])
            assert rel(got_o[r], torch.stack(ref)) < 2e-6, i
            assert rel(state[slots[i]], S) < 2e-6, i


def test_scan_in_blocks_keeps_the_future_out():
    """Values behind a token, whatever they are, do not reach its output."""
    H, D, DV, T, rows = 2, 128, 40, 32, 600      # rows behind the portion: as many as make blocks worth while
    q, k, v = (torch.randn(rows, H, n, generator=gen(i), device="cpu") for i, n in enumerate((D, D, DV)))
    v[21] = float("inf")
    o = torch.zeros(rows, H, DV, device=DEV)
    ops.scan(ops.SCAN_DECAY, F32, 1, H, H, D, DV, q.to(DEV), k.to(DEV), v.to(DEV), torch.full((rows, H), 0.9, device=DEV), torch.ones(rows, H, device=DEV),
             torch.zeros(1, H, DV, D, device=DEV), _portions([T], [0], [0]), out=o)
    assert bool(torch.isfinite(o[:21]).all()) and not bool(torch.isfinite(o[21:T]).any()) and float(o[T:].abs().max()) == 0


# From k = 768 on the products run on the tensor cores: tiles of 128, 64 or 32 weight rows (half of them up rows with GLU) x 32 or 64 rows, chunks
# of 64 k, one to four CTAs for a tile's k.  Sums of 64 products are cut off four times (2^-23 of a sum that is 1/16 of the whole in its
# square and less) and added up in fp32: 1e-7 by measurement; 4e-7 leaves room for the activation, which doubles it.  (Norms of dense
# rows; outputs one by one, rows of few numbers and sums of one sign: test_fp32_product_output_by_output.)
@pytest.mark.parametrize("m,n,k", [(1, 4, 768), (31, 132, 784), (33, 1000, 1040), (64, 260, 1552), (65, 4100, 768), (500, 1028, 3072), (1030, 2300, 816)])
@pytest.mark.parametrize("act", [ops.ACT_NONE, ops.ACT_RELU2, ops.ACT_RELU_GLU, ops.ACT_SILU])
def test_fp32_product_on_tensor_cores(m, n, k, act):
    x, w = torch.randn(m, k + 4 if m % 2 else k, generator=gen(1)), torch.randn(2 * n if act == ops.ACT_RELU_GLU else n, k, generator=gen(2)) * k ** -0.5
    y = torch.full((m + 1, n + 4), 7.0, device=DEV)
    wide = torch.zeros(m, k + 8, device=DEV)
    wide[:, 4 * (m % 2):4 * (m % 2) + k] = x[:, :k].to(DEV)                  # odd m: rows on a boundary of 16 bytes only
    rows = wide[:, 4 * (m % 2):4 * (m % 2) + k]
    ops.gemm(rows, w.to(DEV), y[:m, :n], act=act, act_from=4 if act == ops.ACT_SILU else 0)
    z = x[:, :k].to(DEV, F64) @ w.to(DEV, F64).T
    if act == ops.ACT_RELU2:
        z = torch.relu(z) ** 2
    elif act == ops.ACT_RELU_GLU:
        z = torch.relu(z[:, :n]) * z[:, n:]
    elif act == ops.ACT_SILU:
        z[:, 4:] = torch.nn.functional.silu(z[:, 4:])
    assert rel(y[:m, :n], z) < 4e-7
    assert float((y[:m, n:] - 7).abs().max()) == 0 and float((y[m] - 7).abs().max()) == 0
    assert pkg._lib.device_status() == 0


def test_fp32_product_per_head_and_per_expert_on_tensor_cores():
    heads, n, k, m = 3, 200, 1024, 70
    x, w = torch.randn(m, heads * k, generator=gen(5)).to(DEV), torch.randn(heads, n, k, generator=gen(6)).to(DEV)
    y = ops.gemm_heads(x, w, torch.zeros(m, heads * n, device=DEV))
    ref = torch.einsum("mhk,hnk->mhn", x.double().view(m, heads, k), w.double()).reshape(m, -1)
    assert rel(y, ref) < 4e-7
    tiles = torch.tensor([2, 0, 2], dtype=torch.int32, device=DEV)
    x = torch.randn(4 * 128, k, generator=gen(7)).to(DEV)
    y = torch.full((4 * 128, n), 7.0, device=DEV)
    ops.gemm_experts(x, w, y, tiles, torch.tensor([3, 0, 0, 0], dtype=torch.int32, device=DEV), 128)
    for i, e in enumerate(tiles.tolist()):
        assert rel(y[128 * i:128 * i + 128], x[128 * i:128 * i + 128].double() @ w[e].double().T) < 4e-7
    assert float((y[384:] - 7).abs().max()) == 0 and pkg._lib.device_status() == 0


@pytest.mark.parametrize("m", [5, 400])
def test_fp32_product_of_numbers_that_are_not_finite(m):
    """Infinities and NaN reach the outputs that an fp32 sum gives them, and no others; numbers near the largest stay finite."""
    n, k = 300, 1024
    x, w = torch.randn(m, k, generator=gen(8)), torch.randn(n, k, generator=gen(9))
    x[1, 5], x[2, 7], x[3, 8] = float("inf"), float("nan"), 3e38
    w[4, 5], w[11, 0], w[12, 8], w[13] = 0.0, -float("inf"), 0.5, 0.0
    y = ops.gemm(x.to(DEV), w.to(DEV), torch.zeros(m, n, device=DEV)).cpu()
    ref = x.double() @ w.double().T                                     # inf * 0 is NaN there too
    kind = lambda t: torch.where(t.isnan(), 3.0, torch.where(t.isinf(), t.sign(), 2.0 * torch.ones_like(t)))      # noqa: E731
    big = ref.abs() > 3.4e38
    ref[big & ref.isfinite()] = ref[big & ref.isfinite()].sign() * float("inf")
    assert torch.equal(kind(y.double()), kind(ref))
    assert rel(y[4][ref[4].isfinite()], ref[4][ref[4].isfinite()]) < 4e-7
    assert pkg._lib.device_status() == 0


# Outputs one by one, in 2^-24 of the sum of the sizes of their products (against fp64).  Up to 16 products that are not zero: their roundings
# to 24 bits, half a unit's root mean square and less, however the operands are taken apart; a single one: one rounding, and 2^-6 for
# the sums of small parts.  Sums of one sign, where a sum cut off (at 2 units of itself, after each 16 of 64 products) falls short by up to
# (1 + 2 + 3 + 4) / 4 units of itself on average.
@pytest.mark.parametrize("k", [1024, 3072])
@pytest.mark.parametrize("kind,rms,largest", [("1", 0.5, 1.1), ("4", 0.5, 4.0), ("16", 0.5, 4.0), ("sizes", 2.5, 16.0), ("full", 2.5, 16.0), ("same", 2.5, 16.0)])
@pytest.mark.parametrize("form", ["plain", "glu", "experts"])
def test_fp32_product_output_by_output(k, kind, rms, largest, form):
    m, n = (128, 200) if form == "experts" else (65, 512)
    x, w = torch.randn(m, k, generator=gen(10)), torch.randn(n, k, generator=gen(11))
    if kind.isdigit():      # rows of few numbers that are not zero
        x *= torch.zeros(m, k).scatter_(1, torch.rand(m, k, generator=gen(12)).topk(int(kind), 1).indices, 1.0)
    elif kind == "sizes":
        x, w = x.abs(), w.abs()
    elif kind == "full":    # of one sign, the last 16 bits of the significand set
        x, w = (((t.abs() + 1).view(torch.int32) | 0xffff).view(torch.float32) for t in (x, w))
    else:
        x, w = (torch.full_like(t, 1 + 65535 / 2 ** 23) for t in (x, w))
    x, w = x.to(DEV), w.to(DEV)
    if form == "experts":
        y = ops.gemm_experts(x, torch.stack([w * 0, w]), torch.zeros(m, n, device=DEV), torch.ones(1, dtype=torch.int32, device=DEV),
                             torch.ones(4, dtype=torch.int32, device=DEV), 128)
    else:
        y = ops.gemm(x, w, torch.zeros(m, n // 2 if form == "glu" else n, device=DEV), act=ops.ACT_RELU_GLU if form == "glu" else ops.ACT_NONE)
    z, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    if form == "glu":       # an error of each factor reaches the result times the other
        g, up = torch.relu(z[:, :n // 2]), z[:, n // 2:]
        z, size = g * up, size[:, :n // 2] * up.abs() * (g > 0) + size[:, n // 2:] * g
        rms, largest = rms + 0.5, largest + 1      # and their product is rounded
    some = size > 0
    e = (y.double() - z)[some] / size[some] * 2 ** 24
    assert float(e.square().mean().sqrt()) < rms and float(e.abs().max()) < largest
    assert float(y[~some].abs().max() if bool((~some).any()) else 0) == 0 and pkg._lib.device_status() == 0


def test_fp32_product_beside_rows_that_are_not_finite():
    """Rows nobody reads (the empty rows of an expert's tile hold whatever they held) change neither the other rows nor the time; a NaN
    is one whatever its bits are."""
    n, k, tiles = 1024, 1024, 24
    x, w = torch.randn(tiles * 128, k, generator=gen(13)).to(DEV), torch.randn(1, n, k, generator=gen(14)).to(DEV)
    plan = torch.zeros(tiles, dtype=torch.int32, device=DEV), torch.full((4,), tiles, dtype=torch.int32, device=DEV)
    rows = torch.arange(tiles * 128, device=DEV) % 128 < 5
    odd = x.clone()
    odd.view(torch.int32)[~rows] = -1                # NaN
    odd.view(torch.int32)[5::128] = 0x7f800001       # NaN whose upper half is that of an infinity
    odd[6::128] = float("inf")
    y = [torch.zeros(tiles * 128, n, device=DEV) for _ in range(2)]
    took = []
    for a, b in ((x, y[0]), (odd, y[1])):
        ops.gemm_experts(a, w, b, *plan, 128)
        start, end = torch.cuda.Event(True), torch.cuda.Event(True)
        start.record()
        for _ in range(5):
            ops.gemm_experts(a, w, b, *plan, 128)
        end.record()
        torch.cuda.synchronize()
        took.append(start.elapsed_time(end))
    assert torch.equal(y[0][rows], y[1][rows]) and not bool(torch.isfinite(y[1][~rows]).any())
    assert bool(y[1][5::128].isnan().all())
    assert took[1] < 2 * took[0], took               # (hundreds of times as long where a thread forms such a sum again)
    assert pkg._lib.device_status() == 0


# Every number down to 2^-122 is taken apart exactly: scaled by a power of two the result has the same error.  Down to the smallest normal number
# up to four of 24 bits may go, 2^-19 of a number and, with errors of either sign, far less of a sum.  Products far below 1 end at 2^-149.
@pytest.mark.parametrize("x_exp,w_exp,limit", [(-108, 0, 2e-7), (-114, 0, 2e-7), (-120, 20, 2e-7), (0, -118, 2e-7), (-124, 60, 1e-6), (-60, -60, 2e-7), (90, 20, 2e-7)])
def test_fp32_product_of_small_and_large_numbers(x_exp, w_exp, limit):
    m, n, k = 40, 300, 1024
    x, w = torch.rand(m, k, generator=gen(15)) + 1, torch.rand(n, k, generator=gen(16)) + 1       # sizes in [1, 2), of either sign
    x, w = x * torch.randn(m, k, generator=gen(17)).sign() * 2.0 ** x_exp, w * torch.randn(n, k, generator=gen(18)).sign() * 2.0 ** w_exp
    y = ops.gemm(x.to(DEV), w.to(DEV), torch.zeros(m, n, device=DEV))
    assert rel(y.double() * 2.0 ** -(x_exp + w_exp), x.double() @ w.double().T * 2.0 ** -(x_exp + w_exp)) < limit
    assert pkg._lib.device_status() == 0


# Few rows take tiles of 128, 64 or 32 weight rows (half of them up rows with GLU) in clusters of one, two or four, by the number of columns: the same
# bits as beside 600 rows, and the last tile and the last chunk of k may be partly empty.
@pytest.mark.parametrize("form,n,k", [("plain", 20, 768), ("glu", 20, 768), ("plain", 1028, 1024), ("plain", 2052, 1024), ("glu", 1028, 1040), ("plain", 4352, 1024),
                                      ("heads", 72, 1040), ("plain", 8200, 832), ("glu", 8, 3088)])
def test_fp32_product_of_few_rows(form, n, k):
    heads = 3 if form == "heads" else 1
    x, w = torch.randn(600, heads * k, generator=gen(19)).to(DEV), torch.randn(heads, 2 * n if form == "glu" else n, k, generator=gen(20)).to(DEV)

    def product(rows):
        y = torch.full((len(rows) + 1, heads * n), 7.0, device=DEV)
        if form == "heads":
            ops.gemm_heads(rows, w, y[:-1])
        else:
            ops.gemm(rows, w[0], y[:-1], act=ops.ACT_RELU_GLU if form == "glu" else ops.ACT_NONE)
        assert float((y[-1] - 7).abs().max()) == 0
        return y[:-1]

    whole = product(x)
    z = torch.einsum("mhk,hnk->mhn", x.double().view(600, heads, k), w.double()).reshape(600, -1)
    if form == "glu":
        z = torch.relu(z[:, :n]) * z[:, n:]
    assert rel(whole, z) < 4e-7
    for m in (1, 9, 33, 64, 100):
        assert torch.equal(product(x[:m]), whole[:m]), m
    assert pkg._lib.device_status() == 0


# Either side of where blocks begin (64 tokens for the delta rule with 16 and 32 columns a CTA, 32 with 64 and for the decay scan), and portions of very
# unequal length, told and not told: the form may change, the recurrence does not.  2e-6: as above.
@pytest.mark.parametrize("mode,H,DV,counts", [(ops.SCAN_DELTA, 16, 128, [63, 63]), (ops.SCAN_DELTA, 16, 128, [64, 65]), (ops.SCAN_DELTA, 3, 40, [63]),
                                              (ops.SCAN_DELTA, 3, 40, [64, 66]), (ops.SCAN_DELTA, 64, 80, [31]), (ops.SCAN_DELTA, 64, 80, [33]),
                                              (ops.SCAN_DECAY, 16, 80, [31, 31]), (ops.SCAN_DECAY, 16, 80, [32, 34]),
                                              (ops.SCAN_DELTA, 8, 64, [1] * 15 + [500]), (ops.SCAN_DECAY, 16, 64, [1] * 7 + [260])])
def test_scan_where_blocks_begin(mode, H, DV, counts):
    D, g = 128, gen(21)
    m = sum(counts)
    k = torch.nn.functional.normalize(torch.randn(m, H, D, generator=g), dim=-1)
    q, v, beta = torch.randn(m, H, D, generator=g) * D ** -0.5, torch.randn(m, H, DV, generator=g), torch.rand(m, H, generator=g)
    decay = torch.exp(-torch.exp(torch.randn(m, H, D, generator=g) - 1))
    if mode == ops.SCAN_DECAY:
        decay = decay[..., :1].expand(m, H, D)
    before = decay.double() * k.double().roll(1, 0)
    sc = torch.stack([(k.double() * q.double()).sum(-1), (before * k.double()).sum(-1), (before * q.double()).sum(-1), beta.double()], -1).float().to(DEV)
    p, got = _portions(counts, [0] * len(counts), list(range(len(counts)))), []
    for longest in (0, max(counts)):
        o, state = torch.full((m, H, DV), 9.0, device=DEV), torch.full((len(counts), H, DV, D), 5.0, device=DEV)
        common = (mode, F32, len(counts), H, H, D, DV, q.to(DEV), k.to(DEV), v.to(DEV))
        if mode == ops.SCAN_DELTA:
            ops.scan(*common, None, None, state, p, g=decay.to(DEV), scalars=sc, out=o, max_q=longest)
        else:
            ops.scan(*common, decay[..., 0].contiguous().to(DEV), beta.to(DEV), state, p, out=o, max_q=longest)
        at = 0
        for n in counts:
            r = slice(at, at + n)
            at += n
            qq, kk, vv, dd, bb = (t[r].double() for t in (q, k, v, decay, beta))
            if mode == ops.SCAN_DELTA:
                ref = orc.delta_scan(qq, kk, vv, dd, bb)
            else:
                S, ref = torch.zeros(H, DV, D, dtype=F64), []
                for t in range(n):
                    S = dd[t, :, 0][:, None, None] * S + bb[t][:, None, None] * vv[t][:, :, None] * kk[t][:, None]
                    ref.append(torch.einsum("hvd,hd->hv", S, qq[t]))
                ref = torch.stack(ref)
            assert rel(o[r], ref) < 2e-6, (longest, n)
        got.append(o)
    assert torch.equal(*got) == (len(counts) < 16)     # the two forms round in their own order
    assert pkg._lib.device_status() == 0
