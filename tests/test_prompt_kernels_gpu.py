"""Edges of the kernels of prompts and decode rounds: even row tiles, paired EXL3 products, block masks, per-head products, EXL3 pairs."""
import pytest
import torch

from spark_engine_b200.quant import formats as Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _had(x):
    return (x.view(*x.shape[:-1], -1, 128) @ Q.hadamard128().double().to(x.device)).view(x.shape)


def _ids(sizes, seed):
    ids = torch.tensor([e for e, n in enumerate(sizes) for _ in range(n)], dtype=torch.int32, device=DEV)
    return ids, ids[torch.randperm(len(ids), device=DEV, generator=_gen(seed))].contiguous()


@pytest.mark.parametrize("rows", [64, 96, 192])
@pytest.mark.parametrize("sizes", [[1], [63, 64, 65, 0, 128, 129], [191, 192, 193, 384, 385, 0, 2500], [3] * 300])
def test_even_tiles_cover_every_row_once(sizes, rows):
    from spark_engine_b200.ops import cuda as cu
    ids, shuffled = _ids(sizes, 1)
    perm, inv, offs, tiles, ntile, max_tiles = cu.moe_sort(shuffled, len(sizes), rows)
    t = tiles[: ntile.item()].tolist()
    assert len(t) == sum(-(-n // rows) for n in sizes) <= max_tiles
    assert sorted(r for row, _, _, n in t for r in range(row, row + n)) == list(range(len(ids)))
    for row, end, e, n in t:
        assert 0 < n <= rows and offs[e] <= row and row + n <= end == offs[e + 1]
    assert torch.equal(shuffled[perm.long()], ids)


@pytest.mark.parametrize("rows", [96, 192])
@pytest.mark.parametrize("sizes,K,N", [([96, 97, 0, 16], 256, 256), ([191, 192, 193, 1], 128, 384), ([400, 20], 1024, 128)])
def test_exl3_tc_even_tiles(sizes, K, N, rows):
    from spark_engine_b200.ops import cuda as cu
    w = Q.random_exl3(N, K, 4, len(sizes), 0.05, 2, DEV)
    wd = Q.random_exl3(128, 128, 4, len(sizes), 0.05, 3, DEV)
    ids, shuffled = _ids(sizes, 1)
    x = torch.randn(len(ids), K, device=DEV, generator=_gen(5)).half()
    _, _, _, t128, n128, m128 = cu.moe_sort(shuffled, len(sizes))
    _, _, _, tiles, ntile, max_tiles = cu.moe_sort(shuffled, len(sizes), rows)
    y = cu.exl3_tc(x, w, tiles, ntile, max_tiles, out_f32=True, tile_rows=rows)
    assert torch.equal(y, cu.exl3_tc(x, w, t128, n128, m128, out_f32=True))          # a row's sum does not know its tile
    if N == 256:
        assert torch.equal(cu.exl3_tc(x, w, tiles, ntile, max_tiles, glu=wd, tile_rows=rows), cu.exl3_tc(x, w, t128, n128, m128, glu=wd))
    assert cu.read_status(torch.device(DEV))[0] == 0
    for e in ids.unique().tolist():
        r = ids == e
        ref = _had(x[r].double() @ Q.exl3_inner(w.trellis[e], w.kind).double()) * w.svh[e].double()
        assert ((y[r].double() - ref).norm() / ref.norm()).item() < (K + 128) * 2.0 ** -23


@pytest.mark.parametrize("K", [128, 192 * 2, 1024])
def test_exl3_tc_many_items_of_both_kinds_per_cta(K):
    """Items that take half of the accumulators and items that take all, in changing order, several per CTA."""
    from spark_engine_b200.ops import cuda as cu
    sizes = [(i * 73) % 230 for i in range(300)]
    w = Q.random_exl3(512, K, 4, len(sizes), 0.05, 2, DEV)
    _, shuffled = _ids(sizes, 1)
    x = torch.randn(len(shuffled), K, device=DEV, generator=_gen(5)).half()
    _, _, _, t128, n128, m128 = cu.moe_sort(shuffled, len(sizes))
    y = cu.exl3_tc(x, w, t128, n128, m128)
    assert torch.equal(cu.exl3_tc(x, w, t128, n128, m128, tile_rows=96), y)              # all items read out by the epilogue warps
    for rows in (96, 192):
        _, _, _, tiles, ntile, max_tiles = cu.moe_sort(shuffled, len(sizes), rows)
        assert torch.equal(cu.exl3_tc(x, w, tiles, ntile, max_tiles, tile_rows=rows), y)
    assert cu.read_status(torch.device(DEV))[0] == 0


@pytest.mark.parametrize("M,N,K", [(17, 128, 128), (256, 384, 256), (257, 1024, 2048), (1021, 2048, 512), (2500, 2176, 384)])
def test_paired_exl3_product(M, N, K):
    """Both tile widths, ragged rows, a last tile of half its columns."""
    from spark_engine_b200.ops import cuda as cu
    w = Q.random_exl3(N, K, 4, 0, 0.05, M, DEV)
    xh = torch.randn(M, K, device=DEV, generator=_gen(M)).half()
    wt = cu.exl3_reconstruct(w)
    y = cu.gemm_exl3(xh, wt, w.svh)
    assert torch.equal(y, cu.gemm_exl3(xh, wt, w.svh)) and cu.read_status(torch.device(DEV))[0] == 0
    ref = _had(xh.double() @ wt.double().t()) * w.svh.double()
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -9                 # bf16 rounding of the result
    assert torch.equal(y, cu.exl3_had_rows(cu.gemm_bf16(xh, wt, out_f32=True, fmt=0), w.svh, post=True))


@pytest.mark.parametrize("R,pos0,k", [(40, 100, 8), (64, 4000, 512), (300, 0, 16), (5, 17000, 512)])
def test_block_mask_is_the_token_list(R, pos0, k):
    from spark_engine_b200.ops import cuda as cu, sparse as sp
    pos = torch.arange(pos0, pos0 + R, dtype=torch.int32, device=DEV)
    ctx = pos0 + R
    nb, mw = max(1, ctx // 4), (ctx + 127) // 128
    score = torch.randint(0, 50, (R, nb), device=DEV, generator=_gen(R)).float()       # ties
    sel, sel_n = sp.topk_select(score, nb, pos, 4, k)
    mask = torch.full((R, mw), -1, dtype=torch.int32, device=DEV)
    cu.check(sp._dll().spark_topk_mask(cu.P(score), nb, cu.P(pos), R, k, cu.P(mask), mw, cu.stream(), 0), "spark_topk_mask")
    for r in range(R):
        want = torch.zeros(mw * 32, dtype=torch.bool, device=DEV)
        want[(sel[r, : sel_n[r]] // 4).long()] = True
        got = (mask[r].view(mw, 1) >> torch.arange(32, device=DEV, dtype=torch.int32) & 1).bool().view(-1)
        assert torch.equal(got, want), r


@pytest.mark.parametrize("H,Dm", [(1, 8), (3, 66), (4, 128), (5, 127)])
def test_decode_block_scores(H, Dm):
    from spark_engine_b200.ops import sparse as sp
    g = _gen(H)
    pos = torch.tensor([3, 200, 517], dtype=torch.int32, device=DEV)
    pool = torch.randn(3 * 130, Dm, device=DEV, generator=g)
    qi, hw = torch.randn(3, H, Dm, device=DEV, generator=g), torch.randn(3, H, device=DEV, generator=g)
    row_kv = torch.tensor([0, 520, 1040], dtype=torch.int64, device=DEV)
    for w in (None, hw):
        score, nb = sp.block_scores(qi, pool, row_kv, pos, 4, 518, head_w=w)
        for r in range(3):
            vis = (int(pos[r]) + 1) // 4
            d = (qi[r].double() @ pool[130 * r: 130 * r + vis].double().t()).relu() / Dm ** 0.5
            ref = (d if w is None else d * w[r].double().unsqueeze(1)).sum(0)
            assert torch.allclose(score.view(-1)[r * nb: r * nb + vis].double(), ref, rtol=0, atol=(Dm + H) * 2.0 ** -23 * H * 4 * Dm ** 0.5)


@pytest.mark.parametrize("rows,n,k", [(1, 5, 8), (3, 130, 128), (4, 512, 136), (8, 64, 512), (16, 33, 1024), (2, 16, 1032)])
def test_per_head_products(rows, n, k):
    from spark_engine_b200.ops import cuda as cu
    g, H = _gen(n), 6
    x = torch.randn(rows, H, k + 8, device=DEV, generator=g).bfloat16()
    w = torch.randn(H, n, k, device=DEV, generator=g).bfloat16()
    heads = torch.tensor([5, 0, -1, 2, 1, 4], dtype=torch.int32, device=DEV)
    for early in (False, True):
        y = torch.zeros(rows, H, n, dtype=torch.float32, device=DEV)
        cu.gemv_bf16_items(x, H * (k + 8), k + 8, w, n * k, k, y, H * n, n, H, rows, n, k, heads, pairs_early=early)
        for i, e in enumerate(heads.tolist()):
            ref = x[:, i, :k].double() @ w[e].double().t() if e >= 0 else torch.zeros(rows, n, device=DEV, dtype=torch.float64)
            assert torch.allclose(y[:, i].double(), ref, rtol=0, atol=k * 2.0 ** -24 * 8 * k ** 0.5), (i, early)


@pytest.mark.parametrize("K,N,act", [(512, 256, 1), (2048, 384, 0), (1536, 128, 1), (640, 256, 0)])
def test_exl3_pairs_do_not_depend_on_their_number(K, N, act):
    """Few pairs take more slices than many: the bits of a pair are the same."""
    from spark_engine_b200.ops import cuda as cu
    E, many = 12, 900
    w = Q.random_exl3(N, K, 4, E, 0.05, 4, DEV)
    x = torch.randn(many, 2 * K if act else K, device=DEV, generator=_gen(K)).bfloat16()
    e = torch.randint(0, E, (many,), device=DEV, generator=_gen(N), dtype=torch.int32)
    run = lambda n: cu.exl3_gemv(x[:n], w, items=n, rows_per_item=1, pair_expert=e[:n].contiguous(), act=act, out_f32=True)
    y = run(many)
    for n in (1, 2, 40, 200):
        assert torch.equal(run(n), y[:n]), n
    h = x[:40].double()
    if act:
        h = torch.nn.functional.silu(h[:, :K]) * h[:, K:]
    for i in range(40):
        j = e[i].item()
        xh = _had(h[i: i + 1] * w.suh[j].double()).half().double()
        ref = _had(xh @ Q.exl3_inner(w.trellis[j], w.kind).double()) * w.svh[j].double()
        assert ((y[i].double() - ref).norm() / ref.norm()).item() < 2.0 ** -10          # fp16 rounding of the transformed rows


def test_mxfp4_tiles_of_64_rows():
    from spark_engine_b200.ops import cuda as cu, mx
    E, N, K = 5, 256, 512
    ids, shuffled = _ids([64, 65, 0, 1, 200], 3)
    w = Q.random_mxfp4(N, K, E, 0.05, 3, DEV)
    x = torch.randn(len(ids), K, device=DEV, generator=_gen(8)).bfloat16()
    got = []
    for rows in (64, 128):
        _, _, _, tiles, ntile, max_tiles = cu.moe_sort(shuffled, E, rows)
        got.append(mx.moe_mxfp4_tc(x, w, len(ids), max_tiles, tiles=tiles, ntile=ntile, out_f32=True, tile_rows=rows))
    assert torch.equal(*got) and cu.read_status(torch.device(DEV))[0] == 0


@pytest.mark.parametrize("K,N,act", [(2816, 256, 0), (5632, 128, 1)])
def test_exl3_pairs_of_lengths_in_chunks_of_128(K, N, act):
    """No count of slices leaves these lengths whole chunks of 256."""
    test_exl3_pairs_do_not_depend_on_their_number(K, N, act)


@pytest.mark.parametrize("at", [16, 40, 63, 107])
def test_chunked_delta_rule_in_front_of_a_row_of_nan(at):
    """Rows of earlier blocks than a row of NaN do not see it, as with products of 16 rows (P's blocks above the diagonal are 0, and not
    multiplied).  A chunk's blocks are rows 0, 16 and 32 on: the inverse of its last 32 rows is one product."""
    import dataclasses
    from spark_engine_b200.config import ModelConfig, GdnConfig
    from spark_engine_b200.models.model import GdnMixer
    from spark_engine_b200.models.plan import make_plan
    from spark_engine_b200.ops import cuda as cu
    cfg = dataclasses.replace(ModelConfig(), gdn=GdnConfig(n_k_heads=1, n_v_heads=2, head_dim=128))
    g = _gen(15)
    w = {"conv": torch.rand(512, 4, device=DEV, generator=g) - 0.5, "A_log": torch.zeros(2, device=DEV), "dt_bias": torch.zeros(2, device=DEV),
         "norm": torch.ones(128, device=DEV)}
    proj = torch.randn(130, 768, device=DEV, generator=g).bfloat16()
    ab = torch.randn(130, 4, device=DEV, generator=g).bfloat16()
    outs = []
    for bad in (False, True):
        if bad:
            proj[at] = float("nan")
        m = GdnMixer(cfg, w, 1, DEV, torch.bfloat16)
        outs.append(cu.gdn_mixer(m, proj, ab, make_plan([(0, [1] * 130, 5)], device=DEV), True))
    assert cu.read_status(torch.device(DEV))[0] == 0
    whole = at // 64 * 64 + (0, 16, 32, 32)[at % 64 // 16]
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0][:whole], outs[1][:whole]) and torch.isnan(outs[1][at:]).any(1).all()


def test_exl3_scales_on_any_element():
    """Output scales that start on 2 bytes (a view into a larger buffer) give the bits of aligned ones."""
    from spark_engine_b200.ops import cuda as cu
    w = Q.random_exl3(256, 128, 4, 0, 0.05, 3, DEV)
    x = torch.randn(140, 128, device=DEV, generator=_gen(3)).bfloat16()
    y = cu.exl3_linear(x, w)
    w.svh = torch.cat((w.svh[:1], w.svh))[1:]
    assert w.svh.data_ptr() % 8 == 2 and torch.equal(cu.exl3_linear(x, w), y)


@pytest.mark.parametrize("M,N,pairs", [(31, 4096, 0), (32, 4096, 1), (31, 3968, 1), (128, 9216, 1), (128, 9344, 0), (129, 9344, 1)])
def test_exl3_rows_take_pairs_or_a_pass(monkeypatch, M, N, pairs):
    from spark_engine_b200.ops import cuda as cu
    w = Q.random_exl3(N, 128, 4, 0, 0.05, M, DEV)
    x = torch.randn(M, 128, device=DEV, generator=_gen(M)).bfloat16()
    calls, gemm = [], cu.gemm_exl3
    monkeypatch.setattr(cu, "gemm_exl3", lambda *a: calls.append(1) or gemm(*a))
    y = cu.exl3_linear(x, w)
    assert len(calls) == pairs and torch.equal(y, gemm(cu.exl3_had_rows(x, w.suh, post=False), cu.exl3_reconstruct(w), w.svh))


@pytest.mark.parametrize("M,N,K", [(129, 24576, 2048), (257, 16384, 4096), (150, 9216, 128), (257, 641, 128)])
def test_rows_of_a_product_do_not_depend_on_the_tile_width(M, N, K):
    """Few rows, matrices that L2 keeps and that it does not, against rows in batches of 128 (other tile widths)."""
    from spark_engine_b200.ops import cuda as cu
    x = torch.randn(M, K, device=DEV, generator=_gen(M)).bfloat16()
    w = torch.randn(N, K, device=DEV, generator=_gen(N)).bfloat16()
    for f32 in (False, True):
        assert torch.equal(cu.gemm_bf16(x, w, f32), torch.cat([cu.gemm_bf16(x[i: i + 128], w, f32) for i in range(0, M, 128)]))


@pytest.mark.parametrize("limit", [0.0, 3.0])
@pytest.mark.parametrize("K,N", [(128, 128), (512, 256), (1152, 128), (2048, 1024)])
def test_exl3_gated_rows_do_not_depend_on_their_number(K, N, limit):
    """Few blocks are gated and transformed a warp each, many by eight lanes each: the bits of a row are the same, from rows on any alignment."""
    from spark_engine_b200.ops import cuda as cu
    w = Q.random_exl3(N, K, 4, 0, 0.05, 4, DEV)
    x = 2 * torch.randn(16, 2 * K + 8, device=DEV, generator=_gen(K))
    for shift in (0, 4, 1):
        h = x.bfloat16()[:, shift: shift + 2 * K]
        y = cu.exl3_gemv(h, w, act=1, limit=limit, out_f32=True)
        for n in (1, 2, 5, 9):
            assert torch.equal(cu.exl3_gemv(h[:n], w, act=1, limit=limit, out_f32=True), y[:n]), (shift, n)


@pytest.mark.parametrize("H", [64, 1028, 2050])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 33])
def test_combine_of_few_and_many_slots(H, k):
    """Slots looked up by every thread and through the row's table; vectors and single columns; pairs of experts on other ranks."""
    from spark_engine_b200.ops import cuda as cu
    P, R, g = cu.P, 5, _gen(H + k)
    w, sg = torch.rand(R, k, device=DEV, generator=g), torch.rand(R, device=DEV, generator=g)
    inv = torch.randperm(R * k, device=DEV, generator=g).int()
    pe = torch.randint(-1, 2, (R * k,), device=DEV, generator=g, dtype=torch.int32)
    shared, res0 = torch.randn(R, H, device=DEV, generator=g).bfloat16(), torch.randn(R, H, device=DEV, generator=g)
    for dtype in (torch.float32, torch.bfloat16):
        y = torch.randn(R * k, H, device=DEV, generator=g).to(dtype)
        res, out = res0.clone(), torch.empty(R, H, device=DEV, dtype=torch.bfloat16)
        cu.check(cu.lib().spark_moe_combine(P(res), P(y), int(dtype == torch.float32), P(inv), P(w), R, k, P(shared), P(sg), H, P(out), cu.stream(),
                                            P(pe)), "spark_moe_combine")
        terms = (y[inv.long()].double() * (w.view(-1, 1) * (pe >= 0).view(-1, 1)).double()).view(R, k, H)
        ref = terms.sum(1) + sg.double().unsqueeze(1) * shared.double()
        size = terms.abs().sum(1) + (sg.unsqueeze(1) * shared).double().abs()
        assert ((res.double() - res0.double() - ref).abs() <= (k + 2) * 2.0 ** -24 * (size + res0.double().abs())).all()
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (k + 2) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("E", [1, 7, 640, 641])
@pytest.mark.parametrize("P", [1, 33, 640, 641])
def test_sort_of_few_pairs(E, P):
    """One launch and three: stable order, pairs of other ranks (-1) left out."""
    from spark_engine_b200.ops import cuda as cu
    ids = torch.randint(-1, E, (P,), dtype=torch.int32, generator=torch.Generator().manual_seed(P))
    perm, inv, offs, tiles, ntile, _ = cu.moe_sort(ids.to(DEV), E, 64)
    local = (ids >= 0).nonzero()[:, 0]
    order = local[torch.sort(ids[local], stable=True).indices]
    n = torch.bincount(ids[local].long(), minlength=E)
    want = torch.full((P,), -1, dtype=torch.int32)
    want[order] = torch.arange(len(order), dtype=torch.int32)
    assert torch.equal(perm[: len(order)].cpu().long(), order) and torch.equal(inv.cpu(), want)
    assert torch.equal(offs.cpu().long(), torch.cat((torch.zeros(1, dtype=torch.int64), n.cumsum(0))))
    t = tiles[: ntile.item()].tolist()
    assert [e for _, _, e, _ in t] == [e for e in range(E) for _ in range(-(-int(n[e]) // 64))]
    assert sorted(r for row, _, _, m in t for r in range(row, row + m)) == list(range(len(order)))


@pytest.mark.parametrize("rows,pos0,k", [(40, 200, 16), (129, 0, 8), (200, 1900, 256)])
def test_masked_attention_on_the_selection_masks(rows, pos0, k):
    """The masks as the selection leaves them, through the prompt tiles: attention over the tokens of its token list, in 64 bits."""
    from spark_engine_b200.ops import cuda as cu, sparse as sp
    P, g, D, Hq, Hkv = cu.P, _gen(rows), 64, 4, 2
    ctx = pos0 + rows
    q = torch.randn(rows, Hq, D, device=DEV, generator=g).bfloat16()
    kv = torch.randn(2, ctx, Hkv, D, device=DEV, generator=g).bfloat16()
    pos = torch.arange(pos0, ctx, dtype=torch.int32, device=DEV)
    nb, mw = ctx // 4, (ctx + 127) // 128
    score = torch.randint(0, 50, (rows, nb), device=DEV, generator=g).float()
    sel, sel_n = sp.topk_select(score, nb, pos, 4, k)
    mask = torch.full((rows, mw), -1, dtype=torch.int32, device=DEV)
    cu.check(sp._dll().spark_topk_mask(P(score), nb, P(pos), rows, k, P(mask), mw, cu.stream(), 0), "spark_topk_mask")
    out = torch.empty(rows, Hq, D, device=DEV, dtype=torch.bfloat16)
    seg = torch.tensor([[0, 0, rows, pos0]], dtype=torch.int32, device=DEV)
    row_kv = torch.zeros(rows, dtype=torch.int64, device=DEV)
    cu.check(cu.lib().spark_attn_prefill_masked(P(q), P(kv[0]), P(kv[1]), P(row_kv), P(seg), 1, rows, P(q), Hq * D, 0, P(out), Hq, Hkv, D, D ** -0.5,
                                                None, None, 0, rows, P(mask), mw, ctx, P(cu.status_word(torch.device(DEV))), cu.stream()), "masked")
    assert cu.read_status(torch.device(DEV))[0] == 0
    kk, vv = (t.double().repeat_interleave(Hq // Hkv, 1) for t in kv)
    hide = torch.ones(rows, ctx, dtype=torch.bool, device=DEV)
    for r in range(rows):
        hide[r, sel[r, : sel_n[r]].long()] = False
    s = torch.einsum("rhd,khd->hrk", q.double(), kk) * D ** -0.5
    ref = torch.einsum("hrk,khd->rhd", torch.softmax(s.masked_fill(hide, -float("inf")), -1), vv)
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2.0 ** -7.5             # as the token lists' test: two bf16 roundings and their sums


@pytest.mark.parametrize("D", [80, 128])
@pytest.mark.parametrize("ctx", [3, 64, 250, 256, 257])
def test_decode_attention_of_few_splits(D, ctx):
    """Up to four splits and more, rows that see the first split only (the others are empty, their partial rows not written)."""
    from spark_engine_b200.ops import cuda as cu
    P, g, Hq, Hkv, ns = cu.P, _gen(ctx), 8, 4, (ctx + 63) // 64
    q, qkv = torch.randn(2, Hq, D, device=DEV, generator=g).bfloat16(), torch.randn(2, 2 * Hq * D, device=DEV, generator=g).bfloat16()
    kv = torch.randn(2, ctx, Hkv, D, device=DEV, generator=g).bfloat16()
    pos = torch.tensor([ctx - 1, min(ctx - 1, 40)], dtype=torch.int32, device=DEV)
    row_kv = torch.zeros(2, dtype=torch.int64, device=DEV)
    po, pm = (torch.full((2 * Hq * ns * n,), float("nan"), device=DEV) for n in (D, 2))
    out = torch.empty(2, Hq, D, device=DEV, dtype=torch.bfloat16)
    cu.check(cu.lib().spark_attn_decode(P(q), P(kv[0]), P(kv[1]), None, None, 0, P(pos), P(row_kv), None, None, 0, P(po), P(pm), ns, P(qkv), 2 * Hq * D, 1,
                                        2, Hq, Hkv, D, D ** -0.5, P(out), cu.stream(), None, None, None, 1), "spark_attn_decode")
    kk, vv = (t.double().repeat_interleave(Hq // Hkv, 1) for t in kv)
    s = torch.einsum("rhd,khd->hrk", q.double(), kk) * D ** -0.5
    s = s.masked_fill(torch.arange(ctx, device=DEV) > pos.unsqueeze(1), -float("inf"))
    ref = torch.einsum("hrk,khd->rhd", torch.softmax(s, -1), vv) * torch.sigmoid(qkv.view(2, Hq, 2, D)[:, :, 1].double())
    assert ((out.double() - ref).norm() / ref.norm()).item() < 2.0 ** -7.5             # probabilities and results in bf16


@pytest.mark.parametrize("H,L", [(64, 128), (40, 256), (64, 512)])
def test_latent_attention_does_not_depend_on_the_warps(H, L):
    """Few rows take sixteen warps per CTA, many eight (where two CTAs fit an SM): the bits of a row are the same."""
    from spark_engine_b200.ops import cuda as cu
    P, g, rope, ctx, rows = cu.P, _gen(H + L), 64, 200, 160
    KW, ns = L + rope, (ctx + 63) // 64
    q, lat = torch.randn(rows, H, KW, device=DEV, generator=g).bfloat16(), torch.randn(ctx, KW, device=DEV, generator=g).bfloat16()
    pos = torch.arange(ctx - rows, ctx, dtype=torch.int32, device=DEV)
    row_kv, sink = torch.zeros(rows, dtype=torch.int64, device=DEV), torch.randn(H, device=DEV, generator=g)

    def run(lo, hi):
        R = hi - lo
        po, pm, out = torch.empty(R * H * ns * L, device=DEV), torch.empty(R * H * ns * 2, device=DEV), torch.empty(R, H, L, device=DEV, dtype=torch.bfloat16)
        cu.check(cu.lib().spark_mla_attn(P(q[lo:hi]), P(lat), P(pos[lo:hi]), P(row_kv), None, None, 0, P(po), P(pm), ns, P(sink), R, H, L, rope, KW ** -0.5,
                                         P(out), cu.stream(), None, None, None, 0), "spark_mla_attn")
        return out
    y = run(0, rows)
    for lo, hi in ((0, 1), (7, 40), (100, 160)):
        assert torch.equal(run(lo, hi), y[lo:hi])
    s = torch.einsum("rhd,kd->hrk", q.double(), lat.double()) * KW ** -0.5
    s = s.masked_fill(torch.arange(ctx, device=DEV) > pos.unsqueeze(1), -float("inf"))
    w = torch.softmax(torch.cat((s, sink.double().view(H, 1, 1).expand(H, rows, 1)), -1), -1)[..., :-1]
    ref = torch.einsum("hrk,kd->rhd", w, lat[:, :L].double())
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -7.5             # probabilities and results in bf16


@pytest.mark.parametrize("K", [128, 512, 640])
def test_rows_quantised_before_and_behind_their_gather(monkeypatch, K):
    from spark_engine_b200.ops import mx
    h = 3 * torch.randn(37, K, device=DEV, generator=_gen(K)).bfloat16()
    rows = torch.randint(0, 37, (300,), device=DEV, generator=_gen(K), dtype=torch.int32)
    behind = mx._quantised_rows(h, rows)
    monkeypatch.setattr(mx, "QUANTISE_FIRST", 0)
    for a, b in zip(mx._quantised_rows(h, rows), behind):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
