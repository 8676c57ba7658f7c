"""Prompt attention on tcgen05 against 64-bit softmax attention: head widths, ragged row and key tiles, several segments behind
committed prefixes, block masks, a cache that holds NaN where no key is."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _run(D, Hq, Hkv, segs, gated, masked, seed=0, grow=1.0):
    """segs: (rows, earlier keys, cache base).  Returns (device output, 64-bit output)."""
    from spark_engine_b200.ops import cuda as cu
    P = cu.P
    g = torch.Generator(device=DEV).manual_seed(seed)
    R = sum(n for n, _, _ in segs)
    end = max(b + p + n for n, p, b in segs)
    k = torch.full((end + 70, Hkv, D), float("nan"), device=DEV, dtype=torch.bfloat16)
    v = k.clone()
    q = torch.randn(R, Hq, D, device=DEV, generator=g).bfloat16()
    ld = Hq * 2 * D + 8
    qkv = torch.randn(R, ld, device=DEV, generator=g).bfloat16()
    seg, row_kv, r0 = [], [], 0
    for n, p, b in segs:
        kk = torch.randn(p + n, Hkv, D, device=DEV, generator=g)
        kk *= torch.linspace(1, grow, p + n, device=DEV).view(-1, 1, 1)         # later keys are larger: maxima keep growing
        k[b: b + p + n] = kk.bfloat16()
        v[b: b + p + n] = torch.randn(p + n, Hkv, D, device=DEV, generator=g).bfloat16()
        seg.append((0, r0, n, p))
        row_kv += [b] * n
        r0 += n
    seg_t = torch.tensor(seg, dtype=torch.int32, device=DEV)
    row_kv = torch.tensor(row_kv, dtype=torch.int64, device=DEV)
    out = torch.full((R, Hq * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    status = cu.status_word(torch.device(DEV))
    scale = 1 / math.sqrt(D)
    nctx = max(p + n for n, p, _ in segs)
    vis = None
    tail = (R, end, P(status), cu.stream())
    if masked:
        nb = (nctx + 3) // 4
        pick = torch.rand(R, nb, device=DEV, generator=g) < 0.3
        pos = torch.cat([torch.arange(p, p + n, device=DEV) for n, p, _ in segs])
        pick[torch.arange(R, device=DEV), pos // 4] = True                      # a row sees at least its own block
        pick &= torch.arange(nb, device=DEV) <= (pos // 4).unsqueeze(1)
        toks = [(pick[i].repeat_interleave(4).nonzero()[:, 0]) for i in range(R)]
        sel_ld = max(len(t) for t in toks)
        sel = torch.zeros(R, sel_ld, dtype=torch.int32, device=DEV)
        for i, t in enumerate(toks):
            sel[i, : len(t)] = t.int()
        sel_n = torch.tensor([len(t) for t in toks], dtype=torch.int32, device=DEV)
        mw = (nctx + 127) // 128
        bm = torch.empty(R * mw, dtype=torch.int32, device=DEV)
        cu.check(cu.lib().spark_attn_prefill_masked(P(q), P(k), P(v), P(row_kv), P(seg_t), len(segs), max(s[0] for s in segs), P(qkv), ld,
                                                    int(gated), P(out), Hq, Hkv, D, scale, P(sel), P(sel_n), sel_ld, R, P(bm), mw, end,
                                                    P(status), cu.stream()), "masked")
        vis = pick.repeat_interleave(4, 1)[:, :nctx]
    else:
        cu.check(cu.lib().spark_attn_prefill(P(q), P(k), P(v), P(row_kv), P(seg_t), len(segs), max(s[0] for s in segs), P(qkv), ld,
                                             int(gated), P(out), Hq, Hkv, D, scale, *tail), "dense")
    torch.cuda.synchronize()
    assert cu.read_status(torch.device(DEV))[0] == 0
    ref = torch.empty(R, Hq, D, dtype=torch.float64, device=DEV)
    for (_, r0, n, p), (_, _, b) in zip(seg, segs):
        kk, vv = (t[b: b + p + n].double().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
        s = torch.einsum("rhd,khd->hrk", q[r0: r0 + n].double(), kk) * scale
        hide = torch.arange(p + n, device=DEV) > (p + torch.arange(n, device=DEV)).unsqueeze(1)
        if vis is not None:
            hide = hide | ~vis[r0: r0 + n, : p + n]
        ref[r0: r0 + n] = torch.einsum("hrk,khd->rhd", torch.softmax(s.masked_fill(hide, -math.inf), -1), vv)
    if gated:
        ref *= torch.sigmoid(qkv[:, : Hq * 2 * D].double().view(R, Hq, 2, D)[:, :, 1])
    return out.view(R, Hq, D), ref


@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 2), (128, 2, 1), (256, 16, 2), (256, 3, 3)])
@pytest.mark.parametrize("segs", [[(1, 0, 0)], [(64, 0, 5)], [(128, 0, 0)], [(129, 63, 2)], [(33, 700, 10), (200, 1, 900), (65, 127, 1200)]])
@pytest.mark.parametrize("masked", [False, True])
def test_against_64_bits(D, Hq, Hkv, segs, masked):
    out, ref = _run(D, Hq, Hkv, segs, gated=D != 64, masked=masked, seed=len(segs))
    assert torch.isfinite(out).all()
    err = ((out.double() - ref).norm() / ref.norm()).item()
    assert err < 2.0 ** -7.5, err               # probabilities and results in bf16: two roundings of 2^-9 and their sums


@pytest.mark.parametrize("masked", [False, True])
def test_growing_maxima(masked):
    """Scores that grow along the context: references are replaced and the accumulator rescaled many times."""
    out, ref = _run(256, 2, 1, [(300, 1500, 3)], gated=False, masked=masked, grow=12.0)
    err = ((out.double() - ref).norm() / ref.norm()).item()
    assert err < 2.0 ** -7.5, err


def test_repeats_bitwise():
    a, _ = _run(256, 4, 2, [(257, 100, 0)], gated=True, masked=True)
    b, _ = _run(256, 4, 2, [(257, 100, 0)], gated=True, masked=True)
    assert torch.equal(a, b)


@pytest.mark.parametrize("sparse", [0, 8])
def test_captured_rows_follow_their_plan(sparse):
    """A captured round of 32 and more rows per sequence replayed further along its sequence: the keys it reads follow the staged
    positions (dense rows, and rows whose blocks are selected)."""
    import dataclasses
    from spark_engine_b200.config import tiny_hybrid
    from spark_engine_b200.models.model import Model
    from spark_engine_b200.models.plan import make_plan
    from spark_engine_b200.models.weights import init_weights, to_device
    from spark_engine_b200.serving.graphs import RoundGraph
    cfg = tiny_hybrid()
    cfg.n_layers, cfg.layer_types = 1, ["attn"]
    cfg.attn = dataclasses.replace(cfg.attn, sparse_topk_blocks=sparse)
    cfg.moe = dataclasses.replace(cfg.moe, dense_layers=1, dense_ffn=128)
    W = to_device(init_weights(cfg, seed=0), DEV)
    ids = torch.randint(0, cfg.vocab, (240,), generator=torch.Generator().manual_seed(1)).tolist()
    n = 37

    def model():
        m = Model(cfg, W, device=DEV, dtype=torch.bfloat16, n_slots=1, kv_tokens=256)
        m.forward(make_plan([(0, ids[:40], 0)], device=DEV))
        return m
    eager, m = model(), model()
    graph = RoundGraph(m, [0], n, 256)
    for p in range(40, 240 - n, n):
        want = eager.forward(make_plan([(0, ids[p: p + n], p)], device=DEV)).float()
        graph.stage([ids[p: p + n]], [p])
        graph.run(commit=True)
        torch.cuda.synchronize()
        got = graph.logits.float()
        assert ((got - want).norm() / want.norm()).item() < 2.0 ** -7, p


def test_heaviest_weight_is_exact():
    """Two keys with the same value share a row's weight, the later one 2 to 2^8 times the earlier.  Each is the largest where it comes
    up, so its weight is 1 there and the earlier sum is scaled in 32 bits: the result is that value.  (A weight of 2^x in bf16, as a
    reference that lags behind the maximum gives it, moves the result by up to 2^-8 of it.)"""
    from spark_engine_b200.ops import cuda as cu
    P, D, n, p = cu.P, 64, 200, 128
    q = torch.zeros(n, 1, D, device=DEV, dtype=torch.bfloat16)
    q[:, 0, 0] = torch.linspace(1, 8, n, device=DEV).bfloat16()
    k = torch.zeros(p + n, 1, D, device=DEV, dtype=torch.bfloat16)
    k[1:, 0, 0] = -2000
    k[64, 0, 0] = 5.5                                               # log2 of its weight over the first key's: 0.99 q
    v = torch.zeros_like(k)
    v[0, 0] = v[64, 0] = (1 + 127 / 128 - torch.arange(D, device=DEV) / 128).bfloat16()
    out = torch.empty(n, D, device=DEV, dtype=torch.bfloat16)
    seg = torch.tensor([[0, 0, n, p]], dtype=torch.int32, device=DEV)
    row_kv = torch.zeros(n, dtype=torch.int64, device=DEV)
    cu.check(cu.lib().spark_attn_prefill(P(q), P(k), P(v), P(row_kv), P(seg), 1, n, None, 0, 0, P(out), 1, 1, D, 0.125, n, p + n,
                                         P(cu.status_word(torch.device(DEV))), cu.stream()), "dense")
    assert torch.equal(out, v[0, 0].expand_as(out))
