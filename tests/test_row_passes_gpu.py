"""The vectorised row passes at the edges of their forms: rows that do not start on 16 bytes, widths that are no multiple of the
vector, last lanes and warps that are not full, ties and infinities in the router."""
import pytest
import torch

from spark_engine_b200.quant import formats as Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen(seed=0):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("R,K,block", [(1, 32, 32), (3, 96, 32), (5, 128, 128), (7, 4096, 32), (33, 384, 128), (300, 1024, 32)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("act", [0, 1])
def test_act_quant_forms_agree(R, K, block, dtype, act):
    """Rows on odd addresses give the same bytes as aligned ones, and the scales are those of the plain formula."""
    from spark_engine_b200.ops import mx
    W = K * (1 + act)
    wide = (torch.randn(R, W + 1, device=DEV, generator=_gen()) * 3).to(dtype)
    x = wide[:, 1:]
    qa, sa = mx.act_quant(x, block=block, act=act, limit=2.0 * act)
    qb, sb = mx.act_quant(x.contiguous(), block=block, act=act, limit=2.0 * act)
    assert torch.equal(qa.view(torch.uint8), qb.view(torch.uint8)) and torch.equal(sa, sb)
    if act:
        return
    qr, sr = Q.act_quant_fp8(x.float().cpu(), block=block, pow2=block == 32)
    sc = sa.cpu().float() if block == 128 else Q.e8m0_to_float(sa.cpu())
    assert torch.allclose(sc, sr, rtol=1e-6)
    step = (qa.cpu().float() - qr.float()).abs()                  # a tie of the division may fall to the other neighbour
    assert (step > 0.125 * qr.float().abs() + 2.0 ** -9).sum() == 0


def _had(x):
    return (x.view(*x.shape[:-1], -1, 128) @ Q.hadamard128().double().to(x.device)).view(x.shape)


@pytest.mark.parametrize("R,C", [(1, 128), (3, 384), (31, 256), (5, 2048)])
@pytest.mark.parametrize("shift", [0, 4])
def test_hadamard_rows(R, C, shift):
    from spark_engine_b200.ops import cuda as cu
    x = torch.randn(R, C + shift, device=DEV, generator=_gen(1)).bfloat16()[:, shift:]
    sc = torch.randn(C, device=DEV, generator=_gen(2)).half()
    y = cu.exl3_had_rows(x, sc, post=False)
    ref = _had(x.double() * sc.double())
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -11          # one fp16 rounding
    xf = torch.randn(R, C, device=DEV, generator=_gen(3))
    y = cu.exl3_had_rows(xf, sc, post=True)
    ref = _had(xf.double()) * sc.double()
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8           # one bf16 rounding


@pytest.mark.parametrize("R,H,k", [(1, 8, 1), (3, 100, 3), (17, 2048, 10), (9, 2056, 4), (5, 33, 5)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("local", [False, True])
def test_combine(R, H, k, dtype, local):
    from spark_engine_b200.ops import cuda as cu
    P, g = cu.P, _gen(4)
    y = torch.randn(R * k, H, device=DEV, generator=g).to(dtype)
    inv = torch.randperm(R * k, device=DEV, generator=g).int()
    wts = torch.rand(R, k, device=DEV, generator=g)
    sh = torch.randn(R, H, device=DEV, generator=g).bfloat16()
    sg = torch.rand(R, device=DEV, generator=g)
    pe = torch.randint(-1, 3, (R, k), device=DEV, generator=g).int() if local else None
    if local:
        inv = torch.where(pe.view(-1) < 0, -1, inv)
    out = torch.empty(R, H, dtype=torch.bfloat16, device=DEV)
    res = torch.randn(R, H, device=DEV, generator=g)
    res0 = res.clone()
    cu.check(cu.lib().spark_moe_combine(P(res), P(y), int(dtype == torch.float32), P(inv), P(wts), R, k, P(sh), P(sg), H, P(out),
                                        cu.stream(), P(pe)), "combine")
    w = wts.double() * (pe >= 0) if local else wts.double()
    ref = (w.unsqueeze(-1) * y.double()[inv.view(R, k).clamp_min(0).long()]).sum(1) + sg.double().unsqueeze(1) * sh.double()
    assert torch.allclose(out.double(), ref, rtol=2.0 ** -8, atol=1e-5 * k)
    assert torch.allclose((res - res0).double(), ref, rtol=1e-5, atol=2e-6 * (k + 2))


@pytest.mark.parametrize("R,H", [(1, 4), (3, 128), (2, 2050), (5, 2052), (2, 8192), (2, 8196)])
@pytest.mark.parametrize("dtype", [None, torch.bfloat16, torch.float32])
def test_add_norm(R, H, dtype):
    from spark_engine_b200.ops import cuda as cu
    g = _gen(5)
    res = torch.randn(R, H, device=DEV, generator=g)
    w = torch.randn(H, device=DEV, generator=g)
    d = None if dtype is None else torch.randn(R, H, device=DEV, generator=g).to(dtype)
    x = res.double() + (0 if d is None else d.double())
    h, X = cu.add_rmsnorm(d, res.clone(), w, 1e-6)
    assert torch.allclose(X.double(), x, rtol=1e-6, atol=1e-6)
    ref = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    assert torch.allclose(h.double(), ref, rtol=2.0 ** -8, atol=1e-6)


@pytest.mark.parametrize("E,k", [(8, 8), (64, 6), (65, 4), (512, 10), (513, 10), (1024, 32)])
@pytest.mark.parametrize("kind", range(6))
@pytest.mark.parametrize("R", [1, 17])
def test_route(E, k, kind, R):
    """Choices of every router kind against a stable sort (ties to the lowest expert), weights against 64 bits."""
    from spark_engine_b200.ops import cuda as cu
    P, g = cu.P, _gen(6)
    x = torch.randn(R, E + 1, device=DEV, generator=g)
    x[:, : E // 2] = (x[:, : E // 2] * 2).round() / 2               # ties, zeros of both signs among them
    if k < E:                                                        # (a row that has to choose it has no weight for it)
        x[0, 1] = -float("inf")
    bias = (torch.randn(E, device=DEV, generator=g) * 0.1).round(decimals=1)
    wts = torch.empty(R, k, device=DEV)
    ids = torch.empty(R, k, dtype=torch.int32, device=DEV)
    row = torch.empty(R, k, dtype=torch.int32, device=DEV)
    sg = torch.empty(R, device=DEV)
    sw = torch.empty(R, device=DEV)
    n_self = 2
    cu.check(cu.lib().spark_moe_route(P(x), E + 1, R, E, k, kind, P(bias), 1.5, 1, P(wts), P(ids), P(row), P(sg), cu.stream(), 0,
                                      E - n_self, n_self, P(sw)), "route")
    z = x[:, :E].double()
    if kind in (0, 3):
        p = torch.softmax(z, -1)
    elif kind in (1, 4):
        p = torch.sigmoid(z)
    else:
        p = torch.nn.functional.softplus(z).sqrt()
    s = {0: z, 1: p + bias, 2: p + bias, 3: p + bias, 4: z, 5: z + bias}[kind]
    full = torch.where((ids >= 0), ids, E - 1).long()
    got = torch.gather(s, 1, full)
    best = torch.sort(s, dim=-1, descending=True, stable=True)
    own = ids < 0                                                  # identity experts (the last two), or none left
    finite = best.values[:, :k] > -float("inf")
    assert torch.allclose(torch.where(own | ~finite, 0.0, got), torch.where(own | ~finite, 0.0, best.values[:, :k]), rtol=0, atol=1e-6)
    if kind in (0, 4, 5):                                          # scores that are the same numbers on both sides
        ref = best.indices[:, :k]
        if kind != 5:
            assert torch.equal(torch.where(finite, ids.long(), -1), torch.where(finite & (ref < E - n_self), ref, -1))
        num = torch.gather(p, 1, ref) if kind != 5 else torch.softmax(best.values[:, :k], -1)
        w = num * 1.5 if kind == 4 else num / num.sum(-1, keepdim=True).clamp_min(1e-20) * 1.5
        assert torch.allclose(wts.double(), w, rtol=1e-4, atol=1e-6)
        if kind != 5:
            assert torch.allclose(sw.double(), (w * (ref >= E - n_self)).sum(-1), rtol=1e-4, atol=1e-6)
    else:                                                          # the scores are rounded, so near-ties may fall either way: the weights
        num = torch.gather(p, 1, full)                             # of the experts that were chosen, from p without the bias
        if not own.any():
            assert torch.allclose(wts.double(), num / num.sum(-1, keepdim=True).clamp_min(1e-20) * 1.5, rtol=1e-4, atol=1e-6)
        else:                                                      # an identity expert's number is not in `ids`: ratios of the others
            a, b = torch.where(own, 0.0, wts.double()), torch.where(own, 0.0, num)
            assert torch.allclose(a * b.sum(-1, keepdim=True), b * a.sum(-1, keepdim=True), rtol=1e-4, atol=1e-6)
    if kind != 4:                                                  # what the other experts leave of the whole is the identity experts'
        assert torch.allclose(sw.double(), 1.5 - torch.where(own, 0.0, wts.double()).sum(-1), rtol=1e-4, atol=1e-5)
    assert torch.equal(row, torch.arange(R, device=DEV, dtype=torch.int32).unsqueeze(1).expand(R, k))
    assert torch.allclose(sg, torch.sigmoid(x[:, E]), rtol=1e-5, atol=1e-6)
