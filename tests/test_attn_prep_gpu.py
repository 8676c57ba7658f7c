"""The two forms of the attention preparation: a warp per head (prompts) and a CTA per head (decode) give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D,rope", [(64, 64), (128, 32), (256, 64)])
@pytest.mark.parametrize("fp8", [0, 1])
@pytest.mark.parametrize("gated", [0, 1])
def test_forms_give_the_same_bits(D, rope, fp8, gated):
    """Two segments that start within a block, in one launch (301 rows of 9 heads: warps, the last CTA not full) and in slices of at most
    150 rows (CTAs), whose pooled keys take their earlier rows from the cache."""
    from spark_engine_b200.ops import cuda as cu
    P, g = cu.P, torch.Generator(device=DEV).manual_seed(D + fp8)
    Hq, Hkv, ih, idim, block = 4, 1, 2, 128, 4
    segs = [(150, 5, 0), (151, 3, 400)]                              # rows, first position, cache row of the sequence's first token
    cuts = [(0, 37), (37, 150), (150, 151), (151, 290), (290, 301)]
    R, jobs, tokens = 301, Hq + 2 * Hkv + ih + 1, 600
    assert R * jobs >= 148 * 16 and R * jobs % 4 and all((b - a) * jobs < 148 * 16 for a, b in cuts)
    ld = Hq * D * (1 + gated) + 2 * Hkv * D + (ih + 1) * idim + 8
    qkv = (torch.randn(R, ld, device=DEV, generator=g) * 2).bfloat16()
    norms = [torch.rand(n, device=DEV, generator=g) - 0.5 for n in (D, D, idim, idim)]
    inv = (1e4 ** (-torch.arange(rope // 2, dtype=torch.float64) * 2 / rope)).to(DEV)
    raw0 = torch.randn(tokens, idim, device=DEV, generator=g)
    pos = torch.tensor([p + i for n, p, _ in segs for i in range(n)], dtype=torch.int32, device=DEV)
    kv = torch.tensor([b for n, _, b in segs for _ in range(n)], dtype=torch.int64, device=DEV)
    first = [0] * segs[0][0] + [segs[0][0]] * segs[1][0]             # first row of a row's segment

    def run(parts):
        f = lambda *s, dt=torch.float32: torch.zeros(*s, dtype=dt, device=DEV)
        cache = torch.float8_e4m3fn if fp8 else torch.bfloat16
        out = [f(R, Hq, D, dt=torch.bfloat16), f(tokens, Hkv, D).to(cache), f(tokens, Hkv, D).to(cache), f(tokens, Hkv), f(tokens, Hkv), f(R, ih, idim),
               raw0.clone(), f(tokens // block, idim)]
        q, k, v, ks, vs, qi, raw, pool = out
        for a, b in parts:
            j = torch.tensor([r - max(a, first[r]) for r in range(a, b)], dtype=torch.int32, device=DEV)
            cu.check(cu.lib().spark_attn_prep(P(qkv[a:]), ld, b - a, Hq, Hkv, D, rope, gated, 1, ih, idim, block, fp8, 1e-6, *map(P, norms),
                                              P(inv), P(pos[a:]), P(kv[a:]), P(j), P(q[a:]), P(k), P(v), P(ks), P(vs), P(qi[a:]), P(raw), P(pool),
                                              cu.stream(), None), "attn_prep")
        torch.cuda.synchronize()
        return out
    for name, x, y in zip(("q", "k", "v", "k scales", "v scales", "index q", "raw keys", "pooled keys"), run([(0, R)]), run(cuts)):
        assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), name
        if "scales" not in name or fp8:
            assert x.float().abs().sum() > 0, name
