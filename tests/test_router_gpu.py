"""The fused decode router at the edges of its tiles: rows around 8 and 16, widths that leave lanes without a vector, expert counts
around the forms' limits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("R", [1, 8, 9, 16])
@pytest.mark.parametrize("K,E,k", [(8, 4, 2), (264, 64, 6), (2048, 257, 10), (4096, 512, 8), (6152, 513, 32)])
def test_logits_and_choice(R, K, E, k):
    from spark_engine_b200.ops import cuda as cu
    P, g = cu.P, torch.Generator(device=DEV).manual_seed(K + R)
    x = torch.randn(R, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(E + 1, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    ld = (E + 8) // 8 * 8
    logits = torch.empty(16, ld, device=DEV)
    counter = torch.zeros(4, dtype=torch.int32, device=DEV)
    wts, ids = torch.empty(R, k, device=DEV), torch.empty(R, k, dtype=torch.int32, device=DEV)
    row, sg = torch.empty(R, k, dtype=torch.int32, device=DEV), torch.empty(R, device=DEV)
    for _ in range(2):                                              # the arrival counter is zero again
        cu.check(cu.lib().spark_moe_router_topk(P(x), K, P(w), K, P(logits), ld, R, K, E, k, 0, None, 1.0, 1, k, E, 0, E, 0, 1, P(wts), P(ids),
                                                P(row), P(sg), P(counter), 0, None, cu.stream()), "router")
    z = x.double() @ w.double().t()
    got = logits[:R, : E + 1].double()
    assert (got - z).abs().max() < K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()).max()
    best = torch.sort(logits[:R, :E], dim=-1, descending=True, stable=True)
    assert torch.equal(ids.long(), best.indices[:, :k])
    p = torch.softmax(best.values[:, :k].double(), -1)
    assert torch.allclose(wts.double(), p, rtol=1e-5, atol=1e-7)
    assert torch.allclose(sg.double(), torch.sigmoid(got[:, E]), rtol=1e-5)
    # a row does not depend on the rows beside it
    alone = torch.empty(16, ld, device=DEV)
    cu.check(cu.lib().spark_moe_router_topk(P(x[R - 1:]), K, P(w), K, P(alone), ld, 1, K, E, k, 0, None, 1.0, 1, k, E, 0, E, 0, 1, P(wts), P(ids),
                                            P(row), P(sg), P(counter), 0, None, cu.stream()), "router")
    assert torch.equal(alone[0, : E + 1], logits[R - 1, : E + 1])


@pytest.mark.parametrize("R", [1, 4, 5, 9, 16])
@pytest.mark.parametrize("K,E", [(8, 3), (2048, 512), (4104, 61), (6152, 513)])
def test_logits_are_32_bit_chains(R, K, E):
    """A logit is the sum the rest of the engine takes for a row: a lane's products in one 32-bit chain, the lanes pairwise.  (A product
    of two bf16 numbers is exact in 32 bits, so the chain can be followed with plain additions.)"""
    from spark_engine_b200.ops import cuda as cu
    P, g = cu.P, torch.Generator(device=DEV).manual_seed(K + R)
    x = (torch.randn(R, K, device=DEV, generator=g).abs() + 0.5).bfloat16()
    w = torch.rand(E + 1, K, device=DEV, generator=g).bfloat16()
    ld = (E + 8) // 8 * 8
    logits = torch.empty(R, ld, device=DEV)
    counter = torch.zeros(4, dtype=torch.int32, device=DEV)
    wts, ids = torch.empty(R, 1, device=DEV), torch.empty(R, 1, dtype=torch.int32, device=DEV)
    row, sg = torch.empty(R, 1, dtype=torch.int32, device=DEV), torch.empty(R, device=DEV)
    cu.check(cu.lib().spark_moe_router_topk(P(x), K, P(w), K, P(logits), ld, R, K, E, 1, 0, None, 1.0, 1, 1, E, 0, E, 0, 1, P(wts), P(ids),
                                            P(row), P(sg), P(counter), 0, None, cu.stream()), "router")
    steps = -(-K // 256)
    prod = torch.zeros(R, E + 1, steps * 256, device=DEV)
    prod[..., :K] = x.float().unsqueeze(1) * w.float()
    prod = prod.view(R, E + 1, steps, 32, 8)
    acc = torch.zeros(R, E + 1, 32, device=DEV)
    for s in range(steps):
        for j in range(8):
            acc = acc + prod[:, :, s, :, j]
    while acc.shape[-1] > 1:
        h = acc.shape[-1] // 2
        acc = acc[..., :h] + acc[..., h:]
    assert torch.equal(logits[:, : E + 1], acc[..., 0])
