"""Exact block selection in both thread counts: ties, candidates beyond one round of a CTA, block sizes, windows that cut a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _expect(score, p, block, k, window):
    vis = (p + 1) // block
    if vis <= k:
        return list(range(p + 1))
    top = torch.sort(score[:vis], descending=True, stable=True).indices[:k].tolist()
    lo = min(max(0, p + 1 - window), vis * block) if window else vis * block
    return sorted({t for b in top for t in range(b * block, b * block + block) if t < lo}) + list(range(lo, p + 1))


@pytest.mark.parametrize("R", [3, 300])
@pytest.mark.parametrize("nb,block,k,window", [(9, 4, 2, 0), (700, 4, 512, 0), (1025, 4, 100, 6), (2100, 8, 64, 21), (4200, 2, 1000, 0), (40, 200, 7, 301)])
@pytest.mark.parametrize("levels", [3, 0])
def test_selection(R, nb, block, k, window, levels):
    from spark_engine_b200.ops import sparse
    g = torch.Generator(device=DEV).manual_seed(R + nb)
    score = torch.randn(R, nb, device=DEV, generator=g)
    if levels:
        score = (score.relu() * levels).round()                     # few distinct values: the threshold is a tie
    pos = torch.randint(0, nb * block, (R,), device=DEV, generator=g).int()
    pos[0] = nb * block - 1
    sel, n = sparse.topk_select(score, nb, pos, block, k, window, ctas=1)
    sel, n, sc, ps = sel.cpu(), n.tolist(), score.cpu(), pos.tolist()
    for r in list(range(0, R, 23)) + [R - 1]:
        assert sel[r, : n[r]].tolist() == _expect(sc[r], ps[r], block, k, window), r
