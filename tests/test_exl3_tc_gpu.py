"""The grouped EXL3 product on tcgen05 (trellis decoded into tensor memory) against 64-bit products of the decoded weights."""
import pytest
import torch

from spark_engine_b200.quant import formats as Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _had(x):
    return (x.view(*x.shape[:-1], -1, 128) @ Q.hadamard128().double().to(x.device)).view(x.shape)


def _setup(sizes, K, N, kind, seed=0):
    """Stack of experts, rows in expert order, tile list; experts without rows in between."""
    from spark_engine_b200.ops import cuda as cu
    E = len(sizes)
    w = Q.random_exl3(N, K, 4, E, 0.05, seed + 1, DEV, kind)
    ids = torch.tensor([e for e, n in enumerate(sizes) for _ in range(n)], dtype=torch.int32, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(seed)
    order = torch.randperm(len(ids), device=DEV, generator=g)
    perm, inv, offs, tiles, ntile, max_tiles = cu.moe_sort(ids[order].contiguous(), E)
    return cu, w, ids, tiles, ntile, max_tiles, g


def _product(x, w, e):
    return _had(x.double() @ Q.exl3_inner(w.trellis[e], w.kind).double()) * w.svh[e].double()


@pytest.mark.parametrize("kind", ["mul1", "mcg"])
@pytest.mark.parametrize("sizes,K,N", [([1], 128, 128), ([15, 0, 16, 17], 256, 384), ([64, 65, 3, 128, 129, 300], 1024, 256),
                                       ([7] * 200, 128, 640), ([40, 90, 20], 2048, 1280)])
def test_plain_product(sizes, K, N, kind):
    cu, w, ids, tiles, ntile, max_tiles, g = _setup(sizes, K, N, kind)
    x = torch.randn(len(ids), K, device=DEV, generator=g).half()
    y = cu.exl3_tc(x, w, tiles, ntile, max_tiles, out_f32=True)
    yb = cu.exl3_tc(x, w, tiles, ntile, max_tiles)
    assert torch.equal(y, cu.exl3_tc(x, w, tiles, ntile, max_tiles, out_f32=True))
    assert cu.read_status(torch.device(DEV))[0] == 0
    for e in ids.unique().tolist():
        r = ids == e
        ref = _product(x[r], w, e)
        err = ((y[r].double() - ref).norm() / ref.norm()).item()
        assert err < (K + 128) * 2.0 ** -23, (e, err)         # one rounding of a 32-bit sum per term
        assert torch.equal(y[r].bfloat16(), yb[r])


@pytest.mark.parametrize("sizes,K,F,limit", [([1, 0, 33], 128, 128, 0.0), ([64, 65, 16, 128, 200], 1024, 384, 1.0), ([5] * 70, 256, 256, 0.0)])
def test_gated_product(sizes, K, F, limit):
    cu, w, ids, tiles, ntile, max_tiles, g = _setup(sizes, K, 2 * F, "mul1")
    wd = Q.random_exl3(128, F, 4, len(sizes), 0.05, 9, DEV)
    x = torch.randn(len(ids), K, device=DEV, generator=g).half()
    y = cu.exl3_tc(x, w, tiles, ntile, max_tiles, glu=wd, limit=limit)
    assert torch.equal(y, cu.exl3_tc(x, w, tiles, ntile, max_tiles, glu=wd, limit=limit))
    assert cu.read_status(torch.device(DEV))[0] == 0
    for e in ids.unique().tolist():
        r = ids == e
        gu = _product(x[r], w, e)
        a, u = gu.chunk(2, -1)
        if limit:
            a, u = a.clamp(max=limit), u.clamp(-limit, limit)
        ref = _had(torch.nn.functional.silu(a) * u * wd.suh[e].double())
        err = ((y[r].double() - ref).norm() / ref.norm()).item()
        assert err < 2.0 ** -7.5, (e, err)                    # three bf16 roundings (2^-9 each) and one fp16


def test_gathered_input_rows():
    from spark_engine_b200.ops import cuda as cu
    g = torch.Generator(device=DEV).manual_seed(3)
    R, k, C, E = 37, 3, 384, 5
    x = torch.randn(R, C, device=DEV, generator=g).bfloat16()
    w = Q.random_exl3(128, C, 4, E, 0.05, 2, DEV)
    ids = torch.randint(-1, E, (R, k), device=DEV, generator=g, dtype=torch.int32)          # -1: an expert of another rank
    perm = torch.randperm(R * k, device=DEV, generator=g).to(torch.int32)
    y = cu.exl3_had_gather(x, w.suh, perm, ids, C)
    e = ids.view(-1)[perm.long()].clamp_min(0).long()
    ref = _had(x[perm.long() // k].double() * w.suh[e].double())
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -11                      # fp16 rounding of the result


def test_trellis_on_any_word():
    """Experts whose packed words start on 4 bytes only (a view of a larger buffer) give the bits of ones on 16."""
    cu, w, ids, tiles, ntile, max_tiles, g = _setup([17, 40], 256, 384, "mul1")
    x = torch.randn(len(ids), 256, device=DEV, generator=g).half()
    y = cu.exl3_tc(x, w, tiles, ntile, max_tiles)
    buf = torch.empty(w.trellis.numel() + 2, dtype=w.trellis.dtype, device=DEV)
    moved = Q.Exl3Weight(buf[2:].view(w.trellis.shape).copy_(w.trellis), w.suh, w.svh, 4, w.kind)
    assert torch.equal(cu.exl3_tc(x, moved, tiles, ntile, max_tiles), y)


@pytest.mark.parametrize("R,dtype", [(96, torch.float32), (97, torch.bfloat16)])
@pytest.mark.parametrize("local", [8, 4])
def test_down_rows_on_both_sides_of_the_format(R, dtype, local):
    """The down rows are fp32 up to 48 pairs per expert of the model (8 experts, top 4: 96 rows), on a rank that holds half of the
    experts as on one that holds all; either way they are the products of their experts."""
    from spark_engine_b200.config import MoeConfig
    from spark_engine_b200.ops import exl3_moe
    from spark_engine_b200.ops import cuda as cu
    g = torch.Generator(device=DEV).manual_seed(R)
    E, k, H, F = 8, 4, 256, 128
    c = MoeConfig(n_experts=E, top_k=k, ffn=F)
    wgu, wd = Q.random_exl3(2 * F, H, 4, local, 0.05, 1, DEV), Q.random_exl3(H, F, 4, local, 0.05, 2, DEV)
    h = torch.randn(R, H, device=DEV, generator=g).bfloat16()
    ids = torch.rand(R, E, device=DEV, generator=g).topk(k, -1).indices.int()
    ids = torch.where(ids < local, ids, -1)                        # the others live on another rank
    perm, inv, offs, tiles, ntile, max_tiles = cu.moe_sort(ids.view(-1), local)
    y = exl3_moe.exl3_grouped_experts(h, wgu, wd, ids, perm, tiles, ntile, max_tiles, c)
    assert y.dtype == dtype and cu.read_status(torch.device(DEV))[0] == 0
    for e in range(local):
        pairs = (ids.view(-1) == e).nonzero()[:, 0]
        x = _had(h[pairs // k].double() * wgu.suh[e].double()).half()
        a, u = _product(x, wgu, e).chunk(2, -1)
        z = _had(torch.nn.functional.silu(a) * u * wd.suh[e].double())
        ref = _product(z, wd, e)
        err = ((y[inv[pairs].long()].double() - ref).norm() / ref.norm()).item()
        assert err < 2.0 ** -7.5, (e, err)                        # roundings of the gated rows (three in bf16, one in fp16) and of the result
