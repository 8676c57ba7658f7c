"""Every CUDA kernel against a plain PyTorch fp32 reference of the same op (small shapes), plus
run-twice bitwise determinism where the kernel promises it."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from spark_engine_b200 import ops
from spark_engine_b200.config import MoeConfig
from spark_engine_b200.quant import formats as Q

DEV = "cuda"


def cu():
    return ops.cuda_ops()


def _status_ok():
    st = cu().read_status(torch.device(DEV))
    assert st[0] == 0, f"device status {st}"


def rel_err(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


# ------------------------------------------------------------------------------ tcgen05 GEMM
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 128, 128), (300, 520, 1000), (1, 256, 512), (257, 96, 72),
                                   (1024, 2048, 2048)])
@pytest.mark.parametrize("out_f32", [False, True])
def test_gemm_tcgen05_matches_fp32_matmul(M, N, K, out_f32):
    g = torch.Generator(device=DEV).manual_seed(1)
    a = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    b = torch.randn(N, K, device=DEV, generator=g).bfloat16()
    c = cu().gemm_bf16(a, b, out_f32=out_f32)
    torch.cuda.synchronize()
    _status_ok()
    ref = a.float() @ b.float().t()
    assert rel_err(c, ref) < (2e-5 if out_f32 else 6e-3)
    c2 = cu().gemm_bf16(a, b, out_f32=out_f32)
    assert torch.equal(c, c2)


def test_gemm_tcgen05_fp16_operands():
    g = torch.Generator(device=DEV).manual_seed(2)
    a = torch.randn(200, 256, device=DEV, generator=g).half()
    b = torch.randn(384, 256, device=DEV, generator=g).half()
    c = cu().gemm_bf16(a, b, out_f32=True, fmt=0)
    _status_ok()
    assert rel_err(c, a.float() @ b.float().t()) < 2e-5


def test_gemm_swiglu_epilogue():
    g = torch.Generator(device=DEV).manual_seed(3)
    M, F, K = 200, 256, 512
    a = (torch.randn(M, K, device=DEV, generator=g) * 0.5).bfloat16()
    b = (torch.randn(2 * F, K, device=DEV, generator=g) * 0.1).bfloat16()
    out = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    rc = cu().lib().spark_gemm_bf16_swiglu(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, F, K, K, K, F, 0.0,
                                           cu().status_word(a.device).data_ptr(), cu().stream())
    assert rc == 0
    gu = a.float() @ b.float().t()
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    _status_ok()
    assert rel_err(out, ref) < 8e-3


# ------------------------------------------------------------------------------ GEMV
@pytest.mark.parametrize("R", [1, 3, 8, 16])
@pytest.mark.parametrize("N,K", [(64, 256), (513, 2048), (2048, 4096)])
def test_gemv_bf16(R, N, K):
    g = torch.Generator(device=DEV).manual_seed(4)
    x = torch.randn(R, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(N, K, device=DEV, generator=g) * 0.05).bfloat16()
    y = cu().gemv_bf16(x, w, out_f32=True)
    ref = x.float() @ w.float().t()
    assert rel_err(y, ref) < 1e-5
    # batch invariance: row 0 alone gives the same bits
    y1 = cu().gemv_bf16(x[:1].contiguous(), w, out_f32=True)
    assert torch.equal(y1[0], y[0])


def test_gemv_pairs_with_swiglu_staging():
    g = torch.Generator(device=DEV).manual_seed(5)
    E, F, H, Pn = 6, 128, 256, 10
    wd = (torch.randn(E, H, F, device=DEV, generator=g) * 0.05).bfloat16()
    gu = torch.randn(Pn, 2 * F, device=DEV, generator=g).bfloat16()
    pe = torch.randint(0, E, (Pn,), device=DEV, generator=g).int()
    y = cu().gemv_bf16(gu, wd, items=Pn, rows_per_item=1, pair_expert=pe, act=1, out_f32=True, expert_stride=H * F, n=H, k=F)
    act = (torch.nn.functional.silu(gu[:, :F].float()) * gu[:, F:].float()).bfloat16().float()
    ref = torch.stack([act[i] @ wd[pe[i]].float().t() for i in range(Pn)])
    assert rel_err(y, ref) < 1e-4


# ------------------------------------------------------------------------------ elementwise
def test_add_rmsnorm_and_friends():
    g = torch.Generator(device=DEV).manual_seed(6)
    R, H = 5, 2048
    res = torch.randn(R, H, device=DEV, generator=g)
    delta = torch.randn(R, H, device=DEV, generator=g).bfloat16()
    w = torch.rand(H, device=DEV, generator=g) + 0.5
    ref_res = res + delta.float()
    ref = ref_res * torch.rsqrt(ref_res.pow(2).mean(-1, keepdim=True) + 1e-6) * w
    out, res2 = cu().add_rmsnorm(delta, res.clone(), w, 1e-6)
    assert torch.allclose(res2, ref_res, atol=1e-6)
    assert rel_err(out, ref) < 4e-3
    sw = cu().swiglu(delta, 0.0)
    F = H // 2
    assert rel_err(sw, torch.nn.functional.silu(delta[:, :F].float()) * delta[:, F:].float()) < 5e-3
    logits = torch.randn(4, 4099, device=DEV, generator=g)
    logits[1, 7] = logits[1, 4000] = 100.0      # tie -> lowest index
    ids = cu().argmax(logits)
    assert ids.tolist() == [int(torch.argmax(logits[0])), 7, int(torch.argmax(logits[2])), int(torch.argmax(logits[3]))]


def test_moe_route_kinds_match_reference():
    g = torch.Generator(device=DEV).manual_seed(7)
    for kind, E, k in (("softmax", 512, 10), ("sigmoid_bias", 288, 8), ("sqrt_softplus", 384, 6)):
        c = MoeConfig(n_experts=E, top_k=k, router=kind, route_scale=2.5 if kind != "softmax" else 1.0,
                      shared_gate=(kind == "softmax"))
        H = 256
        w = {"gate": (torch.randn(E + (1 if c.shared_gate else 0), H, device=DEV, generator=g) * 0.1).bfloat16(),
             "bias": torch.randn(E, device=DEV, generator=g) * 0.01}
        h = torch.randn(7, H, device=DEV, generator=g).bfloat16()
        wts, ids, prow, sg = cu().moe_route(h, w, c)
        wf = {"gate": w["gate"].float(), "bias": w["bias"]}
        rw, ri, rsg = ops.route(h.float().cpu(), {k: v.cpu() for k, v in wf.items()}, c)   # fp32 reference on CPU
        rw, ri = rw.to(DEV), ri.to(DEV)
        rsg = rsg.to(DEV) if rsg is not None else None
        assert torch.equal(ids.long().sort(-1).values, ri.sort(-1).values), kind
        order = torch.argsort(ids.long(), -1)
        rorder = torch.argsort(ri, -1)
        assert torch.allclose(torch.gather(wts, 1, order), torch.gather(rw, 1, rorder), rtol=2e-3, atol=1e-5), kind
        if sg is not None:
            assert torch.allclose(sg, rsg[:, 0], rtol=2e-3, atol=1e-4)


# ------------------------------------------------------------------------------ EXL3
@pytest.mark.parametrize("kind", ["mul1", "mcg"])
def test_exl3_reconstruct_is_bit_exact(kind):
    w = Q.random_exl3(256, 384, bits=4, seed=3, kind=kind)
    ref = Q.exl3_inner(w.trellis, kind)                     # [K, N]
    got = cu().exl3_reconstruct(w.to(DEV)).float().cpu()    # [N, K]
    assert torch.equal(got, ref.t())


@pytest.mark.parametrize("bits", [2, 3, 5, 6, 8])
@pytest.mark.parametrize("kind", ["mul1", "mcg"])
def test_exl3_reconstruct_other_bit_widths_is_bit_exact(bits, kind):
    """Checkpoints mix 3 to 6 bits per tensor: the window extraction for any width against the codec, single tensors
    and an expert stack."""
    w = Q.random_exl3(256, 384, bits=bits, seed=3 + bits, kind=kind)
    assert w.trellis.shape[-1] == 16 * bits
    got = cu().exl3_reconstruct(w.to(DEV)).float().cpu()
    assert torch.equal(got, Q.exl3_inner(w.trellis, kind).t())
    we = Q.random_exl3(128, 256, bits=bits, experts=3, seed=bits, kind=kind)
    gote = cu().exl3_reconstruct(we.to(DEV)).float().cpu()
    for e in range(3):
        assert torch.equal(gote[e], Q.exl3_inner(we.trellis[e], kind).t())


@pytest.mark.parametrize("bits", [3, 6])
@pytest.mark.parametrize("R", [2, 40])
def test_exl3_linear_other_bit_widths(bits, R):
    """Decode rows and prefill rows through a 3- and a 6-bit tensor (Hadamard rows, decoded inner weights, tcgen05 GEMM)."""
    from spark_engine_b200 import ops
    w = Q.random_exl3(512, 1024, bits=bits, seed=11, std=0.05)
    g = torch.Generator(device=DEV).manual_seed(8)
    x = torch.randn(R, 1024, device=DEV, generator=g).bfloat16()
    wd = w.to(DEV)
    y = ops.linear(x, wd).float().cpu()
    ref = x.float().cpu() @ w.dequant().t()
    assert rel_err(y, ref) < 6e-3
    assert torch.equal(ops.linear(x, wd), ops.linear(x, wd))


@pytest.mark.parametrize("bits", [4, 6])
def test_exl3_fold_to_dense_matches_the_codec(bits):
    """Inner weights + both Hadamard / scale sides folded into one dense bf16 matrix on the device."""
    w = Q.random_exl3(384, 256, bits=bits, seed=21, std=0.05)
    got = cu().exl3_fold(w.to(DEV)).float().cpu()            # [N, K]
    ref = w.dequant()                                         # [N, K]
    assert got.shape == ref.shape == (384, 256)
    assert rel_err(got, ref) < 8e-3                           # two bf16 roundings


@pytest.mark.parametrize("R", [1, 4, 16])
@pytest.mark.parametrize("N,K", [(256, 512), (1024, 2048), (2048, 512)])
def test_exl3_gemv_matches_dequant_matmul(R, N, K):
    w = Q.random_exl3(N, K, bits=4, seed=5, std=0.05)
    g = torch.Generator(device=DEV).manual_seed(8)
    x = torch.randn(R, K, device=DEV, generator=g).bfloat16()
    y = cu().exl3_gemv(x, w.to(DEV), out_f32=True)
    ref = x.float().cpu() @ w.dequant().t()
    assert rel_err(y.cpu(), ref) < 3e-3
    y2 = cu().exl3_gemv(x, w.to(DEV), out_f32=True)
    assert torch.equal(y, y2)
    y1 = cu().exl3_gemv(x[:1].contiguous(), w.to(DEV), out_f32=True)
    assert torch.equal(y1[0], y[0])                           # batch-invariant


def test_exl3_gemm_path_matches_dequant_matmul():
    N, K, M = 512, 1024, 200
    w = Q.random_exl3(N, K, bits=4, seed=6, std=0.05)
    g = torch.Generator(device=DEV).manual_seed(9)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    y = cu().exl3_linear(x, w.to(DEV))
    _status_ok()
    ref = x.float().cpu() @ w.dequant().t()
    assert rel_err(y.cpu(), ref) < 8e-3


def test_exl3_moe_pairs():
    E, F, H = 8, 128, 256
    wgu = Q.random_exl3(2 * F, H, bits=4, experts=E, seed=10, std=0.05)
    g = torch.Generator(device=DEV).manual_seed(10)
    x = torch.randn(3, H, device=DEV, generator=g).bfloat16()
    pe = torch.tensor([1, 5, 5, 0, 7, 2], dtype=torch.int32, device=DEV)
    pr = torch.tensor([0, 0, 1, 1, 2, 2], dtype=torch.int32, device=DEV)
    y = cu().exl3_gemv(x, wgu.to(DEV), items=6, rows_per_item=1, pair_expert=pe, pair_row=pr, out_f32=True)
    ref = torch.stack([x[pr[i]].float().cpu() @ wgu.dequant_expert(int(pe[i])).t() for i in range(6)])
    assert rel_err(y.cpu(), ref) < 3e-3


# ------------------------------------------------------------------------------ gated-DeltaNet chunked prefill
@pytest.mark.parametrize("lens", [[64], [200], [1024], [130, 77]])
def test_gdn_chunked_prefill_matches_sequential_kernel(lens):
    """The chunked (WY-form, tf32 tensor-core) prefill against the sequential fp32 kernel on the same projections:
    outputs, final state and conv history, from a non-zero starting state."""
    import dataclasses
    from spark_engine_b200.config import ModelConfig, GdnConfig
    from spark_engine_b200.models.model import GdnMixer
    from spark_engine_b200.models.plan import make_plan
    cfg = dataclasses.replace(ModelConfig(), gdn=GdnConfig(n_k_heads=2, n_v_heads=4, head_dim=128))
    c = cfg.gdn
    g = torch.Generator(device=DEV).manual_seed(11)
    nq, nv = c.n_k_heads * c.head_dim, c.n_v_heads * c.head_dim
    w = {"conv": (torch.rand(2 * nq + nv, c.conv_k, device=DEV, generator=g) - 0.5),
         "A_log": torch.log(torch.rand(c.n_v_heads, device=DEV, generator=g) * 7 + 1),
         "dt_bias": torch.rand(c.n_v_heads, device=DEV, generator=g) * 2 - 1,
         "norm": torch.rand(c.head_dim, device=DEV, generator=g) + 0.5}
    R = sum(lens)
    proj = torch.randn(R, 2 * nq + 2 * nv, device=DEV, generator=g).bfloat16()
    ab = torch.randn(R, 2 * c.n_v_heads, device=DEV, generator=g).bfloat16()
    plan = make_plan([(s, [1] * n, 5) for s, n in enumerate(lens)], device=DEV)
    mods = []
    for chunked in (False, True):
        m = GdnMixer(cfg, w, len(lens), DEV, torch.bfloat16)
        gs = torch.Generator(device=DEV).manual_seed(12)
        m.S.copy_(torch.randn(m.S.shape, device=DEV, generator=gs) * 0.1)
        m.tail.copy_(torch.randn(m.tail.shape, device=DEV, generator=gs))
        cu().GDN_CHUNKED = chunked
        try:
            out = cu().gdn_mixer(m, proj, ab, plan, True)
        finally:
            cu().GDN_CHUNKED = True
        torch.cuda.synchronize()
        mods.append((out.float(), m.S.clone(), m.tail.clone()))
    (o0, S0, t0), (o1, S1, t1) = mods
    assert torch.isfinite(o1).all() and torch.isfinite(S1).all()
    assert rel_err(o1, o0) < 1e-2, rel_err(o1, o0)
    assert rel_err(S1, S0) < 5e-3, rel_err(S1, S0)
    assert torch.equal(t1, t0)
    # worst single row stays close as well (no drift along the sequence)
    row_err = (o1 - o0).norm(dim=1) / o0.norm(dim=1).clamp_min(1e-6)
    assert row_err.max() < 3e-2, row_err.max()


def _gdn_both_forms(rows, eps=1e-6, fill=None, S0=True):
    """(outputs, states) of the sequential and of the chunked form for one segment of `rows` random rows; fill(proj, w, nq) edits the
    projections (columns q | k | v | z) and the weights."""
    import dataclasses
    from spark_engine_b200.config import ModelConfig, GdnConfig
    from spark_engine_b200.models.model import GdnMixer
    from spark_engine_b200.models.plan import make_plan
    cfg = dataclasses.replace(ModelConfig(), gdn=GdnConfig(n_k_heads=1, n_v_heads=2, head_dim=128), norm_eps=eps)
    c = cfg.gdn
    g = torch.Generator(device=DEV).manual_seed(13)
    nq, nv = c.n_k_heads * c.head_dim, c.n_v_heads * c.head_dim
    w = {"conv": (torch.rand(2 * nq + nv, c.conv_k, device=DEV, generator=g) - 0.5),
         "A_log": torch.log(torch.rand(c.n_v_heads, device=DEV, generator=g) * 7 + 1),
         "dt_bias": torch.rand(c.n_v_heads, device=DEV, generator=g) * 2 - 1,
         "norm": torch.rand(c.head_dim, device=DEV, generator=g) + 0.5}
    proj = torch.randn(rows, 2 * nq + 2 * nv, device=DEV, generator=g).bfloat16()
    ab = torch.randn(rows, 2 * c.n_v_heads, device=DEV, generator=g).bfloat16()
    if fill:
        fill(proj, ab, w, nq)
    plan = make_plan([(0, [1] * rows, 5)], device=DEV)
    outs = []
    for chunked in (False, True):
        m = GdnMixer(cfg, w, 1, DEV, torch.bfloat16)
        if S0:
            m.S.copy_(torch.randn(m.S.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(14)) * 0.1)
        cu().GDN_CHUNKED = chunked
        try:
            out = cu().gdn_mixer(m, proj, ab, plan, True)
        finally:
            cu().GDN_CHUNKED = True
        torch.cuda.synchronize()
        outs.append((out.double(), m.S.double()))
    return outs


@pytest.mark.parametrize("rows", [64, 200])
@pytest.mark.parametrize("noise", [0.0, 0.05, 0.5])
def test_gdn_chunked_correlated_keys(rows, noise):
    """Keys that are nearly the same, written with strength near 1 and hardly forgotten: I + A is close to a full triangle of ones,
    where the inverse lives on cancellation between its blocks."""
    def fill(proj, ab, w, nq):
        g = torch.Generator(device=DEV).manual_seed(17)
        base = torch.randn(1, 2 * nq, device=DEV, generator=g) + 1
        proj[:, : 2 * nq] = (base + noise * torch.randn(rows, 2 * nq, device=DEV, generator=g)).bfloat16()
        ab[:, :2] = 6.0
        w["A_log"].fill_(-6.0)
    (o0, S0), (o1, S1) = _gdn_both_forms(rows, fill=fill)
    assert rel_err(o1, o0) < 1e-2 and rel_err(S1, S0) < 5e-3


def test_gdn_chunked_history_on_any_float():
    """A history of earlier inputs that does not start on 16 bytes (views of a larger buffer) gives the bits of one that does."""
    import dataclasses
    from spark_engine_b200.config import ModelConfig, GdnConfig
    from spark_engine_b200.models.model import GdnMixer
    from spark_engine_b200.models.plan import make_plan
    cfg = dataclasses.replace(ModelConfig(), gdn=GdnConfig(n_k_heads=1, n_v_heads=2, head_dim=128))
    g = torch.Generator(device=DEV).manual_seed(15)
    w = {"conv": torch.rand(512, 4, device=DEV, generator=g) - 0.5, "A_log": torch.zeros(2, device=DEV), "dt_bias": torch.zeros(2, device=DEV),
         "norm": torch.ones(128, device=DEV)}
    proj = torch.randn(70, 768, device=DEV, generator=g).bfloat16()
    ab = torch.randn(70, 4, device=DEV, generator=g).bfloat16()
    outs = []
    for shift in (0, 1):
        m = GdnMixer(cfg, w, 1, DEV, torch.bfloat16)
        tail = torch.randn(m.tail.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(16))
        m.tail = torch.empty(tail.numel() + shift, device=DEV)[shift:].view(tail.shape).copy_(tail)
        outs.append((cu().gdn_mixer(m, proj, ab, make_plan([(0, [1] * 70, 5)], device=DEV), True), m.S, m.tail))
    assert all(torch.equal(a, b) for a, b in zip(*outs))


def test_gdn_chunked_silu_of_very_negative_values():
    """Values whose SiLU is near the smallest normal number (1 + e^87.5 is beyond what an approximate division takes) reach the state."""
    def fill(proj, ab, w, nq):
        w["conv"][2 * nq:] = torch.tensor([0.0, 0.0, 0.0, 1.0], device=DEV)
        proj[:, 2 * nq: 2 * nq + 256] = -87.5
    (_, S0), (_, S1) = _gdn_both_forms(64, fill=fill, S0=False)
    assert S0.norm() > 0
    # a term below the smallest normal number (1.2e-38 beside a state of about 1e-37) may count as 0
    assert ((S1 - S0).norm() / S0.norm()).item() < 0.1


def test_gdn_chunked_ragged_end_without_eps():
    """Rows past the end of the last chunk are zero rows; with eps 0 they have no norm to divide by."""
    (o0, S0), (o1, S1) = _gdn_both_forms(77, eps=0.0)
    assert torch.isfinite(o1).all() and torch.isfinite(S1).all()
    assert rel_err(o1, o0) < 1e-2 and rel_err(S1, S0) < 5e-3


# ------------------------------------------------------------------------------ KDA
@pytest.mark.parametrize("D", [32, 64, 128])
def test_kda_kernel_matches_torch_recurrence(D):
    """Conv + norms + per-channel-decay delta rule + gated RMS output in one launch against the same math in
    PyTorch fp32 (on the device), from a non-zero state; then a verify-without-commit followed by a commit of a prefix."""
    import dataclasses
    from spark_engine_b200.config import ModelConfig, KdaConfig
    from spark_engine_b200.models.model import KdaMixer
    from spark_engine_b200.models.plan import make_plan
    c = KdaConfig(n_heads=3, head_dim=D, gate_rank=16)
    cfg = dataclasses.replace(ModelConfig(), kda=c)
    n, r = c.n_heads * D, c.gate_rank
    g = torch.Generator(device=DEV).manual_seed(21)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    w = {"conv": torch.rand(3 * n, c.conv_k, device=DEV, generator=g) - 0.5, "f_b": rnd(n, r).bfloat16().float() * 0.3,
         "g_b": rnd(n, r).bfloat16().float() * 0.3, "A_log": torch.log(torch.rand(c.n_heads, device=DEV, generator=g) * 3 + 1),
         "dt_bias": torch.rand(n, device=DEV, generator=g) * 2 - 1, "o_norm": torch.rand(D, device=DEV, generator=g) + 0.5}
    T = 23
    pre = rnd(T, 3 * n).bfloat16()
    lr = rnd(T, 2 * r + c.n_heads).bfloat16()
    plan = make_plan([(0, [1] * T, 3)], device=DEV)
    m = KdaMixer(cfg, w, 1, DEV, torch.bfloat16)
    gs = torch.Generator(device=DEV).manual_seed(22)
    S0 = torch.randn(m.S.shape, device=DEV, generator=gs) * 0.1
    t0 = torch.randn(m.tail.shape, device=DEV, generator=gs)
    m.S.copy_(S0); m.tail.copy_(t0)
    o_ref, S_ref, tail_ref = m._seg(pre, lr, S0[0], t0[0])
    out = cu().kda_mixer(m, pre, lr, plan, True)
    torch.cuda.synchronize()
    assert rel_err(out, o_ref) < 1e-2
    assert rel_err(m.S[0], S_ref) < 1e-3
    assert torch.allclose(m.tail[0], tail_ref)
    # verify 13 rows without commit, then commit the first 9: equals a plain 9-row step (both row counts run the
    # batch-invariant GEMV for the gate projections, as verify and decode rounds do)
    pre, lr = pre[:13].contiguous(), lr[:13].contiguous()
    plan = make_plan([(0, [1] * 13, 3)], device=DEV)
    m.S.copy_(S0); m.tail.copy_(t0)
    cu().kda_mixer(m, pre, lr, plan, False)
    assert torch.equal(m.S, S0)
    cu().kda_commit(m, pre, lr, plan, [list(range(9))])
    m2 = KdaMixer(cfg, w, 1, DEV, torch.bfloat16)
    m2.S.copy_(S0); m2.tail.copy_(t0)
    cu().kda_mixer(m2, pre[:9].contiguous(), lr[:9].contiguous(), make_plan([(0, [1] * 9, 3)], device=DEV), True)
    assert torch.equal(m.S, m2.S) and torch.equal(m.tail, m2.tail)


@pytest.mark.parametrize("lens", [[64], [200], [1024], [130, 77]])
def test_kda_chunked_prefill_matches_sequential_kernel(lens):
    """The chunked (16-row chunks, per-channel decay, tf32 tensor-core) KDA prefill against the sequential fp32 kernel
    on the same projections: outputs, final state and conv history, from a non-zero starting state."""
    import dataclasses
    from spark_engine_b200.config import ModelConfig, KdaConfig
    from spark_engine_b200.models.model import KdaMixer
    from spark_engine_b200.models.plan import make_plan
    c = KdaConfig(n_heads=3, head_dim=128, gate_rank=16)
    cfg = dataclasses.replace(ModelConfig(), kda=c)
    n, r = c.n_heads * 128, c.gate_rank
    g = torch.Generator(device=DEV).manual_seed(31)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    w = {"conv": torch.rand(3 * n, c.conv_k, device=DEV, generator=g) - 0.5, "f_b": rnd(n, r).bfloat16().float() * 0.5,
         "g_b": rnd(n, r).bfloat16().float() * 0.3, "A_log": torch.log(torch.rand(c.n_heads, device=DEV, generator=g) * 3 + 1),
         "dt_bias": torch.rand(n, device=DEV, generator=g) * 2 - 1, "o_norm": torch.rand(128, device=DEV, generator=g) + 0.5}
    R = sum(lens)
    pre = rnd(R, 3 * n).bfloat16()
    lr = rnd(R, 2 * r + c.n_heads).bfloat16()
    plan = make_plan([(s, [1] * m, 5) for s, m in enumerate(lens)], device=DEV)
    res = []
    for chunked in (False, True):
        m = KdaMixer(cfg, w, len(lens), DEV, torch.bfloat16)
        gs = torch.Generator(device=DEV).manual_seed(32)
        m.S.copy_(torch.randn(m.S.shape, device=DEV, generator=gs) * 0.1)
        m.tail.copy_(torch.randn(m.tail.shape, device=DEV, generator=gs))
        cu().KDA_CHUNKED = chunked
        try:
            out = cu().kda_mixer(m, pre, lr, plan, True)
        finally:
            cu().KDA_CHUNKED = True
        torch.cuda.synchronize()
        res.append((out.float(), m.S.clone(), m.tail.clone()))
    (o0, S0, t0), (o1, S1, t1) = res
    assert torch.isfinite(o1).all() and torch.isfinite(S1).all()
    assert rel_err(o1, o0) < 1e-2, rel_err(o1, o0)
    assert rel_err(S1, S0) < 5e-3, rel_err(S1, S0)
    assert torch.equal(t1, t0)
    row_err = (o1 - o0).norm(dim=1) / o0.norm(dim=1).clamp_min(1e-6)
    assert row_err.max() < 3e-2, row_err.max()


def test_embedding_rejects_out_of_range_ids():
    """A token id outside the table never reaches memory: zero row + status word {bounds, row, id}."""
    table = torch.randn(100, 64, device=DEV).bfloat16()
    ids = torch.tensor([3, 100, 7, -1, 99], dtype=torch.int32, device=DEV)
    cu().reset_status(torch.device(DEV))
    out = cu().embed(table, ids)
    torch.cuda.synchronize()
    assert torch.equal(out[0], table[3].float()) and torch.equal(out[4], table[99].float())
    assert float(out[1].abs().sum()) == 0 and float(out[3].abs().sum()) == 0
    st = cu().read_status(torch.device(DEV))
    assert st[0] == 8 and st[1] in (1, 3)
    cu().reset_status(torch.device(DEV))


def test_mla_fp8_latent_rows_kernels_equal_generic_path():
    """FP8 latent cache rows (e4m3 codes + tile scales + bf16 rope): the prep kernel writes the same packed bytes as the
    torch packer, and decode over packed rows matches the masked-softmax path on the dequantised cache."""
    import dataclasses
    from spark_engine_b200.config import get_model_config, scaled_down
    from spark_engine_b200.models.model import Model, pack_latent_fp8, unpack_latent_fp8
    from spark_engine_b200.models.plan import make_plan
    from spark_engine_b200.models.weights import init_weights, to_device
    from spark_engine_b200.ops import cuda as cuo
    x = torch.randn(5, 256 + 64, device=DEV) * 3
    back = unpack_latent_fp8(pack_latent_fp8(x, 256), 256)
    assert rel_err(back[:, :256], x[:, :256]) < 4e-2 and rel_err(back[:, 256:], x[:, 256:]) < 4e-3
    cfg = scaled_down(get_model_config("glm-style"))
    cfg.mtp_layers = 0
    cfg.kv_dtype = "fp8"
    cfg.mla = dataclasses.replace(cfg.mla, kv_lora=256, rope_dim=32)
    W = to_device(init_weights(cfg, seed=0), DEV)
    g = torch.Generator().manual_seed(11)
    prompt = torch.randint(0, cfg.vocab, (150,), generator=g).tolist()
    outs, lats = [], []
    for kernels in (True, False):
        m = Model(cfg, W, device=DEV, dtype=torch.bfloat16, n_slots=1, kv_tokens=512)
        old = cuo.MLA_KERNELS
        cuo.MLA_KERNELS = kernels
        try:
            lg = [m.forward(make_plan([(0, prompt[:140], 0)], device=DEV, all_logits=False), commit=True).float()]
            lg.append(m.forward(make_plan([(0, prompt[140:144], 140)], device=DEV), commit=True).float())     # verify-style rows
            lg.append(m.forward(make_plan([(0, prompt[144:145], 144)], device=DEV), commit=True).float())
        finally:
            cuo.MLA_KERNELS = old
        outs.append(torch.cat(lg))
        mla = [mix for _, mix, _ in m.layers if hasattr(mix, "lat")]
        assert mla and mla[0].lat.dtype == torch.uint8 and mla[0].fp8
        lats.append(mla[0].lat[:145].clone())
    # the first latent layer sees identical inputs on both paths: packed bytes agree except for rounding ties
    same = (lats[0] == lats[1]).float().mean().item()
    assert same > 0.9, same
    assert rel_err(outs[0], outs[1]) < 4e-2


def _topk_reference(score, p, block, k, window):
    vis = (p + 1) // block
    if vis <= k:
        return list(range(p + 1))
    order = torch.sort(score[:vis].cpu(), descending=True, stable=True).indices[:k]
    taken = sorted(order.tolist())
    tail0 = vis * block
    lo = min(max(0, p + 1 - window), tail0) if window > 0 else tail0
    out = []
    for b in taken:
        out += [t for t in range(b * block, (b + 1) * block) if t < lo]
    return out + list(range(lo, p + 1))


@pytest.mark.parametrize("window", [0, 130])
def test_topk_select_multi_cta_equals_single_cta_and_reference(window):
    """Exact top-k over 70K candidates per row: one CTA per row, 18 CTAs per row (three digit passes over global
    histograms, per-slice counts, ordered emission) and a stable sort agree element for element, ties included."""
    from spark_engine_b200.ops import sparse as sp
    g = torch.Generator(device=DEV).manual_seed(21)
    block, k, nb = 4, 512, 70000
    pos = torch.tensor([nb * block - 1, 250001, 1999, 279998], dtype=torch.int32, device=DEV)
    R = pos.shape[0]
    score = torch.randn(R, nb, device=DEV, generator=g)
    score[0] = torch.randint(0, 40, (nb,), device=DEV, generator=g).float() / 8          # heavy ties, also at the threshold
    score[3] = torch.relu(score[3])                                                       # half the keys are +0
    score[3, ::3] = -0.0
    one, one_n = sp.topk_select(score, nb, pos, block, k, window, ctas=1)
    many, many_n = sp.topk_select(score, nb, pos, block, k, window, ctas=18)
    auto, auto_n = sp.topk_select(score, nb, pos, block, k, window)
    torch.cuda.synchronize()
    assert torch.equal(one_n, many_n) and torch.equal(one_n, auto_n)
    for r in range(R):
        n = int(one_n[r])
        ref = _topk_reference(score[r], int(pos[r]), block, k, window)
        assert n == len(ref), (r, n, len(ref))
        assert one[r, :n].tolist() == ref, r
        assert many[r, :n].tolist() == ref, r
        assert auto[r, :n].tolist() == ref, r


@pytest.mark.parametrize("H,Dm,weighted", [(4, 128, False), (32, 128, True), (2, 32, True), (16, 64, False)])
def test_indexer_scores_on_tensor_cores_equal_the_per_row_kernel(H, Dm, weighted):
    """Prefill rows scored as (row, head) x pooled-key tiles with 3xTF32 MMAs against the fp32 per-row kernel: two ragged
    segments at different offsets of their sequences, with and without per-head weights; the selections agree."""
    from spark_engine_b200.models.plan import make_plan
    from spark_engine_b200.ops import sparse as sp
    g = torch.Generator(device=DEV).manual_seed(31)
    block, topk = 4, 16
    n0, n1, p0, p1 = 150, 77, 260, 0
    plan = make_plan([(0, [1] * n0, p0), (1, [1] * n1, p1)], device=DEV)
    d = plan.dev
    R = n0 + n1
    cap = 1024                                                    # tokens per sequence
    row_kv = torch.tensor([0] * n0 + [cap] * n1, dtype=torch.int64, device=DEV)
    pool = torch.randn(2 * cap // block + 2, Dm, device=DEV, generator=g)
    qi = torch.randn(R, H, Dm, device=DEV, generator=g)
    hw = torch.rand(R, H, device=DEV, generator=g) if weighted else None
    max_ctx = p0 + n0
    outs = []
    for segs in (None, (d["seg"], 2, max(n0, n1))):
        sel, sel_n = sp.select_tokens(qi, pool, row_kv, d["pos32"], block, topk, max_ctx, head_w=hw, window=8, segs=segs)
        nb_max = max_ctx // block
        score = cu().scratch("idx_score", R * nb_max, torch.float32, torch.device(DEV))[: R * nb_max].view(R, nb_max).clone()
        outs.append((sel.clone(), sel_n.clone(), score))
    vis = ((d["pos32"] + 1) // block).long()
    live = torch.arange(outs[0][2].shape[1], device=DEV).unsqueeze(0) < vis.unsqueeze(1)
    a, b = outs[0][2][live], outs[1][2][live]
    assert torch.isfinite(b).all()
    assert (a - b).abs().max().item() <= 2e-5 * a.abs().max().item()
    assert torch.equal(outs[0][1], outs[1][1])
    same = sum(int(torch.equal(outs[0][0][r, : int(outs[0][1][r])], outs[1][0][r, : int(outs[1][1][r])])) for r in range(R))
    assert same >= R - 2, same            # a near-tie at the threshold may pick the other block
