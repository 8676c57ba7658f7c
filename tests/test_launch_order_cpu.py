"""What kernels may read before their dependency wait: tables that are at least two launches old (shown on the CPU, launches recorded)."""
import os
import re
from types import SimpleNamespace

import pytest
import torch

from spark_engine_b200 import build
from spark_engine_b200.models.plan import make_plan
from spark_engine_b200.ops import cuda as cu


def _record(monkeypatch):
    log = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: log.append((name, a)) or 0
    monkeypatch.setattr(cu, "lib", lambda: Lib())
    monkeypatch.setattr(cu, "stream", lambda: 0)
    return log


def test_head_table_of_latent_attention_is_two_launches_old(monkeypatch):
    log = _record(monkeypatch)
    H, D, L, Rr, R, hidden = 4, 16, 32, 8, 2, 24
    c = SimpleNamespace(n_heads=H, head_dim=D, kv_lora=L, rope_dim=Rr, q_lora=16, idx_dim=8, idx_heads=2, pool=4, topk_pools=8, window=0,
                        rope_theta=1e4, sink=False)
    width = c.q_lora + L + Rr + 2 * c.idx_dim + c.idx_heads
    f = torch.zeros
    w = {"a": f(width, hidden), "q_b": f(H * (D + Rr) + c.idx_heads * c.idx_dim, c.q_lora), "ape": f(4, 8), "q_a_norm": f(16), "kv_a_norm": f(L),
         "k_ln_w": f(8), "k_ln_b": f(8)}
    mixer = SimpleNamespace(c=c, w=w, cfg=SimpleNamespace(norm_eps=1e-6), fp8=False, w_uk=f(H, D, L), w_uv=f(H, D, L), lat=f(64, L + Rr), ik=f(64, 8),
                            ig=f(64, 8), pool=f(18, 8))
    monkeypatch.setattr(cu, "linear_any", lambda x, m: log.append(("linear", ())) or f(x.shape[0], m.shape[0], dtype=torch.bfloat16))
    made = {}
    arange = torch.arange

    def logged(*a, **k):
        t = arange(*a, **k)
        made[t.data_ptr()] = (len(log), t)
        return t
    monkeypatch.setattr(torch, "arange", logged)
    plan = make_plan([(0, [1, 2], 0)])
    seqs = [SimpleNamespace(kv_base=0, kv_cap=64)]
    cu.mla_mixer(mixer, f(R, hidden, dtype=torch.bfloat16), plan, seqs)
    items = [(i, a) for i, (name, a) in enumerate(log) if name == "spark_gemv_bf16_items"]
    assert len(items) == 2
    for i, a in items:
        table, early = a[13], a[-1]
        at, t = made[table]
        assert torch.equal(t, arange(H, dtype=torch.int32))
        assert not early or i - at >= 2, (i, at)


@pytest.mark.parametrize("source,kernel", [("gemv.cu", "gemv_bf16_kernel"), ("gemv.cu", "gemv_wide_mma_kernel"), ("gemv.cu", "gemv_long_mma_kernel"),
                                           ("mx.cu", "mx_gemv_kernel")])
def test_single_matrices_are_asked_for_after_the_dependency_wait(source, kernel):
    """Their weights may come from the launch directly before (expansions on first use), and no argument says otherwise."""
    with open(os.path.join(build.CSRC, "kernels", source)) as f:
        body = f.read().split(f"\n{kernel}(", 1)[1].split("\n}\n", 1)[0]
    wait = re.search(r"^  pdl_wait\(\);", body, re.M)
    first = re.search(r"^  (?!auto)[^/\n]*\bload\(", body, re.M) or re.search(r"__ldg\(", body)
    assert wait and first and wait.start() < first.start()
