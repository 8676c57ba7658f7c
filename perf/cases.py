"""The engine's layer work at the sizes its presets serve, one sublayer per case.

A decoder layer is two sublayers, each followed by the residual update with the next norm.  A case is one sublayer of one of
the large presets, with that update, on rows of a round:

  moe   router, routed experts (EXL3 4 bpw or MXFP4) and shared expert, combined
  gdn   gated DeltaNet: EXL3 projections, short convolution, delta rule, gated norm; the slots' states advance
  attn  grouped-query attention behind its projection: norms, rotation, cache write, block selection, softmax, EXL3 output
  mla   latent attention: low-rank projections, packed FP8 cache rows, indexer, absorbed attention, MXFP8 output

Rounds of up to 16 rows (decode: one row per stream; verification: a stream's drafts) replay a captured CUDA graph, as the
serving loop does; longer ones (prompts) are called eagerly, as prefill is.
"""
import dataclasses
import math

import torch
import torch.nn.functional as F

from spark_engine_b200 import ops
from spark_engine_b200.config import get_model_config
from spark_engine_b200.models.build import build_random_model
from spark_engine_b200.models.model import Model
from spark_engine_b200.models.plan import make_plan
from spark_engine_b200.serving.graphs import ctx_bucket

GRAPH_ROWS = 16
PRESET = {"gdn": "qwen3next-style", "attn": "qwen3next-style", "mla": "ds4-style"}


def listed():
    return [
        # one interactive stream: the smallest call, launches and latency count
        {"name": "gdn-decode-1", "op": "gdn", "streams": 1, "rows": 1, "context": 200},
        # a prompt chunk through the linear-attention layers (three of four layers of that preset)
        {"name": "gdn-prompt-4096", "op": "gdn", "streams": 1, "rows": 4096, "context": 0},
        # four streams behind long prompts, FP8 cache, blocks selected
        {"name": "attn-decode-4-16k", "op": "attn", "streams": 4, "rows": 1, "context": 16001, "kv": "fp8"},
        # a prompt chunk of odd length; its later rows select blocks
        {"name": "attn-prompt-3999", "op": "attn", "streams": 1, "rows": 3999, "context": 0, "kv": "bf16"},
        # four streams of latent attention
        {"name": "mla-decode-4-1500", "op": "mla", "streams": 4, "rows": 1, "context": 1500, "kv": "fp8"},
        # the headline's decode round: four streams, ten experts each
        {"name": "moe-exl3-decode-4", "op": "moe", "preset": "qwen3next-style", "rows": 4},
        # a verification round: four streams, three drafts each
        {"name": "moe-exl3-verify-16", "op": "moe", "preset": "qwen3next-style", "rows": 16},
        # a prompt of about a thousand tokens (time to first token): some twenty rows per expert
        {"name": "moe-exl3-prompt-1021", "op": "moe", "preset": "qwen3next-style", "rows": 1021},
        # a full prefill chunk
        {"name": "moe-exl3-prompt-8192", "op": "moe", "preset": "qwen3next-style", "rows": 8192},
        # two streams of the preset with the widest EXL3 experts
        {"name": "moe-glm-decode-2", "op": "moe", "preset": "glm-style", "rows": 2},
        # four streams on MXFP4 experts
        {"name": "moe-mx-decode-4", "op": "moe", "preset": "ds4-style", "rows": 4},
        # a prompt on MXFP4 experts
        {"name": "moe-mx-prompt-2048", "op": "moe", "preset": "ds4-style", "rows": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["gdn", "attn", "mla", "moe", "moe", "moe"])
    if op == "moe":
        preset = rng.choice(["qwen3next-style", "qwen3next-style", "glm-style", "ds4-style"])
        if preset == "glm-style":
            return {"op": op, "preset": preset, "rows": _log(rng, 1, 16)}
        if rng.random() < 0.5:
            return {"op": op, "preset": preset, "rows": rng.randint(1, 16)}
        return {"op": op, "preset": preset, "rows": _log(rng, 100, 8192 if preset[0] == "q" else 2048)}
    if op == "mla":
        return {"op": op, "streams": rng.randint(1, 4), "rows": rng.randint(1, 4), "context": _log(rng, 100, 2000), "kv": "fp8"}
    if rng.random() < 0.5:
        case = {"op": op, "streams": rng.randint(1, 4), "rows": rng.randint(1, 4), "context": _log(rng, 100, 400 if op == "gdn" else 16000)}
    else:
        case = {"op": op, "streams": 1, "rows": _log(rng, 100, 4096), "context": 0}
    if op == "attn":
        case["kv"] = rng.choice(["bf16", "fp8"]) if case["rows"] <= 4 else "bf16"
    return case


def _config(case):
    """The preset with one layer, and in a mixer's case without its experts."""
    op = case["op"]
    cfg = get_model_config(case["preset"] if op == "moe" else PRESET[op], n_layers=1)
    cfg.vocab, cfg.mtp_layers, cfg.ngram_layers = 4096, 0, []
    if op == "moe":
        cfg.moe = dataclasses.replace(cfg.moe, dense_layers=0)
        if cfg.family == "ds4":             # the layer's mixer is not run
            cfg.layer_types, cfg.gdn = ["gdn"], dataclasses.replace(cfg.gdn, head_dim=128)
    else:
        cfg.layer_types = [op]
        cfg.moe = dataclasses.replace(cfg.moe, dense_layers=1, dense_ffn=128)
        cfg.kv_dtype = case.get("kv", "bf16")
    return cfg


def _inputs(case, seed):
    """(config, weights, earlier rows of every stream, the pass's rows, residual).  Rows of `attn` are projections."""
    cfg = _config(case)
    W = build_random_model(cfg, "cuda", seed=seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, ctx = case.get("streams", 1), case.get("context", 0)
    width = W["layers"][0]["mix"]["qkv"].n if case["op"] == "attn" else cfg.hidden
    past = [torch.randn(ctx, width, device="cuda", generator=g).to(torch.bfloat16) for _ in range(n)]
    h = torch.randn(n * case["rows"], width, device="cuda", generator=g).to(torch.bfloat16)
    X = torch.randn(n * case["rows"], cfg.hidden, device="cuda", generator=g) * 0.02
    return cfg, W, past, h, X


def _plan(model, items):
    p = make_plan(items, device=model.device)
    p.dev["row_kv"] = torch.tensor([model.seqs[s.slot].kv_base for s in p.segs for _ in range(s.n)], dtype=torch.int64, device=model.device)
    last = max(s.pos0 + s.n for s in p.segs)
    p.dev["max_ctx"] = ctx_bucket(last) if p.rows <= GRAPH_ROWS else last       # a captured round serves a bucket of contexts
    return p


def _sublayer(s, h, plan):
    mix, mlp = s["mix"], s["mlp"]
    if s["op"] == "moe":
        return mlp.forward(h, defer=h.shape[0] <= GRAPH_ROWS)
    if s["op"] == "attn":
        return ops.row_parallel(ops.attn_mixer(mix, h, plan, s["seqs"]), mix.w["o"])
    return mix.forward(h, plan, s["seqs"], True)


def _pass(s):
    h, X = ops.add_rmsnorm(_sublayer(s, s["h"], s["plan"]), s["X"], s["norm"], s["eps"])
    return {"h": h, "X": X, **s["updated"]}


def prepare(case, seed):
    cfg, W, past, h, X = _inputs(case, seed)
    n, rows, ctx = case.get("streams", 1), case["rows"], case.get("context", 0)
    per = (ctx + rows + 63) // 64 * 64
    model = Model(cfg, W, device="cuda", dtype=torch.bfloat16, n_slots=n, kv_tokens=n * per, slot_tokens=per)
    lw, mix, mlp = model.layers[0]
    s = {"op": case["op"], "model": model, "mix": mix, "mlp": mlp, "seqs": model.seqs, "h": h, "X": X, "norm": lw["post_norm"],
         "eps": cfg.norm_eps, "updated": {}, "plan": None}
    if case["op"] != "moe":
        s["plan"] = _plan(model, [(i, [0] * rows, ctx) for i in range(n)])
        if ctx:
            s["past"] = _plan(model, [(i, [0] * ctx, 0) for i in range(n)])
            _sublayer(s, torch.cat(past), s["past"])
        names = {"gdn": ("S", "tail"), "attn": ("k", "v"), "mla": ("ik", "ig")}[case["op"]]
        for name in names:
            t = getattr(mix, name)
            if case["op"] == "gdn":
                s["updated"][name] = t
            else:
                for i, q in enumerate(model.seqs[:n]):
                    s["updated"]["%s%d" % (name, i)] = t[q.kv_base + ctx: q.kv_base + ctx + rows]
    if n * rows <= GRAPH_ROWS:
        carried = [X] + ([mix.S, mix.tail] if case["op"] == "gdn" else [])
        before = [t.clone() for t in carried]
        _pass(s)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = _pass(s)
        for t, b in zip(carried, before):
            t.copy_(b)
    return s


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return _pass(state)


# --------------------------------------------------------------------------------------------------- work and tolerance
def _expert_bytes(cfg):
    return 3 * cfg.hidden * cfg.moe.ffn * (0.5 if cfg.weight_format == "exl3" else 0.5 + 1 / 32)


def work(case):
    cfg = _config(case)
    n, rows, ctx, H = case.get("streams", 1), case["rows"], case.get("context", 0), cfg.hidden
    R = n * rows
    io = R * H * (2 + 2 + 4 + 4)                                     # rows in and out, residual in and out
    if case["op"] == "moe":
        m = cfg.moe
        touched = m.n_experts * (1 - (1 - m.top_k / m.n_experts) ** R)
        gate = m.n_experts * H
        return {"bytes": io + 2 * gate + (touched + 1) * _expert_bytes(cfg), "flops": 2 * R * (gate + (m.top_k + 1) * 3 * H * m.ffn)}
    if case["op"] == "gdn":
        c = cfg.gdn
        D, nv = c.head_dim, c.n_v_heads
        w = (2 * c.n_k_heads + 3 * nv) * D * H
        return {"bytes": io + w // 2 + 2 * n * nv * D * D * 4, "flops": 2 * R * (w + 4 * nv * D * D)}
    keys = sum(min(ctx + j + 1, 2048) for j in range(rows)) * n       # of all rows; every sparse layer selects 2048
    if case["op"] == "attn":
        c = cfg.attn
        D, wide = c.head_dim, H * c.n_q_heads * c.head_dim
        cached = n * min(ctx + rows, 2048 * rows) * 2 * c.n_kv_heads * D * (1 if case["kv"] == "fp8" else 2)
        scored = n * (ctx + rows) // c.block * c.idx_dim * 4 if ctx + rows > 2048 else 0
        proj = 2 * (2 * c.n_q_heads * D + 2 * c.n_kv_heads * D + (c.idx_heads + 1) * c.idx_dim)
        return {"bytes": R * (H * 10 + proj) + wide // 2 + cached + scored, "flops": 2 * R * wide + 4 * keys * c.n_q_heads * D}
    c = cfg.mla
    a, b = c.q_lora + c.kv_lora + c.rope_dim + 2 * c.idx_dim + c.idx_heads, c.n_heads * (c.head_dim + c.rope_dim) + c.idx_heads * c.idx_dim
    dense, up, out = a * H + b * c.q_lora, 2 * c.n_heads * c.head_dim * c.kv_lora, H * c.n_heads * c.head_dim
    return {"bytes": io + 2 * (dense + up) + out + n * (ctx + rows) * 656,
            "flops": 2 * R * (dense + up + out) + 2 * keys * c.n_heads * (2 * c.kv_lora + c.rope_dim)}


def tolerance(case):
    """Four times the largest distance between `exact` and the device: 4e-3 where rows are bf16 in and between the products (EXL3);
    2e-2 to 5e-2 where rows or caches are quantised to 8 bits on the way, of which no more than 3e-2 is allowed."""
    op = case["op"]
    if op == "mla" or case.get("kv") == "fp8" or case.get("preset") == "ds4-style":
        return {"rel": 0.03, "max": 0.9}
    return {"rel": 0.016, "max": 0.5}


# --------------------------------------------------------------------------------------------------- the same in 64 bits
def _had(x):
    """128-point Hadamard transforms (orthonormal) along the last axis."""
    h = torch.ones(1, 1, dtype=torch.float64, device=x.device)
    while h.shape[0] < 128:
        h = torch.cat((torch.cat((h, h), 1), torch.cat((h, -h), 1)), 0)
    return (x.view(*x.shape[:-1], -1, 128) @ (h / 128 ** 0.5)).view(x.shape)


_codes = {}


def _exl3_values(trellis):
    """Code book values [K, N] of 4-bit tiles [K/16, N/16, 64]: position t of a tile holds the 16 bits that end 4 (t + 1) bits into
    its ring of 32-bit words, most significant first."""
    dev = trellis.device
    if "value" not in _codes:
        x = torch.arange(65536, device=dev) * 0x83DCD12D & 0xFFFFFFFF
        total = (x & 255) + (x >> 8 & 255) + (x >> 16 & 255) + (x >> 24)
        scale, shift = torch.tensor([0x1EEE, 0xC931 - 0x10000], dtype=torch.int16).view(torch.float16).double().tolist()
        _codes["value"] = ((1024 + total).double() * scale + shift).half().double()
        lane, j = torch.arange(256, device=dev) // 8, torch.arange(256, device=dev) % 8
        at = ((lane % 4) * 2 + j % 2 + j % 4 // 2 * 8) * 16 + lane // 4 + j // 4 * 8
        _codes["order"] = torch.argsort(at)
    Kt, Nt, _ = trellis.shape
    half = trellis.long() & 0xFFFF
    word = half[..., 0::2] | half[..., 1::2] << 16
    ring = word.roll(1, -1) << 32 | word                                                       # the word before and the word
    shift = torch.arange(28, -1, -4, device=dev)
    state = (ring.unsqueeze(-1) >> shift & 0xFFFF).flatten(-2)                               # [Kt, Nt, 256]
    v = _codes["value"][state[..., _codes["order"]]]
    return v.view(Kt, Nt, 16, 16).transpose(1, 2).reshape(Kt * 16, Nt * 16)


def _nibbles(packed, scales):
    grid = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=packed.device)
    v = grid[torch.stack((packed & 15, packed >> 4), -1).long()].flatten(-2)
    return (v.view(*scales.shape, 32) * torch.exp2(scales.double() - 127).unsqueeze(-1)).flatten(-2)


def _product(x, w, e=None):
    """x W^T in 64 bits for any weight format (`e`: of that expert of a stack)."""
    if isinstance(w, torch.Tensor):
        return x @ (w if e is None else w[e]).double().t()
    at = (lambda t: t) if e is None else (lambda t: t[e])
    if hasattr(w, "trellis"):
        return _had(_had(x * at(w.suh).double()) @ _exl3_values(at(w.trellis))) * at(w.svh).double()
    if hasattr(w, "packed"):
        return x @ _nibbles(at(w.packed), at(w.scales)).t()
    v = w.q.double().view(*w.scales.shape, 32) * torch.exp2(w.scales.double() - 127).unsqueeze(-1)
    return x @ v.flatten(-2).t()


def _rms(x, w=None, eps=1e-6):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _glu(gu, limit):
    g, u = gu.chunk(2, -1)
    if limit:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return F.silu(g) * u


def _exact_moe(cfg, w, h):
    c, x = cfg.moe, h.double()
    logits = x @ w["gate"].double().t()
    shared = torch.sigmoid(logits[:, c.n_experts:]) if c.shared_gate else 1.0
    logits = logits[:, : c.n_experts]
    p = {"softmax": lambda t: torch.softmax(t, -1), "sigmoid_bias": torch.sigmoid,
         "sqrt_softplus": lambda t: F.softplus(t).sqrt()}[c.router](logits)              # the presets' biases are zero
    top = torch.sort(p, descending=True, stable=True, dim=-1)
    ids, wts = top.indices[:, : c.top_k], top.values[:, : c.top_k]
    wts = wts / wts.sum(-1, keepdim=True) * c.route_scale
    out = torch.zeros_like(x)
    for e in ids.unique().tolist():
        r, slot = (ids == e).nonzero(as_tuple=True)
        y = _product(_glu(_product(x[r], w["w_gu"], e), c.swiglu_limit), w["w_down"], e)
        out.index_add_(0, r, y * wts[r, slot].unsqueeze(1))
    return out + shared * _product(_glu(_product(x, w["s_gu"]), c.swiglu_limit), w["s_down"])


def _exact_gdn(cfg, w, x, rows):
    """x: one stream's rows from its start.  Returns (the last `rows` outputs, state, last three rows in front of the convolution)."""
    c, T = cfg.gdn, x.shape[0]
    D, nk, nv = c.head_dim, c.n_k_heads, c.n_v_heads
    proj, ab = _product(x, w["in"]), _product(x, w["ab"])
    pre, z = proj.split([(2 * nk + nv) * D, nv * D], -1)
    conv = F.pad(pre, (0, 0, 3, 0)).unfold(0, 4, 1) * w["conv"].double()
    q, k, v = F.silu(conv.sum(-1)).split([nk * D, nk * D, nv * D], -1)
    unit = lambda t: (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + cfg.norm_eps)).repeat_interleave(nv // nk, 1)
    q, k, v = unit(q.view(T, nk, D)) * D ** -0.5, unit(k.view(T, nk, D)), v.view(T, nv, D)
    beta = torch.sigmoid(ab[:, :nv])
    decay = torch.exp(-torch.exp(w["A_log"].double()) * F.softplus(ab[:, nv:] + w["dt_bias"].double()))
    S, o = x.new_zeros(nv, D, D), x.new_empty(T, nv, D)
    for t in range(T):
        S.mul_(decay[t].view(nv, 1, 1))
        S.baddbmm_((beta[t].unsqueeze(1) * (v[t] - (S @ k[t].unsqueeze(2)).squeeze(2))).unsqueeze(2), k[t].unsqueeze(1))
        o[t] = (S @ q[t].unsqueeze(2)).squeeze(2)
    o = _rms(o, w["norm"].double(), cfg.norm_eps) * torch.sigmoid(z.view(T, nv, D))
    last = F.pad(pre, (0, 0, 3, 0))[-3:]
    spread = lambda t: t.view(3, nk, D).repeat_interleave(nv // nk, 1)
    tail = torch.cat((spread(last[:, : nk * D]), spread(last[:, nk * D: 2 * nk * D]), last[:, 2 * nk * D:].view(3, nv, D)), -1)
    return _product(o[-rows:].reshape(rows, nv * D), w["o"]), S, tail


def _turn(x, pos, inv):
    """Rotation of the first 2 len(inv) dimensions of x [T, heads, D], halves paired."""
    n = inv.shape[0]
    a = (pos.double().unsqueeze(1) * inv).unsqueeze(1)
    u, v = x[..., :n], x[..., n: 2 * n]
    return torch.cat((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., 2 * n:]), -1)


def _yarn(dim, theta, factor, length):
    i = torch.arange(dim // 2, dtype=torch.float64, device="cuda")
    inv = theta ** (-2 * i / dim)
    edge = lambda turns: dim * math.log(length / (turns * 2 * math.pi)) / (2 * math.log(theta))
    lo, hi = max(math.floor(edge(32.0)), 0), min(math.ceil(edge(1.0)), dim // 2 - 1)
    ramp = ((i - lo) / max(hi - lo, 1e-3)).clamp(0, 1)
    return inv / factor * ramp + inv * (1 - ramp)


def _visible(scores, first, T, block, top):
    """[rows, T] bool: the top blocks of the complete ones by score (all while there are no more than that), and what follows them.
    scores [rows, T // block] for queries at first, first + 1, ..."""
    rows = scores.shape[0]
    p = torch.arange(first, first + rows, device=scores.device)
    done = (p + 1) // block
    live = torch.arange(scores.shape[1], device=scores.device) < done.unsqueeze(1)
    order = torch.sort(scores.masked_fill(~live, -math.inf), dim=1, descending=True, stable=True).indices[:, :top]
    chosen = torch.zeros_like(live).scatter_(1, order, True) & live
    tok = torch.arange(T, device=scores.device)
    mask = (tok >= (done * block).unsqueeze(1)) & (tok <= p.unsqueeze(1))
    mask[:, : scores.shape[1] * block] |= chosen.repeat_interleave(block, 1)
    return mask


def _exact_attn(cfg, w, qkv, rows):
    c, T = cfg.attn, qkv.shape[0]
    D, nq, nkv, pos = c.head_dim, c.n_q_heads, c.n_kv_heads, torch.arange(T, device="cuda")
    inv = _yarn(c.rope_dim, c.rope_theta, c.yarn_factor, c.yarn_orig_len)
    norm = lambda t, name: _rms(t, 1 + w[name].double(), cfg.norm_eps)
    qg, k, v, qi, ki = qkv.double().split([nq * 2 * D, nkv * D, nkv * D, c.idx_heads * c.idx_dim, c.idx_dim], -1)
    qg = qg[-rows:].view(rows, nq, 2 * D)
    q = _turn(norm(qg[..., :D], "q_norm"), pos[-rows:], inv)
    k, v = _turn(norm(k.view(T, nkv, D), "k_norm"), pos, inv), v.view(T, nkv, D)
    nb = T // c.block
    pooled = ki[: nb * c.block].view(nb, c.block, c.idx_dim).mean(1, keepdim=True)
    kc = _turn(norm(pooled, "ik_norm"), pos[: nb * c.block: c.block], inv)[:, 0]
    qi = _turn(norm(qi[-rows:].view(rows, c.idx_heads, c.idx_dim), "iq_norm"), pos[-rows:], inv)
    score = sum(F.relu(qi[:, i] @ kc.t()) for i in range(c.idx_heads))
    hidden = ~_visible(score, T - rows, T, c.block, c.sparse_topk_blocks)
    o = torch.empty_like(q)
    for i in range(nq):
        j = i // (nq // nkv)
        o[:, i] = torch.softmax((q[:, i] @ k[:, j].t() * D ** -0.5).masked_fill_(hidden, -math.inf), -1) @ v[:, j]
    o = o * torch.sigmoid(qg[..., D:])
    return _product(o.reshape(rows, nq * D), w["o"]), k[-rows:], v[-rows:]


def _exact_mla(cfg, w, x, rows):
    c, T = cfg.mla, x.shape[0]
    H, D, L, Rr, pos = c.n_heads, c.head_dim, c.kv_lora, c.rope_dim, torch.arange(T, device="cuda")
    inv = c.rope_theta ** (-2 * torch.arange(Rr // 2, dtype=torch.float64, device="cuda") / Rr)
    cq, ckv, kr, ik, ig, hw = _product(x, w["a"]).split([c.q_lora, L, Rr, c.idx_dim, c.idx_dim, c.idx_heads], -1)
    q = _product(_rms(cq[-rows:], w["q_a_norm"].double(), cfg.norm_eps), w["q_b"])[:, : H * (D + Rr)].view(rows, H, D + Rr)
    ckv = _rms(ckv, w["kv_a_norm"].double(), cfg.norm_eps)
    up = w["kv_b"].double().view(H, 2 * D, L)
    key = torch.cat((ckv, _turn(kr.unsqueeze(1), pos, inv)[:, 0]), -1)
    ql = torch.cat((torch.einsum("thd,hdl->thl", q[..., :D], up[:, :D]), _turn(q[..., D:], pos[-rows:], inv)), -1)
    s = torch.einsum("thl,sl->hts", ql, key) / math.sqrt(D + Rr)
    s = s.masked_fill(pos > pos[-rows:].unsqueeze(1), -math.inf)          # every pool is selected in these contexts
    sink = w["sink"].double().view(H, 1, 1).expand(H, rows, 1)
    p = torch.softmax(torch.cat((s, sink), -1), -1)[..., :-1]
    o = torch.einsum("hts,sl,hdl->thd", p, ckv, up[:, D:])
    mu = ik - ik.mean(-1, keepdim=True)
    ik = mu * torch.rsqrt(mu.square().mean(-1, keepdim=True) + 1e-6) * w["k_ln_w"].double() + w["k_ln_b"].double()
    return _product(o.reshape(rows, H * D), w["o"]), ik[-rows:], ig[-rows:]


def exact(case, seed):
    cfg, W, past, h, X = _inputs(case, seed)
    lw, rows, n = W["layers"][0], case["rows"], case.get("streams", 1)
    more = {}
    if case["op"] == "moe":
        y = _exact_moe(cfg, lw["mlp"], h)
    else:
        f = {"gdn": _exact_gdn, "attn": _exact_attn, "mla": _exact_mla}[case["op"]]
        got = [f(cfg, lw["mix"], torch.cat((past[i], h[i * rows: (i + 1) * rows])).double(), rows) for i in range(n)]
        y = torch.cat([t[0] for t in got])
        if case["op"] == "gdn":
            more = {"S": torch.stack([t[1] for t in got]), "tail": torch.stack([t[2] for t in got])}
        else:
            for i, t in enumerate(got):
                for name, u in zip(("k", "v") if case["op"] == "attn" else ("ik", "ig"), t[1:]):
                    more["%s%d" % (name, i)] = None if case["op"] == "attn" and case["kv"] == "fp8" else u    # codes
    X = X.double() + y
    return {"h": _rms(X, lw["post_norm"].double(), cfg.norm_eps), "X": X, **more}
