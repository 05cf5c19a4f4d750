"""The work of a serving engine on one GPU, as cases that can be timed and compared.

A case is one pass of one of six kinds, through the package's public entry points:

``dense``   a step of a dense GQA decoder (``Qwen3Model.forward``): decode rows or ragged prompt chunks over the paged cache
``hybrid``  a step of a Gated-DeltaNet / full-attention decoder (``Qwen35Model.forward``)
``experts`` routing and routed experts of a mixture-of-experts layer (``ops.router_topk``, ``ops.moe_experts*``)
``latent``  latent attention over the paged latent cache (``ops.mla_rope_q``, ``ops.mla_attention``)
``kda``     the delta rule with a decay per key channel (``ops.kda_recurrent``)
``sample``  temperature / top-k / top-p / min-p sampling of a batch's logits (``ops.sample``)

Models are slices of the presets: four layers and a vocabulary shard, so that the output projection keeps about the share of
a step that it has in the whole model.  Decode steps are captured in a CUDA graph once, as the engine does it, and a pass
is one replay; prompt steps run kernel by kernel.
"""
from __future__ import annotations

import math

import torch

from pegainfer_b200 import ops
from pegainfer_b200.config import preset
from pegainfer_b200.kv.buffer import KvBuffer, KvLayout
from pegainfer_b200.kv.request_kv import KvView
from pegainfer_b200.loader.sources import DictSource
from pegainfer_b200.models.qwen3 import Qwen3Model
from pegainfer_b200.models.qwen35 import Qwen35Model
from pegainfer_b200.sched.executor import SeqStep, build_meta

DEV = "cuda:0"
PAGE = 16
LAYERS = 4
# 151936 / 8 and 248320 / 16: 4 of 36 layers, 4 of 64
VOCAB = {"qwen3-0.6b": 18992, "qwen3-4b": 18992, "qwen3-8b": 18992, "qwen3.5-27b": 15520}
BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
# experts' shapes: (hidden, inner width, local experts, experts per token, scoring, weights normalised, scale)
EXPERTS = {"bf16": (2048, 1408, 64, 6, "softmax", False, 1.0), "fp8": (2048, 1408, 64, 6, "softmax", False, 1.0), "int4": (7168, 2048, 48, 8, "sigmoid", True, 2.827)}


def listed():
    return [
        # one user: the latency of a token, on the smallest model
        dict(name="dense decode 1", kind="dense", model="qwen3-0.6b", decode=1, seqs=1, tokens=1, past=700),
        # a full batch in steady state: 1024-token prompts, 256 tokens out
        dict(name="dense decode 64", kind="dense", model="qwen3-8b", decode=1, seqs=64, tokens=64, past=1100),
        # a step that admits a few short questions of odd lengths
        dict(name="dense prompts 7 ragged", kind="dense", model="qwen3-8b", decode=0, seqs=7, tokens=1337, past=0),
        # the second chunk of a long prompt: the largest prompt step the scheduler forms by default
        dict(name="dense prompt chunk 4096", kind="dense", model="qwen3-8b", decode=0, seqs=1, tokens=4096, past=4096),
        dict(name="hybrid decode 32", kind="hybrid", decode=1, seqs=32, tokens=32, past=2176),
        # a 2048-token prompt beside the rest of another one
        dict(name="hybrid prompts 2 ragged", kind="hybrid", decode=0, seqs=2, tokens=2777, past=0),
        # one GPU's share of an expert-parallel decode step, INT4 weights
        dict(name="experts int4 128", kind="experts", format="int4", tokens=128),
        # a prompt step through bf16 experts, an odd number of rows
        dict(name="experts bf16 1711", kind="experts", format="bf16", tokens=1711),
        dict(name="latent decode 128", kind="latent", heads=64, decode=1, seqs=128, tokens=128, past=1150),
        dict(name="latent prompts 3 ragged", kind="latent", heads=16, decode=0, seqs=3, tokens=2999, past=0),
        dict(name="kda prompts 2 ragged", kind="kda", heads=96, decode=0, seqs=2, tokens=3001),
        dict(name="sample 64", kind="sample", rows=64, vocab=151936, top_k=50, top_p=0.9, min_p=0.0),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("dense", "dense", "dense", "hybrid", "hybrid", "experts", "experts", "latent", "latent", "kda", "sample"))
    if kind == "experts":
        fmt = rng.choice(("bf16", "fp8", "int4"))
        return dict(kind=kind, format=fmt, tokens=log(1, 512 if fmt == "int4" else 4096))
    if kind == "sample":
        k, p, m = rng.choice(((50, 0.9, 0.0), (0, 0.95, 0.0), (20, 0.8, 0.0), (0, 1.0, 0.05), (0, 1.0, 0.0), (40, 1.0, 0.0)))
        return dict(kind=kind, rows=log(1, 64), vocab=rng.choice((32000, 102400, 151936, 163840)), top_k=k, top_p=p, min_p=m)
    decode = rng.choice((0, 1))
    c = dict(kind=kind)
    if kind == "dense":
        c["model"] = rng.choice(("qwen3-0.6b", "qwen3-4b", "qwen3-8b"))
    if kind in ("latent", "kda"):
        c["heads"] = rng.choice((16, 64) if kind == "latent" else (16, 32, 96))
    if decode:
        seqs = log(1, {"latent": 128, "hybrid": 32}.get(kind, 64))
        c.update(decode=1, seqs=seqs, tokens=seqs)
    else:
        tokens = log(40, {"kda": 3000, "hybrid": 2700}.get(kind, 4096))
        c.update(decode=0, seqs=min(rng.randint(1, 8), tokens // 20), tokens=tokens)
    if kind != "kda":
        c["past"] = log(16, 1200 if decode else 4096) if decode or rng.random() < 0.3 else 0
    return c


# ----------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------
class _Draw:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed))

    def normal(self, *shape, scale=1.0, shift=0.0, dtype=BF):
        x = torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, 1.0, generator=self.g)
        x = x.mul_(scale) if scale != 1.0 else x
        return x.add_(shift) if shift else x

    def uniform(self, lo, hi, *shape):
        return torch.empty(shape, dtype=F32, device=DEV).uniform_(lo, hi, generator=self.g)

    def ints(self, n, *shape, dtype=torch.int32):
        return torch.randint(0, n, shape, dtype=dtype, device=DEV, generator=self.g)


def _lengths(case):
    """(new tokens, tokens already in the cache) of every sequence: spread around the case's mean, a fixed spread for every
    size."""
    n = case["seqs"]
    r = torch.Generator().manual_seed(case["tokens"] * 7919 + case.get("past", 0) * 31 + n)
    share = 0.4 + 1.2 * torch.rand(n, generator=r)
    past = [int(case.get("past", 0) * s * n / float(share.sum())) for s in share]
    if case["decode"]:
        return [1] * n, past
    share = (0.2 + torch.rand(n, generator=r)).flip(0)
    new = [max(1, int(case["tokens"] * s / float(share.sum()))) for s in share]
    new[-1] += case["tokens"] - sum(new)
    return new, past


def _pages(new, past, seed):
    """Page ids of every sequence, scattered as after some hours of serving; the pages that the step writes to come first,
    so that they are one slice of the pool."""
    spans = []
    nxt = 1
    for n, p in zip(new, past):
        first, total = p // PAGE, (p + n + PAGE - 1) // PAGE
        spans.append((first, list(range(nxt, nxt + total - first))))
        nxt += total - first
    written = nxt
    order = (torch.randperm(sum(f for f, _ in spans), generator=torch.Generator().manual_seed(int(seed) + 3)) + nxt).tolist()
    pages, at = [], 0
    for first, tail in spans:
        pages.append(order[at : at + first] + tail)
        at += first
    return pages, written, nxt + at


def _step(case, seed, vocab=1000):
    """Token ids, ragged step description and page lists of a case."""
    new, past = _lengths(case)
    pages, written, total = _pages(new, past, seed)
    toks = torch.randint(0, vocab, (sum(new),), generator=torch.Generator().manual_seed(int(seed) + 5)).tolist()
    seqs, at = [], 0
    for i, (n, p) in enumerate(zip(new, past)):
        seqs.append(SeqStep(rid=i, input_tokens=toks[at : at + n], start_pos=p, view=KvView(pages[i], p + n, PAGE)))
        at += n
    ids, meta = build_meta(seqs, PAGE, DEV)
    meta.state_slots = torch.arange(1, len(new) + 1, dtype=torch.int32, device=DEV)
    return dict(ids=ids, meta=meta, new=new, past=past, pages=pages, written=written, total=total)


def _last_rows(new):
    return torch.tensor(new, device=DEV).cumsum(0).sub_(1).to(torch.int32)


def _config(case):
    name = case.get("model", "qwen3.5-27b")
    kw = dict(num_layers=LAYERS, vocab_size=VOCAB[name], max_position=16384)
    if case["kind"] == "hybrid":
        kw["layer_types"] = preset(name).layer_types[:LAYERS]
    return preset(name, **kw)


def _dense_weights(cfg, d):
    h, hd = cfg.hidden_size, cfg.head_dim
    mat = lambda *s: d.normal(*s, scale=0.02)  # noqa: E731
    norm = lambda n: d.normal(n, scale=0.1, shift=1.0)  # noqa: E731
    w = {"model.embed_tokens.weight": mat(cfg.vocab_size, h), "model.norm.weight": norm(h)}
    if not cfg.tie_word_embeddings:
        w["lm_head.weight"] = mat(cfg.vocab_size, h)
    for i in range(cfg.num_layers):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = norm(h), norm(h)
        w[p + "self_attn.q_proj.weight"], w[p + "self_attn.o_proj.weight"] = mat(cfg.num_q_heads * hd, h), mat(h, cfg.num_q_heads * hd)
        w[p + "self_attn.k_proj.weight"], w[p + "self_attn.v_proj.weight"] = mat(cfg.num_kv_heads * hd, h), mat(cfg.num_kv_heads * hd, h)
        w[p + "self_attn.q_norm.weight"], w[p + "self_attn.k_norm.weight"] = norm(hd), norm(hd)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = mat(cfg.intermediate_size, h), mat(cfg.intermediate_size, h)
        w[p + "mlp.down_proj.weight"] = mat(h, cfg.intermediate_size)
    return w


def _hybrid_weights(cfg, d):
    h, hd, dk = cfg.hidden_size, cfg.head_dim, cfg.gdn_head_dim
    hk, hv = cfg.gdn_num_k_heads, cfg.gdn_num_v_heads
    mat = lambda *s: d.normal(*s, scale=0.02)  # noqa: E731
    norm = lambda n: d.normal(n, scale=0.1)  # noqa: E731
    wp = "model.language_model."
    w = {wp + "embed_tokens.weight": mat(cfg.vocab_size, h), wp + "norm.weight": norm(h), "lm_head.weight": mat(cfg.vocab_size, h)}
    for i in range(cfg.num_layers):
        p = f"{wp}layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = norm(h), norm(h)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = mat(cfg.intermediate_size, h), mat(cfg.intermediate_size, h)
        w[p + "mlp.down_proj.weight"] = mat(h, cfg.intermediate_size)
        if cfg.layer_type(i) == "full_attention":
            a = p + "self_attn."
            w[a + "q_proj.weight"], w[a + "o_proj.weight"] = mat(cfg.num_q_heads * hd * 2, h), mat(h, cfg.num_q_heads * hd)
            w[a + "k_proj.weight"], w[a + "v_proj.weight"] = mat(cfg.num_kv_heads * hd, h), mat(cfg.num_kv_heads * hd, h)
            w[a + "q_norm.weight"], w[a + "k_norm.weight"] = norm(hd), norm(hd)
        else:
            a, c = p + "linear_attn.", (2 * hk + hv) * dk
            w[a + "in_proj_qkv.weight"], w[a + "in_proj_z.weight"] = mat(c, h), mat(hv * dk, h)
            w[a + "in_proj_b.weight"], w[a + "in_proj_a.weight"] = mat(hv, h), mat(hv, h)
            w[a + "conv1d.weight"] = d.normal(c, 1, cfg.gdn_conv_kernel, scale=0.5)
            w[a + "dt_bias"] = d.uniform(-6.0, -2.0, hv)  # step sizes of 0.002 to 0.1 at a gate of zero
            w[a + "A_log"] = d.uniform(0.0, math.log(16.0), hv)
            w[a + "norm.weight"] = d.normal(dk, scale=0.1, shift=1.0, dtype=F32)
            w[a + "out_proj.weight"] = mat(h, hv * dk)
    return w


def _model_inputs(case, seed):
    cfg, d = _config(case), _Draw(seed)
    s = _step(case, seed, cfg.vocab_size)
    s["cfg"], s["w"] = cfg, (_dense_weights if case["kind"] == "dense" else _hybrid_weights)(cfg, d)
    n_kv = sum(cfg.layer_type(i) == "full_attention" for i in range(LAYERS)) if case["kind"] == "hybrid" else LAYERS
    s["kv"] = d.normal(n_kv, s["total"], 2, PAGE, cfg.num_kv_heads, cfg.head_dim)
    if case["kind"] == "hybrid":
        n, lin = len(s["new"]), LAYERS - n_kv
        s["conv"] = d.normal(lin, n + 1, (2 * cfg.gdn_num_k_heads + cfg.gdn_num_v_heads) * cfg.gdn_head_dim, cfg.gdn_conv_kernel - 1)
        s["ssm"] = d.normal(lin, n + 1, cfg.gdn_num_v_heads, cfg.gdn_head_dim, cfg.gdn_head_dim, scale=0.1, dtype=F32)
    return s


def _latent_inputs(case, seed):
    d, s, h = _Draw(seed), _step(case, seed), case["heads"]
    t = sum(s["new"])
    s.update(q=d.normal(t, h, 192), uk=d.normal(h, 128, 512, scale=0.03), uv=d.normal(h, 128, 512, scale=0.03), cache=d.normal(s["total"], PAGE, 576))
    return s


def _kda_inputs(case, seed):
    d, h = _Draw(seed), case["heads"]
    s = _step(case, seed)
    t, n = sum(s["new"]), len(s["new"])
    # q | k | v are slices of one fused buffer and beta is the head of the small projections, as in a layer
    s.update(qkv=d.normal(t, 3 * h * 128), f=d.normal(t, h * 128), small=d.normal(t, h + 128), a_log=d.uniform(0.0, math.log(4.0), h), dt_bias=d.uniform(-6.0, -2.0, h * 128),
             state=d.normal(n + 1, h, 128, 128, scale=0.1, dtype=F32))
    return s


def _experts_inputs(case, seed):
    h, inner, e, k, scoring, _, _ = EXPERTS[case["format"]]
    d, t = _Draw(seed), case["tokens"]
    s = dict(x=d.normal(t, h), logits=d.normal(t, e, dtype=F32), bias=d.normal(e, scale=0.01, dtype=F32) if scoring == "sigmoid" else None)
    for name, m, n in (("w13", 2 * inner, h), ("w2", h, inner)):
        if case["format"] == "int4":  # every eight values one word, a bf16 scale per 32
            s[name] = d.ints(1 << 32, e, m, n // 8, dtype=torch.int64).sub_(1 << 31).to(torch.int32)
            s[name + "_scale"] = d.uniform(0.002, 0.006, e, m, n // 32).to(BF)
        elif case["format"] == "fp8":
            s[name] = d.normal(e, m, n, scale=64.0).clamp_(-448, 448).to(torch.float8_e4m3fn)
            s[name + "_scale"] = d.uniform(0.0002, 0.0004, e, m // 128, n // 128)
        else:
            s[name] = d.normal(e, m, n, scale=0.02)
    return s


def _sample_inputs(case, seed):
    d, r = _Draw(seed), case["rows"]
    s = dict(logits=d.normal(r, case["vocab"], scale=2.5), temperature=d.uniform(0.6, 1.2, r), u=d.uniform(0.0, 1.0, r))
    s["top_k"] = torch.full((r,), case["top_k"], dtype=torch.int32, device=DEV)
    s["top_p"], s["min_p"] = torch.full((r,), case["top_p"], device=DEV), torch.full((r,), case["min_p"], device=DEV)
    return s


# ----------------------------------------------------------------------------------
# a pass
# ----------------------------------------------------------------------------------
def _captured(fn, *mutable):
    """``fn`` as a CUDA graph; the buffers that a pass updates are put back after the warm-up pass."""
    before = [x.clone() for x in mutable]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        fn()
    torch.cuda.current_stream().wait_stream(stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = fn()
    for x, b in zip(mutable, before):
        x.copy_(b)

    def replay():
        g.replay()
        return out

    replay.keeps = fn, mutable  # the buffers that the graph's kernels read
    return replay


def _maybe_captured(case, fn, *mutable):
    return _captured(fn, *mutable) if case.get("decode") or case["kind"] == "experts" and case["tokens"] <= 256 else fn


def _prepare_model(case, seed):
    s = _model_inputs(case, seed)
    cfg, meta = s["cfg"], s["meta"]
    model = (Qwen3Model if case["kind"] == "dense" else Qwen35Model)(cfg, DictSource(s["w"]), device=DEV, dtype=BF)
    geo = model.kv_geometry()
    kv = KvBuffer(KvLayout(geo["num_layers"], s["total"], PAGE, geo["kv_heads"], geo["head_dim"]), DEV)
    kv.data.copy_(s["kv"])
    rows = None if case["decode"] else _last_rows(s["new"])  # a prompt's logits are wanted behind its last token
    state = []
    if case["kind"] == "hybrid":
        rec = model.make_state(len(s["new"]))
        rec.conv.copy_(s["conv"])
        rec.ssm.copy_(s["ssm"])
        state = [rec.conv, rec.ssm]
    written = kv.data[:, 1 : s["written"]]

    def step():
        return {"logits": model.forward(s["ids"], meta, kv, rows), "kv": written, "state": [x[:, 1:] for x in state]}

    for name in ("w", "kv", "conv", "ssm"):
        if name in s:
            del s[name]
    return _maybe_captured(case, step, *state)


def _prepare_latent(case, seed):
    s = _latent_inputs(case, seed)
    cos, sin = ops.rope_tables(16384, 64, 10000.0, BF, DEV)
    scale = 192 ** -0.5
    return _maybe_captured(case, lambda: ops.mla_attention(ops.mla_rope_q(s["q"], cos, sin, s["meta"], 128), s["uk"], s["uv"], s["cache"], s["meta"], scale, 512))


def _prepare_kda(case, seed):
    s = _kda_inputs(case, seed)
    h = case["heads"]
    t = s["qkv"].shape[0]
    q, k, v = (s["qkv"][:, j * h * 128 : (j + 1) * h * 128].view(t, h, 128) for j in range(3))
    return _maybe_captured(case, lambda: {"out": ops.kda_recurrent(q, k, v, s["f"], s["small"][:, :h], s["a_log"], s["dt_bias"], -5.0, s["state"], s["meta"]), "state": s["state"][1:]}, s["state"])


def _prepare_experts(case, seed):
    s = _experts_inputs(case, seed)
    _, _, _, k, scoring, norm, scale = EXPERTS[case["format"]]
    if case["format"] == "int4":  # the loader's repack
        s["w13"], s["w2"] = ops.repack_int4_pairs(s["w13"]), ops.repack_int4_pairs(s["w2"])

    def layer():
        ids, w = ops.router_topk(s["logits"], k, scoring, s["bias"], norm_topk_prob=norm, scale=scale)
        if case["format"] == "bf16":
            return ops.moe_experts(s["x"], ids, w, s["w13"], s["w2"])
        fn = ops.moe_experts_int4 if case["format"] == "int4" else ops.moe_experts_fp8
        return fn(s["x"], ids, w, s["w13"], s["w13_scale"], s["w2"], s["w2_scale"])

    return _maybe_captured(case, layer)


def _prepare_sample(case, seed):
    s = _sample_inputs(case, seed)
    return lambda: ops.sample(s["logits"], s["temperature"], s["top_k"], s["top_p"], s["min_p"], s["u"])


def prepare(case, seed):
    return {"dense": _prepare_model, "hybrid": _prepare_model, "latent": _prepare_latent, "kda": _prepare_kda, "experts": _prepare_experts, "sample": _prepare_sample}[case["kind"]](case, seed)


def run(state):
    return state()


# ----------------------------------------------------------------------------------
# work
# ----------------------------------------------------------------------------------
def _pairs(new, past):
    """(query, key) pairs of causal attention."""
    return sum(n * p + n * (n + 1) / 2 for n, p in zip(new, past))


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": case["rows"] * (case["vocab"] * 2 + 24), "flops": 0}
    if kind == "experts":
        h, inner, e, k, _, _, _ = EXPERTS[case["format"]]
        t = case["tokens"]
        hit = e * (1 - (1 - k / e) ** t)  # experts that at least one of the tokens goes to
        each = {"bf16": 2.0, "fp8": 1.0 + 4 / 16384, "int4": 0.5 + 2 / 32}[case["format"]]
        return {"bytes": hit * 3 * h * inner * each + t * (2 * h + 4 * e + 4 * h), "flops": 2.0 * t * k * 3 * h * inner}
    new, past = _lengths(case)
    t, n, pairs, held = sum(new), len(new), _pairs(new, past), sum(new) + sum(past)
    if kind == "kda":
        h = case["heads"]
        return {"bytes": n * h * 16384 * 8 + t * h * (128 * 5 + 1) * 2, "flops": 8.0 * t * h * 16384}
    if kind == "latent":
        h = case["heads"]
        up = 2.0 * h * 512 * 256 * (t if case["decode"] else min(t, held))
        return {"bytes": held * 576 * 2 + t * h * 320 * 2 + h * 256 * 512 * 2, "flops": up + 2.0 * pairs * h * ((576 + 512) if case["decode"] else 320)}
    cfg = _config(case)
    h, hd, hq, hkv, ff = cfg.hidden_size, cfg.head_dim, cfg.num_q_heads, cfg.num_kv_heads, cfg.intermediate_size
    full = sum(cfg.layer_type(i) == "full_attention" for i in range(LAYERS)) if kind == "hybrid" else LAYERS
    gate = 2 if kind == "hybrid" else 1
    params = LAYERS * 3 * h * ff + full * h * hd * (hq * gate + 2 * hkv + hq)
    by = full * (held * 2 * hkv * hd * 2 + t * 2 * hkv * hd * 2)
    fl = full * 4.0 * pairs * hq * hd
    if kind == "hybrid":
        dk, hk, hv = cfg.gdn_head_dim, cfg.gdn_num_k_heads, cfg.gdn_num_v_heads
        lin = LAYERS - full
        params += lin * h * ((2 * hk + hv) * dk + hv * dk + 2 * hv + hv * dk)
        by += lin * n * (hv * dk * dk * 8 + (2 * hk + hv) * dk * 3 * 4)
        fl += lin * 8.0 * t * hv * dk * dk
    by += (params + cfg.vocab_size * h) * 2 + t * h * 2 + n * cfg.vocab_size * 2
    return {"bytes": by, "flops": fl + 2.0 * t * params + 2.0 * n * cfg.vocab_size * h}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    # bf16 rows through four layers, two roundings a sublayer: logits measured 0.017 off the 64-bit result, 5.5 sigma of it at
    # the largest of some millions
    if kind in ("dense", "hybrid"):
        return {"rel": 0.03, "max": 0.3}
    # e4m3 activations have three bits of mantissa; the others are one operation in bf16, measured 0.002 to 0.004 off
    return {"rel": 0.03, "max": 0.3} if case.get("format") == "fp8" else {"rel": 0.012, "max": 0.1}


# ----------------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _angles(pos, rot, theta):
    a = torch.outer(pos.double(), 1.0 / theta ** (torch.arange(0, rot // 2, device=DEV, dtype=F64) * 2.0 / rot))
    return a.cos()[:, None], a.sin()[:, None]


def _rotate(x, c, s):
    half = c.shape[-1]
    a, b, rest = x[..., :half], x[..., half : 2 * half], x[..., 2 * half :]
    return torch.cat([a * c - b * s, b * c + a * s, rest], -1)


def _silu(x):
    return x * torch.sigmoid(x)


def _causal(q, k, v, scale):
    """One sequence: ``q`` [n, H, D] over ``k``, ``v`` [m, G, D], the last n keys its own."""
    n, m, rep = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    mask = torch.arange(m, device=DEV)[None] > torch.arange(m - n, m, device=DEV)[:, None]
    out = torch.empty(n, q.shape[1], v.shape[-1], dtype=F64, device=DEV)
    for g in range(k.shape[1]):
        for h in range(g * rep, (g + 1) * rep) if n > 64 else (slice(g * rep, (g + 1) * rep),):
            sc = torch.tensordot(q[:, h], k[:, g], dims=([-1], [1])) * scale
            p = sc.masked_fill(mask if sc.dim() == 2 else mask[:, None], float("-inf")).softmax(-1)
            out[:, h] = p @ v[:, g]
    return out


def _positions(s):
    return torch.cat([torch.arange(p, p + n, device=DEV) for n, p in zip(s["new"], s["past"])])


def _attend(s, layer, q, k, v, scale):
    """Appends k and v to the pages of ``layer`` [pages, 2, PAGE, G, D] (64 bits) and attends, sequence by sequence."""
    out, at = [], 0
    for n, p, pages in zip(s["new"], s["past"], s["pages"]):
        idx = torch.tensor(pages, device=DEV)
        pos = torch.arange(p, p + n, device=DEV)
        layer[idx[pos // PAGE], 0, pos % PAGE] = k[at : at + n]
        layer[idx[pos // PAGE], 1, pos % PAGE] = v[at : at + n]
        held = layer[idx]
        out.append(_causal(q[at : at + n], held[:, 0].flatten(0, 1)[: p + n], held[:, 1].flatten(0, 1)[: p + n], scale))
        at += n
    return torch.cat(out)


def _delta(S, q, k, v, dec, beta, out):
    """Gated delta rule of one sequence, token by token: ``S`` [H, Dk, Dv], ``dec`` [n, H, Dk or 1]."""
    for i in range(q.shape[0]):
        S = S * dec[i].unsqueeze(-1)
        d = (v[i] - torch.einsum("hkv,hk->hv", S, k[i])) * beta[i].unsqueeze(-1)
        S = torch.baddbmm(S, k[i].unsqueeze(2), d.unsqueeze(1))
        out[i] = torch.einsum("hkv,hk->hv", S, q[i])
    return S


def _unit(x):
    return x * torch.rsqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)


def _exact_linear_attention(s, cfg, w, a, x, j, conv, ssm):
    hk, hv, dk = cfg.gdn_num_k_heads, cfg.gdn_num_v_heads, cfg.gdn_head_dim
    mixed, z = x @ w(a + "in_proj_qkv.weight").T, x @ w(a + "in_proj_z.weight").T
    b, al = x @ w(a + "in_proj_b.weight").T, x @ w(a + "in_proj_a.weight").T
    dec = torch.exp(-torch.exp(w(a + "A_log")) * torch.nn.functional.softplus(al + w(a + "dt_bias"), threshold=100.0))
    taps, out, at = w(a + "conv1d.weight").squeeze(1), torch.empty(x.shape[0], hv, dk, dtype=F64, device=DEV), 0
    for i, n in enumerate(s["new"]):
        seq = torch.cat([conv[j, i + 1].T, mixed[at : at + n]])
        conv[j, i + 1] = seq[-(taps.shape[1] - 1) :].T
        y = _silu(sum(seq[r : r + n] * taps[:, r] for r in range(taps.shape[1])))
        q, k, v = y[:, : hk * dk].view(n, hk, dk), y[:, hk * dk : 2 * hk * dk].view(n, hk, dk), y[:, 2 * hk * dk :].view(n, hv, dk)
        q, k = (_unit(u).repeat_interleave(hv // hk, 1) for u in (q, k))
        sl = slice(at, at + n)
        ssm[j, i + 1] = _delta(ssm[j, i + 1], q * dk ** -0.5, k, v, dec[sl].unsqueeze(-1), torch.sigmoid(b[sl]), out[sl])
        at += n
    return (_rms(out, w(a + "norm.weight"), cfg.rms_eps) * _silu(z.view(out.shape))).flatten(1) @ w(a + "out_proj.weight").T


def _exact_model(case, seed):
    s = _model_inputs(case, seed)
    cfg, hybrid = s["cfg"], case["kind"] == "hybrid"
    wp = "model.language_model." if hybrid else "model."
    w = lambda name: s["w"][name].double()  # noqa: E731
    norm = lambda x, name: _rms(x, w(name) + (1.0 if hybrid else 0.0), cfg.rms_eps)  # noqa: E731
    kv = s["kv"].double()
    conv, ssm = (s["conv"].double(), s["ssm"].double()) if hybrid else (None, None)
    hq, hkv, hd = cfg.num_q_heads, cfg.num_kv_heads, cfg.head_dim
    x = s["w"][wp + "embed_tokens.weight"][s["ids"].long()].double()
    cos, sin = _angles(_positions(s), cfg.rotary_dim, cfg.rope_theta)
    t, n_full, n_lin = x.shape[0], 0, 0
    for i in range(LAYERS):
        p = f"{wp}layers.{i}."
        y = norm(x, p + "input_layernorm.weight")
        if hybrid and cfg.layer_type(i) != "full_attention":
            x = x + _exact_linear_attention(s, cfg, w, p + "linear_attn.", y, n_lin, conv, ssm)
            n_lin += 1
        else:
            a = p + "self_attn."
            q, k, v = (y @ w(f"{a}{c}_proj.weight").T for c in "qkv")
            q = q.view(t, hq, -1)
            gate = torch.sigmoid(q[..., hd:]) if hybrid else 1.0
            q = _rotate(norm(q[..., :hd], a + "q_norm.weight"), cos, sin)
            k = _rotate(norm(k.view(t, hkv, hd), a + "k_norm.weight"), cos, sin)
            o = _attend(s, kv[n_full], q, k, v.view(t, hkv, hd), hd ** -0.5) * gate
            x = x + o.flatten(1) @ w(a + "o_proj.weight").T
            n_full += 1
        y = norm(x, p + "post_attention_layernorm.weight")
        x = x + (_silu(y @ w(p + "mlp.gate_proj.weight").T) * (y @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    if not case["decode"]:
        x = x[_last_rows(s["new"]).long()]
    x = norm(x, wp + "norm.weight")
    head = "lm_head.weight" if "lm_head.weight" in s["w"] else wp + "embed_tokens.weight"
    return {"logits": x @ w(head).T, "kv": kv[:, 1 : s["written"]], "state": [conv[:, 1:], ssm[:, 1:]] if hybrid else []}


def _exact_latent(case, seed):
    s = _latent_inputs(case, seed)
    cos, sin = _angles(_positions(s), 64, 10000.0)
    q, uk, uv = s["q"].double(), s["uk"].double(), s["uv"].double()
    pe = torch.cat([q[..., 128::2], q[..., 129::2]], -1)
    pe = _rotate(pe, cos, sin)
    out, at = [], 0
    for n, p, pages in zip(s["new"], s["past"], s["pages"]):
        rows = s["cache"][torch.tensor(pages, device=DEV)].flatten(0, 1)[: p + n].double()
        sl, heads = slice(at, at + n), []
        for h in range(case["heads"]) if n > 64 else (slice(0, case["heads"]),):
            if n > 64:  # expand keys and values of one head
                k = torch.cat([rows[:, :512] @ uk[h].T, rows[:, 512:]], -1)
                heads.append(_causal(torch.cat([q[sl, h, :128], pe[sl, h]], -1).unsqueeze(1), k.unsqueeze(1), (rows[:, :512] @ uv[h].T).unsqueeze(1), 192 ** -0.5))
            else:  # all heads share one key of 512 + 64
                qa = torch.cat([torch.einsum("nhd,hdc->nhc", q[sl, :, :128], uk), pe[sl]], -1)
                heads.append(torch.einsum("nhc,hvc->nhv", _causal(qa, rows.unsqueeze(1), rows[:, None, :512], 192 ** -0.5), uv))
        out.append(torch.cat(heads, 1))
        at += n
    return torch.cat(out).flatten(1)


def _exact_kda(case, seed):
    s, h = _kda_inputs(case, seed), case["heads"]
    t = s["qkv"].shape[0]
    q, k, v = (s["qkv"][:, j * h * 128 : (j + 1) * h * 128].view(t, h, 128).double() for j in range(3))
    q, k = _unit(q) * 128 ** -0.5, _unit(k)
    dec = torch.exp(-5.0 * torch.sigmoid(torch.exp(s["a_log"].double()).view(h, 1) * (s["f"].double() + s["dt_bias"].double()).view(t, h, 128)))
    beta, out, state, at = torch.sigmoid(s["small"][:, :h].double()), torch.empty(t, h, 128, dtype=F64, device=DEV), s["state"].double(), 0
    for i, n in enumerate(s["new"]):
        sl = slice(at, at + n)
        state[i + 1] = _delta(state[i + 1], q[sl], k[sl], v[sl], dec[sl], beta[sl], out[sl])
        at += n
    return {"out": out, "state": state[1:]}


def _matrix(s, name, e):
    w = s[name][e]
    if w.dtype == torch.int32:
        q = ((w.unsqueeze(-1) >> torch.arange(0, 32, 4, device=DEV, dtype=torch.int32)) & 15).flatten(1).double() - 8.0
        return q * s[name + "_scale"][e].double().repeat_interleave(32, 1)
    if w.dtype == torch.float8_e4m3fn:
        return w.double() * s[name + "_scale"][e].double().repeat_interleave(128, 0).repeat_interleave(128, 1)
    return w.double()


def _exact_experts(case, seed):
    s = _experts_inputs(case, seed)
    _, inner, e, k, scoring, norm, scale = EXPERTS[case["format"]]
    lg = s["logits"].double()
    score = lg.softmax(-1) if scoring == "softmax" else torch.sigmoid(lg)
    ids = (score + (s["bias"].double() if s["bias"] is not None else 0.0)).topk(k, -1).indices
    w = score.gather(1, ids)
    w = (w / w.sum(-1, keepdim=True) if norm else w) * scale
    x, out = s["x"].double(), torch.zeros(case["tokens"], s["x"].shape[1], dtype=F64, device=DEV)
    for i in range(e):
        rows, pick = (ids == i).nonzero(as_tuple=True)
        if rows.numel():
            y = x[rows] @ _matrix(s, "w13", i).T
            out.index_add_(0, rows, (_silu(y[:, :inner]) * y[:, inner:]) @ _matrix(s, "w2", i).T * w[rows, pick, None])
    return out


def exact(case, seed):
    if case["kind"] == "sample":
        return None  # token ids
    return {"dense": _exact_model, "hybrid": _exact_model, "latent": _exact_latent, "kda": _exact_kda, "experts": _exact_experts}[case["kind"]](case, seed)
