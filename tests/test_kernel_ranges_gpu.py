"""Kernels at the edges of the ranges that their launch rules draw: tile and segment edges, remainders, odd widths, the
smallest and largest sizes, against the PyTorch restatements."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from pegainfer_b200.ops import reference as R
from tests.test_kernels_gpu import DEV, _state_meta, cu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels,taps", [(64, 4), (1040, 4), (1040, 2), (136, 3), (37, 4)])  # 16-byte pieces; one channel per thread
def test_gdn_conv1d_segments(channels, taps):
    torch.manual_seed(channels + taps)
    q_lens = [1, 2, 3, 4, 15, 16, 17, 31, 33, 64, 5]  # around the carried rows and around segments of 16 tokens
    meta = _state_meta(q_lens, [3, 1, 4, 2, 8, 5, 7, 6, 9, 10, -1])
    x = torch.randn(sum(q_lens), channels + 24, device=DEV).bfloat16()[:, 8 : 8 + channels]
    w = (torch.randn(channels, taps, device=DEV) * 0.5).bfloat16()
    st1 = torch.randn(11, channels, taps - 1, device=DEV).bfloat16()
    st2 = st1.clone()
    y1, y2 = cu().gdn_conv1d(x, w, st1, meta), R.gdn_conv1d(x, w, st2, meta)
    # the sum is rounded to bf16 once; its order may move it by one step, and SiLU's slope is at most 1.1: two steps of bf16
    assert ((y1.float() - y2.float()).abs() <= 2 ** -7 * y2.float().abs() + 2 ** -9).all()
    assert torch.equal(st1, st2)


@pytest.mark.parametrize("routes,e0,e_local,total", [(1, 0, 1, 1), (31, 0, 3, 5), (256, 3, 16, 40), (255, 0, 16, 16), (257, 3, 16, 40), (200, 5, 17, 30), (100, 0, 1, 4), (512, 8, 64, 96), (513, 0, 384, 384), (8193, 16, 48, 384), (40007, 0, 512, 512)])
def test_route_sort_is_stable(routes, e0, e_local, total):
    g = torch.Generator().manual_seed(routes)
    ids = torch.randint(0, total, (routes, 1), generator=g, dtype=torch.int32)
    if routes > 600:
        ids[100:400] = e0 + e_local - 1  # a run of one expert
    offsets, src, pos = cu().moe_route_plan(ids.to(DEV), e0, e_local)
    local = ids.flatten().long() - e0
    local[(local < 0) | (local >= e_local)] = e_local
    order = torch.argsort(local, stable=True)
    n = int((local < e_local).sum())
    want = torch.full((routes,), -1)
    want[order[:n]] = torch.arange(n)
    assert torch.equal(offsets.cpu().long(), torch.searchsorted(local[order], torch.arange(e_local + 1)))
    assert torch.equal(pos.cpu().long()[:routes], want) and torch.equal(src.cpu().long()[:n], order[:n])


@pytest.mark.parametrize("dv", [64, 128])
def test_kda_blocks_of_four_tokens(dv):
    torch.manual_seed(dv)
    heads, dk, q_lens, slots = 3, 128, [5, 1, 16, 17, 4, 33, 130, 9], [3, 1, 4, 2, 8, 5, 7, -1]  # around blocks of 4 and stages of 16
    meta, t = _state_meta(q_lens, slots), sum(q_lens)
    qkv = torch.randn(t, heads * (2 * dk + dv) + 8, device=DEV).bfloat16()
    q, k = (qkv[:, j * heads * dk : (j + 1) * heads * dk].view(t, heads, dk) for j in range(2))
    v = qkv[:, 2 * heads * dk : 2 * heads * dk + heads * dv].view(t, heads, dv)
    f, b = torch.randn(t, heads * dk, device=DEV).bfloat16(), torch.randn(t, heads + 5, device=DEV).bfloat16()[:, :heads]
    a_log, dt = torch.randn(heads, device=DEV) * 0.5, torch.randn(heads * dk, device=DEV) - 2
    st1 = torch.randn(9, heads, dk, dv, device=DEV)
    st2 = st1.double()
    o1 = cu().kda_recurrent(q, k, v, f, b, a_log, dt, -5.0, st1, meta)
    # the rule in 64 bits: the kernel works in f32 (2^-23 a step, fewer than 2^6 steps that matter) and rounds its output to bf16
    unit = lambda x: x * torch.rsqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    qd, kd = unit(q.double()) * dk ** -0.5, unit(k.double())
    dec = torch.exp(-5.0 * torch.sigmoid(a_log.double().exp().view(heads, 1) * (f.double() + dt.double()).view(t, heads, dk)))
    beta, at = torch.sigmoid(b.double()), 0
    for n, slot in zip(q_lens, slots):
        for i in range(at, at + n):
            if slot < 0:
                continue
            S = st2[slot] * dec[i].unsqueeze(-1)
            d = (v[i].double() - torch.einsum("hkv,hk->hv", S, kd[i])) * beta[i].unsqueeze(-1)
            st2[slot] = S + kd[i].unsqueeze(-1) * d.unsqueeze(1)
            want = torch.einsum("hkv,hk->hv", st2[slot], qd[i])
            assert (o1[i].double() - want).abs().max() <= 2 ** -8 * want.abs().max() + 1e-5
        at += n
    assert (st1.double() - st2).abs().max() < 2 ** -17 * st2.abs().max()


@pytest.mark.parametrize("vocab,dtype", [(9, torch.bfloat16), (1023, torch.float32), (24577, torch.bfloat16), (49160, torch.float32), (151936, torch.bfloat16), (163841, torch.bfloat16)])
def test_sampler_brackets(vocab, dtype):
    """Thresholds where the coarse bracket is hard: every token alike, tokens spread over few bins (more of them than the
    list holds), a limit of no mass, masked tokens, infinities; odd vocabularies (rows that are not 16-byte aligned)."""
    g = torch.Generator(device=DEV).manual_seed(vocab)
    lg = torch.randn(12, vocab, device=DEV, generator=g)
    lg[1] = 1.25
    lg[2] *= 0.002
    lg[3] = lg[3] * 2.5
    lg[4, vocab // 2 :] = float("-inf")
    lg[5] = float("-inf")
    lg[5, vocab - 1] = 0.0
    lg[6, 3] = float("inf")
    lg[7, 0] = float("nan")
    lg[8] *= 30
    lg = lg.to(dtype)
    one = torch.ones(12, device=DEV)
    for k, p, m in ((0, 0.95, 0.0), (0, 0.5, 0.0), (40, 1.0, 0.0), (3, 0.9, 0.0), (1, 1.0, 0.0), (0, 0.0, 0.0), (0, 1.0, 0.05), (0, 1.0, 0.0), (vocab - 1, 0.999, 0.001)):
        u = torch.rand(12, device=DEV, generator=g)
        got = cu().sample(lg, one, torch.full((12,), k, dtype=torch.int32, device=DEV), one * p, one * m, u).long()
        assert ((got >= 0) & (got < vocab)).all()
        assert got[5] == vocab - 1 and got[6] == 3 and (got[7] != 0 or p == 0.0)
        rows = [0, 1, 2, 3, 4, 8]  # finite maxima: the kernel's e = exp(s - max) is within 2^-20 of this one
        s = lg[rows].double()
        e = torch.exp(s - s.amax(-1, keepdim=True))
        srt = e.sort(-1, descending=True).values
        before = srt.cumsum(-1) - srt
        keep = (torch.arange(vocab, device=DEV) < (k if 0 < k < vocab else vocab)).expand(len(rows), -1)
        if p < 1:
            keep = keep & (before < p * e.sum(-1, keepdim=True) * (1 + 1e-5))  # a hair wide: the tokens at the crossing
        keep = keep | (torch.arange(vocab, device=DEV) == 0)
        thr = torch.where(keep, srt, torch.full_like(srt, 2.0)).amin(-1, keepdim=True)
        pick = e.gather(-1, got[rows, None])
        assert (pick >= thr * (1 - 1e-5)).all() and (pick >= m * (1 - 1e-5)).all()
        if p == 1.0:  # the keep-set is known: the draw is the one that the cumulative mass in vocabulary order names
            mass = torch.where((e >= thr * (1 - 1e-9)) & (e >= m), e, torch.zeros_like(e))
            cdf = mass.cumsum(-1)
            target = u[rows, None].double() * cdf[:, -1:]
            slack = cdf[:, -1:] * 2e-5
            at = cdf.gather(-1, got[rows, None])
            assert (at >= target - slack).all() and (at - mass.gather(-1, got[rows, None]) <= target + slack).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("temp", [1e-5, 7e-5, 3e-4, 1e-3])
def test_sampler_at_low_temperatures(temp, dtype):
    """Tempered logits of 10^4 to 10^7, whose products round by more than tokens of mass may differ: only the largest has mass (the next one
    is a thousand units and more below it), so every row gives the largest, whatever its piece of eight."""
    g = torch.Generator(device=DEV).manual_seed(1)
    top = torch.arange(128, 512, device=DEV)
    top = torch.cat([(1 + (top % 128) / 128) * 2.0 ** (top // 128 + 2), -(1 + (top % 128) / 128) * 2.0 ** (top // 128 + 2)])  # every bf16 number of 8 to 64
    rows, vocab = top.numel(), 24577
    lg = (top[:, None] - 1 - torch.rand(rows, vocab, device=DEV, generator=g) * 8).to(dtype)
    want = torch.randint(0, vocab, (rows,), device=DEV, generator=g)
    lg[torch.arange(rows, device=DEV), want] = top.to(dtype)
    one = torch.ones(rows, device=DEV)
    for k, p, m in ((1, 1.0, 0.0), (50, 1.0, 0.0), (0, 0.9, 0.0), (0, 1.0, 1.0), (0, 1.0, 0.05), (0, 1.0, 0.0), (20, 0.8, 0.1)):
        got = cu().sample(lg, one * temp, torch.full((rows,), k, dtype=torch.int32, device=DEV), one * p, one * m, torch.rand(rows, device=DEV, generator=g))
        assert torch.equal(got.long(), want)


@pytest.mark.parametrize("heads,page,splits", [(16, 16, 1), (16, 64, 5), (32, 32, 2), (64, 16, 1), (64, 16, 3), (96, 16, 2)])
def test_latent_decode_tiles(heads, page, splits, monkeypatch):
    """Absorbed attention around tiles of 64 keys, padding rows, blocks of 16 to 64 heads (``splits``: blocks that a row may have, from
    which their heads follow; where its keys are cut follows from all rows' lengths), and rows behind a sequence's end that hold NaN."""
    torch.manual_seed(heads + page)
    kv_lens = [1, 63, 64, 65, 0, 129, 200, 511, 1000, 77]
    n = len(kv_lens)
    per = [(x + page - 1) // page for x in kv_lens]
    table, at = torch.zeros(n, max(per), dtype=torch.int32), 1
    for i, m in enumerate(per):
        table[i, :m] = torch.arange(at, at + m)
        at += m
    cache = torch.randn(at, page, 576, device=DEV).bfloat16()
    for i, (x, m) in enumerate(zip(kv_lens, per)):
        if m and x % page:
            cache[table[i, m - 1].item(), x % page :] = float("nan")
    pos = torch.tensor([max(x - 1, 0) for x in kv_lens], dtype=torch.int32, device=DEV)
    meta = R.AttnMeta(torch.arange(n + 1, dtype=torch.int32, device=DEV), torch.tensor(kv_lens, dtype=torch.int32, device=DEV), table.to(DEV), pos, pos, page, n, n, 1, max(kv_lens), True,
                      list(range(n + 1)), kv_lens)
    q = torch.randn(n, heads, 192, device=DEV).bfloat16()
    uk, uv = (torch.randn(heads, 128, 512, device=DEV) * 0.05).bfloat16(), (torch.randn(heads, 128, 512, device=DEV) * 0.05).bfloat16()
    q[2] *= 8  # scores that pass the reference value by far in a later tile
    cos, sin = R.rope_tables(2048, 64, 1e4, torch.bfloat16, DEV)
    monkeypatch.setattr(cu(), "_latent_splits", lambda *a: splits)
    got = cu().mla_attention(cu().mla_rope_q(q, cos, sin, meta, 128), uk, uv, cache, meta, 0.07, 512)
    want = R.mla_attention(R.mla_rope_q(q, cos, sin, meta, 128), uk, uv, cache, meta, 0.07, 512)
    assert not got[4].any() and torch.isfinite(got.float()).all()
    # weights and outputs of both are rounded to bf16 (2^-8 each), the sums are of some hundred terms: 2^-6 of the largest
    assert (got.float() - want.float()).abs().max() <= 2 ** -6 * want.float().abs().max()
    assert cu().read_status(DEV) == 0


@pytest.mark.parametrize("dim,heads,act", [(128, 6, "silu"), (128, 5, "sigmoid"), (256, 3, "silu"), (64, 7, "silu"), (96, 3, "sigmoid")])
@pytest.mark.parametrize("t", [37, 4001])  # one row per warp and several, rows that do not fill the last block
def test_gated_norm_reads_the_gate_in_place(dim, heads, act, t):
    torch.manual_seed(dim)
    x = torch.randn(t, heads, dim, device=DEV).bfloat16()
    fused = torch.randn(t, heads * dim + 24, device=DEV).bfloat16()
    w = torch.rand(dim, device=DEV) + 0.5
    # 16-byte pieces; not even aligned; a dense gate
    for gate in (fused[:, 8 : 8 + heads * dim].view(t, heads, dim), fused[:, 1 : 1 + heads * dim].view(t, heads, dim), fused[:, 8 : 8 + heads * dim].reshape(t, heads * dim).view(t, heads, dim)):
        got, want = cu().gated_rms_norm(x, gate, w, 1e-6, act), R.gated_rms_norm(x, gate, w, 1e-6, act)
        # f32 sums in another order: one step of bf16, two where two rounded factors meet
        assert ((got.float() - want.float()).abs() <= 2 ** -7 * want.float().abs() + 1e-6).all()


def test_gated_norm_of_no_rows():
    w = torch.ones(128, device=DEV)
    for shape in ((0, 4, 128), (5, 0, 128), (0, 128)):
        x = torch.zeros(shape, device=DEV).bfloat16()
        assert cu().gated_rms_norm(x, x, w, 1e-6).shape == shape


@pytest.mark.parametrize("t", [1, 2, 3, 4])
@pytest.mark.parametrize("h,hq,hkv,inter", [(1024, 16, 8, 3072), (2560, 32, 8, 9728), (256, 2, 1, 512), (4096, 32, 8, 12288)])
def test_chain_of_few_rows(t, h, hq, hkv, inter):
    """One to four rows through the streamed form of the decode chain, phase by phase against f64 of the same bf16 inputs."""
    K = cu()
    torch.manual_seed(t + h)
    page, eps, d = 16, 1e-6, 128
    mat = lambda m, k: (torch.randn(m, k, device=DEV) * 0.03).bfloat16()  # noqa: E731
    o, gu, down, qkv = mat(h, hq * d), mat(2 * inter, h), mat(h, inter), mat((hq + 2 * hkv) * d, h)
    n1, n2, qn, kn = ((torch.rand(s, device=DEV) + 0.5).bfloat16() for s in (h, h, d, d))
    a, res = torch.randn(t, hq * d, device=DEV).bfloat16(), torch.randn(t, h, device=DEV).bfloat16()
    cos, sin = R.rope_tables(512, d, 1e4, torch.bfloat16, DEV)
    kv = torch.zeros(8, 2, page, hkv, d, device=DEV).bfloat16()
    pos = torch.tensor([3, 77, 5, 400][:t], dtype=torch.int32, device=DEV)
    slots = torch.tensor([18, 35, 100, 127][:t], dtype=torch.int32, device=DEV)
    meta = R.AttnMeta(torch.arange(t + 1, dtype=torch.int32, device=DEV), pos + 1, torch.zeros(t, 8, dtype=torch.int32, device=DEV), slots, pos, page, t, t, 1, 512, True)
    spec = dict(q_norm=qn, k_norm=kn, cos=cos, sin=sin, meta=meta, kv_layer=kv, hq=hq, hkv=hkv, eps=eps)
    r1 = res.clone()
    outs = K.decode_chain(a, [(o, K.CH_RESID_NORM, n1, False), (gu, K.CH_SWIGLU, None, False), (down, K.CH_RESID_NORM, n2, True), (qkv, K.CH_QKV_ROPE, spec, False)], residual=r1, eps=eps)

    def near(got, want, roundings):  # every rounding to bf16 on the way is at most 2^-9 of a value; products add up as their squares
        err = (got.double() - want.double()).norm() / want.double().norm()
        assert err < roundings * 2 ** -9, float(err)

    h1 = res.double() + a.double() @ o.double().t()
    near(outs[0].xw, h1 * n1.double(), 2)
    inv = lambda x: torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)  # noqa: E731
    x1 = outs[0].xw.double() * torch.rsqrt(outs[0].ssp[:, : outs[0].parts].double().sum(-1, keepdim=True) / h + eps)
    near(x1, h1 * inv(h1) * n1.double(), 2)
    y = x1 @ gu.double().t()
    near(outs[1], torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2], 3)
    h2 = h1 + outs[1].double() @ down.double().t()
    near(r1, h2, 2)
    near(outs[2].xw, h2 * (n2.double() + 1), 3)
    x2 = outs[2].xw.double() * torch.rsqrt(outs[2].ssp[:, : outs[2].parts].double().sum(-1, keepdim=True) / h + eps)
    z = (x2 @ qkv.double().t()).bfloat16()
    kv2 = torch.zeros_like(kv)
    q = R.qk_norm_rope_append(z, qn, kn, cos, sin, meta, kv2, hq, hkv, d, eps)
    near(outs[3], q, 4)
    near(kv, kv2, 4)
    assert not K.ctx(DEV).chain_counters.any() and K.read_status(DEV) == 0


@pytest.mark.parametrize("t,m,k", [(1, 2, 256), (2, 130, 512), (3, 4098, 768), (4, 1000, 12288), (1, 40000, 256), (4, 64, 5120)])
def test_linear_of_few_rows(t, m, k):
    torch.manual_seed(m)
    x, w = torch.randn(t, k + 8, device=DEV).bfloat16()[:, :k], torch.randn(m, k, device=DEV).bfloat16()
    want = x.double() @ w.double().t()
    lim = k * 2 ** -24 * (x.double().abs() @ w.double().abs().t())  # f32 sums of k products
    for dtype in (torch.bfloat16, torch.float32):
        got = cu().linear(x, w, dtype).double()
        assert ((got - want).abs() <= lim + (2 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)).all()


@pytest.mark.parametrize("dv", [64, 128])
@pytest.mark.parametrize("lens,room", [([32, 63, 64, 65, 1, 129, 0, 31], None), ([700, 33, 450], 7), ([140] * 9 + [3] + [200] * 4, 5), ([260], 1)])
def test_gated_delta_chunks_in_segments(lens, room, dv, monkeypatch):
    """All chunks at once, segments of the sequences, and one kernel (short sequences; scratch for less than two chunks of each) give
    the same bytes, and the token-by-token rule's values."""
    torch.manual_seed(sum(lens) + dv)
    hk, hv, dk = 2, 4, 128
    meta = _state_meta(lens, list(range(1, len(lens) + 1)))
    t = meta.num_tokens
    x = torch.randn(t, 2 * hk * dk + hv * dv, device=DEV).bfloat16()
    q, k, v = (y.view(t, -1, d) for y, d in zip(x.split([hk * dk, hk * dk, hv * dv], 1), (dk, dk, dv)))
    g, beta = -torch.rand(t, hv, device=DEV), torch.rand(t, hv, device=DEV)
    s0 = torch.randn(len(lens) + 2, hv, dk, dv, device=DEV) * 0.1
    want_s, runs = s0.clone(), []
    want = R.gdn_recurrent(q, k, v, g, beta, want_s, meta)
    for limit, known in ((256 << 20, True), (256 << 20, False)) + (((room * hv * (16384 * 3 + 8192 * 2 + 256 + 128 * dv), True),) if room else ()):
        monkeypatch.setattr(cu(), "_GDN_WS_BYTES", limit)
        meta.h_q_indptr = meta.q_indptr.tolist() if known else None
        s = s0.clone()
        runs.append((cu().gdn_recurrent(q, k, v, g, beta, s, meta, chunked=True), s))
    for o, s in runs[1:]:
        assert torch.equal(o, runs[0][0]) and torch.equal(s, runs[0][1])
    short = _state_meta([128], [1])  # the first 128 tokens of the first sequence, in one kernel and beside a longer sequence
    if lens[0] > 128:
        both = _state_meta([128, lens[0]], [1, 2])
        sa, sb = s0.clone(), s0.clone()
        cat = lambda y: torch.cat((y[:128], y[: lens[0]]))  # noqa: E731
        a = cu().gdn_recurrent(q[:128], k[:128], v[:128], g[:128], beta[:128], sa, short, chunked=True)
        b = cu().gdn_recurrent(cat(q), cat(k), cat(v), cat(g), cat(beta), sb, both, chunked=True)
        assert torch.equal(a, b[:128]) and torch.equal(sa[1], sb[1])
    # operands of the products are bf16 (2^-9 each), sums f32: the limits of the chunk scan against the f32 rule
    assert (runs[0][0].float() - want.float()).abs().max() < 0.03 * want.float().abs().max() + 2e-3
    assert (runs[0][1] - want_s).abs().max() < 0.03 * want_s.abs().max()


@pytest.mark.parametrize(
    "t,m,k,splits,rounds",
    # whole tiles only; cut tiles alone, in two, three and four ranges, some of them uneven, m and t ragged; cut tiles behind a whole round
    [(257, 1024, 2048, 1, 0), (1337, 4096, 1024, 1, 1), (700, 5008, 1096, 1, 0), (4100, 4112, 512, 1, 3), (1200, 1504, 776, 1, 0), (300, 1280, 8704, 4, 0), (65, 528, 4104, 4, 0), (300, 4096, 4096, 2, 0),
     (512, 2576, 4104, 3, 0), (1290, 4112, 8200, 2, 1), (1100, 4096, 12288, 3, 1), (842, 5136, 5128, 4, 1)],
)
def test_two_sm_gemm_cuts_the_last_round(t, m, k, splits, rounds):
    """Tiles of the last round cut in ranges of k: a few tiles only, tiles behind whole rounds, ragged edges, uneven ranges."""
    K = cu()
    plan = K.gemm2sm_plan(t, m, k)
    # with 72 or 74 pairs at once; the rule's lines may move, the ranges that they are to reach may not go untested
    assert plan["splits"] == splits and (plan["whole"] > 0) == (rounds > 0 or splits == 1), plan
    torch.manual_seed(m)
    x, w = torch.randn(t, k + 8, device=DEV).bfloat16()[:, :k], torch.randn(m, k, device=DEV).bfloat16()
    want = x.double() @ w.double().t()
    lim = 2 ** -8 * want.abs() + k * 2 ** -24 * (x.double().abs() @ w.double().abs().t())  # f32 sums of k products, rounded to bf16
    y = K.linear_2sm(x, w)
    assert ((y.double() - want).abs() <= lim).all()
    assert torch.equal(y, K.linear_2sm(x, w)) and not K.ctx(DEV).gemm_counters.any() and K.read_status(DEV) == 0
    glu = K.linear_swiglu_2sm(x, w)
    assert glu is None or torch.equal(glu, K.swiglu(y, True))


@pytest.mark.parametrize("t", [1, 3, 4, 64])
def test_chain_of_two_residual_phases(t):
    """Two residual + norm phases in a row update the same residual rows: the second may not do so before the sums of squares of
    the first are formed."""
    K = cu()
    torch.manual_seed(t)
    h, eps = 1024, 1e-6
    w1, w2 = ((torch.randn(h, h, device=DEV) * 0.03).bfloat16() for _ in range(2))
    n1, n2 = ((torch.rand(h, device=DEV) + 0.5).bfloat16() for _ in range(2))
    a, res = torch.randn(t, h, device=DEV).bfloat16(), torch.randn(t, h, device=DEV).bfloat16()
    inv = lambda x: torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)  # noqa: E731
    for _ in range(5):
        r = res.clone()
        o1, o2 = K.decode_chain(a, [(w1, K.CH_RESID_NORM, n1, False), (w2, K.CH_RESID_NORM, n2, False)], residual=r, eps=eps)
        h1 = res.double() + a.double() @ w1.double().t()
        s1 = o1.ssp[:, : o1.parts].double().sum(-1)
        # the residual is rounded to bf16 (2^-9 a value) before it is squared: the sum of 1024 squares is within 2^-8 of the exact one
        assert ((s1 - h1.pow(2).sum(-1)).abs() <= 2 ** -8 * s1).all()
        h2 = h1 + (h1 * inv(h1) * n1.double()) @ w2.double().t()
        err = (r.double() - h2).norm() / h2.norm()
        assert err < 3 * 2 ** -9  # three roundings to bf16: the residual twice, the rows between
        assert ((o2.ssp[:, : o2.parts].double().sum(-1) - r.double().pow(2).sum(-1)).abs() <= 2 ** -16 * r.double().pow(2).sum(-1)).all()
    assert not K.ctx(DEV).chain_counters.any() and K.read_status(DEV) == 0


@pytest.mark.parametrize("t", [1, 4])
def test_chain_that_gives_up_leaves_nothing_behind(t):
    """A chain whose status word is set gives up at a barrier that it has to wait at: counters back at zero, the next launch right."""
    K = cu()
    torch.manual_seed(t)
    w = [(torch.randn(m, k, device=DEV) * 0.03).bfloat16() for m, k in ((1024, 2048), (6144, 1024), (1024, 3072))]
    n1, n2 = ((torch.rand(1024, device=DEV) + 0.5).bfloat16() for _ in range(2))
    a, res = torch.randn(t, 2048, device=DEV).bfloat16(), torch.randn(t, 1024, device=DEV).bfloat16()

    def chain():
        r = res.clone()
        K.decode_chain(a, [(w[0], K.CH_RESID_NORM, n1, False), (w[1], K.CH_SWIGLU, None, False), (w[2], K.CH_RESID_NORM, n2, False)], residual=r, eps=1e-6)
        return r

    want = chain()
    for _ in range(20):
        K.ctx(DEV).status[0] = 2
        chain()
        assert not K.ctx(DEV).chain_counters.any()
        K.clear_status(DEV)
        assert torch.equal(chain(), want) and K.read_status(DEV) == 0


@pytest.mark.parametrize("extras", [False, True])
@pytest.mark.parametrize(
    "heads,rot,window,splits,reps,tc",
    # blocks of 16 heads; of 32 (60 rows of 64 heads) and 64 (120 rows), and a second group of 32 heads
    [(16, 64, 70, 1, 1, True), (64, 64, 70, 3, 1, True), (5, 0, 33, 1, 1, True), (40, 64, 200, 2, 1, True), (64, 0, 64, 16, 1, True), (16, 64, 0, 16, 1, True),
     (64, 64, 70, 1, 5, True), (64, 64, 0, 1, 10, True), (64, 64, 70, 3, 10, True), (96, 64, 130, 2, 10, True), (33, 0, 33, 1, 15, True),
     (16, 64, 70, 1, 1, False), (5, 0, 64, 3, 1, False), (64, 64, 0, 16, 1, False)],
)
def test_latent_window_and_empty_splits(heads, rot, window, splits, reps, tc, extras, monkeypatch):
    """Rows in front of a window and behind the last key hold NaN (pages that others have written since), also with a sink and a gate per
    head, which belong to the joined row; on both kernels (``splits``: how many blocks share a row on the mma.sync kernel, some without
    keys; on tcgen05 how few heads a block gets)."""
    torch.manual_seed(heads + window)
    kv_lens, page, lat, dim, vdim = [1, 63, 64, 65, 0, 129, 200, 511, 1000, 77, 96, 270] * reps, 16, 512, 128, 128
    n = len(kv_lens)
    per = [(x + page - 1) // page for x in kv_lens]
    table, at = torch.zeros(n, max(per), dtype=torch.int32), 1
    for i, m in enumerate(per):
        table[i, :m] = torch.arange(at, at + m)
        at += m
    cache = torch.randn(at * page, lat + rot, device=DEV).bfloat16()
    for i, (x, m) in enumerate(zip(kv_lens, per)):
        rows = (table[i, :m].long()[:, None] * page + torch.arange(page)).flatten().to(DEV)
        cache[rows[x:]] = float("nan")
        if window:  # (the mma.sync kernel reads the tile of 32 keys that a window begins in)
            first = max(0, x - window)
            cache[rows[: first if tc else first // 32 * 32]] = float("nan")
    pos = torch.tensor([max(x - 1, 0) for x in kv_lens], dtype=torch.int32, device=DEV)
    meta = R.AttnMeta(torch.arange(n + 1, dtype=torch.int32, device=DEV), torch.tensor(kv_lens, dtype=torch.int32, device=DEV), table.to(DEV), pos, pos, page, n, n, 1, max(kv_lens), True,
                      list(range(n + 1)), kv_lens)
    q = torch.randn(n, heads * (dim + rot), device=DEV).bfloat16()
    uk_t, uv = (torch.randn(heads, 512, 128, device=DEV) * 0.05).bfloat16(), (torch.randn(heads, vdim, lat, device=DEV) * 0.05).bfloat16()
    q[2] *= 8  # scores that pass the reference value by far in a later tile
    a = torch.randn(2048, max(rot // 2, 1), device=DEV)
    more = dict(head_gate=torch.randn(n, heads, device=DEV).bfloat16(), sink=torch.randn(heads, device=DEV)) if extras else {}
    monkeypatch.setattr(cu(), "_latent_splits", lambda *a: splits)
    monkeypatch.setattr(cu(), "_latent_tc", lambda *a: tc)
    args = (uk_t, uv, None)
    got = cu().latent_attention(q, *args, cache.view(at, -1), meta, rot, 0.07, window, a.cos(), a.sin(), **more)
    want = R.latent_attention(q, *args, torch.nan_to_num(cache).view(at, -1), meta, rot, 0.07, window, a.cos(), a.sin(), **more)
    assert not got[4].any() and torch.isfinite(got.float()).all()
    # weights and outputs of both are rounded to bf16 (2^-8 each), the sums are of some hundred terms: 2^-6 of the largest
    assert (got.float() - want.float()).abs().max() <= 2 ** -6 * want.float().abs().max()
    assert cu().read_status(DEV) == 0


def _latent_rows(kv_lens, heads, seed, q_lens=None, page=16, lat=512, rot=64, dim=128):
    """A decode step (or rows of up to 16 tokens) over scattered pages: (meta of chosen sequences, q, up-projections, cache, angles)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    q_lens = q_lens or [1] * len(kv_lens)
    per = [(x + page - 1) // page for x in kv_lens]
    order = (torch.randperm(sum(per), device=DEV, generator=g) + 1).int().cpu()
    table, at = torch.zeros(len(kv_lens), max(per), dtype=torch.int32), 0
    for i, m in enumerate(per):
        table[i, :m] = order[at : at + m]
        at += m
    draw = lambda *shape: torch.randn(*shape, device=DEV, generator=g)  # noqa: E731

    def meta(rows):
        n, ql, kl = len(rows), [q_lens[i] for i in rows], [kv_lens[i] for i in rows]
        qi = torch.tensor([0] + ql).cumsum(0)
        pos = torch.cat([torch.arange(k - m, k).clamp(min=0) for k, m in zip(kl, ql)]).int().to(DEV)
        return R.AttnMeta(qi.int().to(DEV), torch.tensor(kl, dtype=torch.int32, device=DEV), table[rows].to(DEV), pos, pos, page, n, sum(ql), max(ql), max(kl), max(ql) == 1, qi.tolist(), kl)

    angles = draw(max(kv_lens) + 1, max(rot // 2, 1))
    return (meta, draw(sum(q_lens), heads * (dim + rot)).bfloat16(), (draw(heads, lat, dim) * 0.05).bfloat16(), (draw(heads, dim, lat) * 0.05).bfloat16(), draw(sum(per) + 1, page * (lat + rot)).bfloat16(),
            (angles.cos(), angles.sin()))


@pytest.mark.parametrize("heads,rot", [(16, 64), (64, 64), (64, 0)])
def test_latent_rows_whatever_shares_their_step(heads, rot):
    """Under the batch-invariant policy a latent decode row has the same bytes alone, beside rows of other lengths and behind a prompt."""
    K = cu()
    kv_lens = [700, 1500, 300, 40, 2000, 3001, 257, 256, 65]
    n = len(kv_lens)
    meta, q, uk_t, uv, cache, cs = _latent_rows(kv_lens + [90], heads, 3, [1] * n + [50], rot=rot)
    uk, turn = uk_t.transpose(1, 2).contiguous(), R.rope_tables(4096, 64, 1e4, torch.bfloat16, DEV)
    before = K.batch_invariant()
    K.set_batch_invariant(True)
    try:
        def run(seqs, x):
            m = meta(seqs)
            y = K.latent_attention(x, uk_t, uv, None, cache, m, rot, 0.07, 0, *cs)
            return torch.cat([y, K.mla_attention(K.mla_rope_q(x.view(-1, heads, 192), *turn, m, 128), uk, uv, cache.view(-1, 16, 576), m, 0.07, 512)], 1) if rot else y

        step, beside = run(list(range(n)), q[:n]), run([n] + list(range(n)), torch.cat([q[n:], q[:n]]))[50:]
        for i in range(n):
            alone = run([i], q[i : i + 1])[0]
            assert torch.equal(step[i], alone) and torch.equal(beside[i], alone), kv_lens[i]
    finally:
        K.set_batch_invariant(before)


@pytest.mark.parametrize("kv_lens,heads", [([40, 200], 16), ([40, 700], 16), ([700] * 64, 64), ([300] * 513, 16)])
def test_latent_launches_are_counted(kv_lens, heads):
    """``launch_count`` against the kernels of a captured graph: steps of short rows, rows that may be cut (with the kernel that joins
    them), and too many for that."""
    K, driver = cu(), ctypes.CDLL("libcuda.so.1")
    meta, q, uk_t, uv, cache, cs = _latent_rows(kv_lens, heads, 4)
    m = meta(list(range(len(kv_lens))))
    uk = uk_t.transpose(1, 2).contiguous()
    hq = K.mla_rope_q(q.view(len(kv_lens), heads, 192), *R.rope_tables(1024, 64, 1e4, torch.bfloat16, DEV), m, 128)
    for call in (lambda: K.latent_attention(q, uk_t, uv, None, cache, m, 64, 0.07, 0, *cs), lambda: K.mla_attention(hq, uk, uv, cache.view(-1, 16, 576), m, 0.07, 512)):
        call()
        torch.cuda.synchronize()
        graph, n0 = torch.cuda.CUDAGraph(keep_graph=True), K.launch_count(DEV)
        with torch.cuda.graph(graph):
            call()
        nodes = ctypes.c_size_t()
        assert driver.cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(nodes)) == 0
        assert nodes.value >= 3 and K.launch_count(DEV) - n0 == nodes.value  # kernels are all that is captured


_SHARED_ROWS = {
    "long": [20000, 1, 0, 300, 65],  # 78 pieces of a row: more than a warp has lanes
    "longest first and last": [9000, 0, 64, 0, 12345],
    "lines": [256, 257, 320, 0, 255, 64, 0, 0, 321, 319] * 3,  # rows of four tiles stay whole, rows of five may be cut
    "wave": [700] * 150 + [0, 3000],
    "most": [270] * 511 + [5000],  # the most rows that are shared
    "more": [270] * 512 + [5000],  # and one more
}


@pytest.mark.parametrize("heads,rot,window,extras", [(16, 64, 0, False), (64, 64, 0, True), (96, 0, 0, False), (40, 64, 3000, True), (16, 0, 130, False)])
@pytest.mark.parametrize("lens", _SHARED_ROWS)
def test_latent_rows_that_blocks_share(lens, heads, rot, window, extras, monkeypatch):
    """Rows cut between blocks, few pieces and many, against the restatement and against whole rows; the same bytes every time."""
    K, kv_lens = cu(), _SHARED_ROWS[lens]
    meta, q, uk_t, uv, cache, cs = _latent_rows(kv_lens, heads, heads, rot=rot)
    n = len(kv_lens)
    m = meta(list(range(n)))
    q[n // 2] *= 8  # scores that pass the reference value by far in a later tile
    g = torch.Generator(device=DEV).manual_seed(1)
    more = dict(head_gate=torch.randn(n, heads, device=DEV, generator=g).bfloat16(), sink=torch.randn(heads, device=DEV, generator=g)) if extras else {}
    run = lambda f: f(q, uk_t, uv, None, cache, m, rot, 0.07, window, *cs, **more).float()  # noqa: E731
    got, want = run(K.latent_attention), run(R.latent_attention)
    monkeypatch.setattr(K, "_latent_scratch", lambda part, longest: 0)
    whole = run(K.latent_attention)
    monkeypatch.undo()
    # weights and rows of all are rounded to bf16 (2^-8 each), the sums are of some hundred terms that matter: 2^-6 of a row's largest
    lim = 2 ** -6 * want.abs().amax(-1, keepdim=True)
    assert ((got - want).abs() <= lim).all() and ((got - whole).abs() <= lim).all() and torch.equal(got, run(K.latent_attention))
    short = torch.tensor([x <= 256 for x in kv_lens], device=DEV)
    assert torch.equal(got[short], whole[short]) and not got[[i for i, x in enumerate(kv_lens) if x == 0]].any()
    assert K.read_status(DEV) == 0


@pytest.mark.parametrize("heads", [16, 64])
def test_latent_rows_behind_prompts_are_shared(heads):
    """Decode rows, long ones among them, behind a prompt that takes the expanded form."""
    K, kv_lens, q_lens = cu(), [200, 700, 4000, 100, 9000, 1], [128, 72, 1, 1, 1, 1]
    meta, q, uk_t, uv, cache, cs = _latent_rows(kv_lens, heads, 7, q_lens)
    m, calls = meta(list(range(6))), K.PREFILL_TC_CALLS["latent"]
    ukv = torch.cat([uk_t.transpose(1, 2).reshape(heads * 128, 512), uv.reshape(heads * 128, 512)])
    got, want = (f(q.clone(), uk_t, uv, ukv, cache, m, 64, 0.07, 0, *cs).float() for f in (K.latent_attention, R.latent_attention))
    assert K.PREFILL_TC_CALLS["latent"] == calls + 1
    assert ((got - want).abs() <= 2 ** -6 * want.abs().amax(-1, keepdim=True)).all()  # as above


@pytest.mark.parametrize("heads", [16, 64])
def test_latent_rows_in_a_graph_with_a_bound(heads):
    """A captured step knows a bound on its rows' keys only: short rows have the bytes of a step whose lengths are known, others those of a
    step with the bound."""
    K, kv_lens = cu(), [1, 64, 65, 200, 256, 0, 129, 1000, 3000]
    meta, q, uk_t, uv, cache, cs = _latent_rows(kv_lens, heads, 9)
    n = len(kv_lens)
    run = lambda m: K.latent_attention(q[: m.num_seqs], uk_t, uv, None, cache, m, 64, 0.07, 0, *cs)  # noqa: E731
    known, bound = meta(list(range(7))), meta(list(range(7)))
    bound.max_kv_len = 4096
    bound.h_kv_lens = bound.h_q_indptr = None
    assert torch.equal(run(known), run(bound))
    m = meta(list(range(n)))
    m.max_kv_len = 4096
    m.h_kv_lens = m.h_q_indptr = None
    eager, real = run(m), m.kv_lens.clone()
    m.kv_lens.fill_(1)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run(m)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run(m)
    m.kv_lens.copy_(real)
    graph.replay()
    assert torch.equal(out, eager)


@pytest.mark.parametrize("lens,past,heads,tc", [([1] * 8, 7, 16, True), ([1] * 150, 100, 16, True), ([16] * 3, 0, 16, True), ([17] * 3, 0, 16, False), ([80], 0, 16, False), ([90], 0, 16, True),
                                                 ([20] * 10, 80, 16, False), ([20] * 10, 130, 16, True), ([20] * 10, 15, 64, False), ([20] * 10, 30, 64, True), ([300] * 3, 0, 32, True)])
def test_latent_kernels_where_the_rule_changes(lens, past, heads, tc, monkeypatch):
    """The rows on either side of each line of the rule, on the kernel that it names, against the restatement."""
    torch.manual_seed(past + heads)
    monkeypatch.setattr(cu(), "_PREFILL_TC", False)
    n, page, kv_lens = len(lens), 16, [x + past for x in lens]
    qi = torch.tensor([0] + lens).cumsum(0)
    per = max((x + page - 1) // page for x in kv_lens)
    table = torch.randperm(n * per).view(n, per).to(torch.int32).to(DEV)
    pos = torch.cat([torch.arange(past, x) for x in kv_lens]).to(torch.int32).to(DEV)
    t, decode = sum(lens), max(lens) == 1
    meta = R.AttnMeta(qi.to(torch.int32).to(DEV), torch.tensor(kv_lens, dtype=torch.int32, device=DEV), table, pos, pos, page, n, t, max(lens), max(kv_lens), decode, qi.tolist(), kv_lens)
    assert cu()._latent_tc(t, heads, 512, 64, cu()._latent_keys(meta), max(lens), 148) == tc
    cache = torch.randn(n * per, page, 576, device=DEV).bfloat16()
    q = torch.randn(t, heads, 192, device=DEV).bfloat16()
    uk, uv = (torch.randn(heads, 128, 512, device=DEV) * 0.05).bfloat16(), (torch.randn(heads, 128, 512, device=DEV) * 0.05).bfloat16()
    cos, sin = R.rope_tables(2048, 64, 1e4, torch.bfloat16, DEV)
    got = cu().mla_attention(cu().mla_rope_q(q, cos, sin, meta, 128), uk, uv, cache, meta, 0.07, 512)
    want = R.mla_attention(R.mla_rope_q(q, cos, sin, meta, 128), uk, uv, cache, meta, 0.07, 512)
    assert (got.float() - want.float()).abs().max() <= 2 ** -6 * want.float().abs().max()  # as above
    assert cu().read_status(DEV) == 0


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("rows", [3, 70, 290])  # decode rows beside the prompts: up to and above the 256 sequences that are ranked by length
def test_gated_delta_prompts_beside_decode_rows(rows, known):
    """Prompts of one to six chunks among decode rows, empty sequences and one without a state: every sequence's bytes are those of a
    step of its own, whichever kernel takes it."""
    torch.manual_seed(rows)
    lens = [200, 64, 0, 129, 128, 330, 32, 129] + [1] * rows + [260, 31, 100]
    slots = list(range(1, len(lens) + 1))
    slots[3] = -1
    meta = _state_meta(lens, slots)
    hk, hv, dk, dv, t = 2, 4, 128, 128, sum(lens)
    x = torch.randn(t, 2 * hk * dk + hv * dv, device=DEV).bfloat16()
    q, k, v = (y.view(t, -1, d) for y, d in zip(x.split([hk * dk, hk * dk, hv * dv], 1), (dk, dk, dv)))
    g, beta = -torch.rand(t, hv, device=DEV), torch.rand(t, hv, device=DEV)
    s0 = torch.randn(len(lens) + 2, hv, dk, dv, device=DEV) * 0.1
    s = s0.clone()
    meta.h_q_indptr = meta.q_indptr.tolist() if known else None
    out, at = cu().gdn_recurrent(q, k, v, g, beta, s, meta, chunked=True), 0
    for i, n in enumerate(lens):
        sl = slice(at, at + n)
        at += n
        if n < 32 and i != 8 or slots[i] < 0:
            continue
        alone, one = s0.clone(), _state_meta([n], [slots[i]])
        y = cu().gdn_recurrent(q[sl], k[sl], v[sl], g[sl], beta[sl], alone, one, chunked=n >= 32)
        if n >= 32:
            assert torch.equal(out[sl], y) and torch.equal(s[slots[i]], alone[slots[i]]), i
        else:  # (a decode row among prompts may sum in another order: the limits of one f32 step, rounded to bf16)
            assert (out[sl].float() - y.float()).abs().max() <= 2 ** -7 * y.float().abs().max()
    assert torch.equal(s[0], s0[0]) and torch.equal(s[4], s0[4]) and torch.equal(s[3], s0[3])  # no one's, the stateless one's, the empty one's


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("lens", [[1] * 5 + [200], [16, 1, 8, 9, 3, 13, 1, 0, 40], [4, 1, 5], [200, 16, 16], [120, 130], [15, 127, 128, 500, 1, 129, 9], [1500] + [20] * 15])
def test_kda_rows_beside_prompts(lens, known):
    """Sequences below the blocks' shortest go token by token, whatever shares their step: decode rows beside prompts have the bytes of a
    step of decode rows, prompts those of a step of their own."""
    K = cu()
    torch.manual_seed(sum(lens))
    heads, dk, dv, t, slots = 3, 128, 128, sum(lens), list(range(1, len(lens) + 1))
    qkv = torch.randn(t, 3 * heads * dk, device=DEV).bfloat16()
    q, k, v = (qkv[:, j * heads * dk : (j + 1) * heads * dk].view(t, heads, dk) for j in range(3))
    f, b = torch.randn(t, heads * dk, device=DEV).bfloat16(), torch.randn(t, heads, device=DEV).bfloat16()
    a_log, dt = torch.randn(heads, device=DEV) * 0.5, torch.randn(heads * dk, device=DEV) - 2
    s0 = torch.randn(len(lens) + 1, heads, dk, dv, device=DEV)

    def run(rows, lens, slots, known):
        meta, s = _state_meta(lens, slots), s0.clone()
        meta.h_q_indptr = meta.q_indptr.tolist() if known else None
        return K.kda_recurrent(q[rows], k[rows], v[rows], f[rows], b[rows], a_log, dt, -5.0, s, meta), s

    out, s = run(slice(0, t), lens, slots, known)
    short, at = max((n for n in lens if n < K._KDA_BLOCK_MIN), default=0), 0
    for n, slot in zip(lens, slots):
        rows = slice(at, at + n)
        at += n
        if n == 0:
            assert torch.equal(s[slot], s0[slot])
            continue
        y, alone = run(rows, [n], [slot], True)
        if n >= K._KDA_BLOCK_MIN or (known and (short <= 4) == (n <= 4)):
            assert torch.equal(out[rows], y) and torch.equal(s[slot], alone[slot])
        else:  # beside rows of five tokens and more the sums of a column are formed in another order: f32, then one rounding to bf16
            assert (out[rows].float() - y.float()).abs().max() <= 2 ** -8 * y.float().abs().max() + 1e-5
            assert (s[slot] - alone[slot]).abs().max() <= 2 ** -17 * alone[slot].abs().max()


@pytest.mark.parametrize("switch,takes", [({}, "11"), ({"PEGAINFER_GEMM_2SM_MAXK": "8192"}, "10"), ({"PEGAINFER_GEMM_2SM_MAXK": "0"}, "11"), ({"PEGAINFER_GEMM_2SM": "0"}, "00")])
def test_two_sm_gemm_switches(switch, takes):
    """The two-SM kernel's switches, read once per process: off, and the longest k that it takes."""
    code = "from pegainfer_b200 import _native as n; print(n.load().pg_gemm2sm_takes(100, 1024, 8192), n.load().pg_gemm2sm_takes(100, 1024, 8256), sep='')"
    env = {k: v for k, v in os.environ.items() if not k.startswith("PEGAINFER_GEMM_2SM")}
    assert subprocess.run([sys.executable, "-c", code], env=env | switch, capture_output=True, text=True, timeout=300).stdout.strip() == takes


def test_gdn_conv1d_beside_many_sequences():
    """Prompts beside so many decode rows that the segments are longer."""
    torch.manual_seed(0)
    q_lens = [70, 1, 33] + [1] * 400 + [64, 65, 2]
    channels, n = 10240, len(q_lens)
    meta = _state_meta(q_lens, list(range(1, n + 1)))
    x = torch.randn(sum(q_lens), channels, device=DEV).bfloat16()
    w = (torch.randn(channels, 4, device=DEV) * 0.5).bfloat16()
    st1 = torch.randn(n + 1, channels, 3, device=DEV).bfloat16()
    st2 = st1.clone()
    y1, y2 = cu().gdn_conv1d(x, w, st1, meta), R.gdn_conv1d(x, w, st2, meta)
    assert ((y1.float() - y2.float()).abs() <= 2 ** -7 * y2.float().abs() + 2 ** -9).all()  # as above
    assert torch.equal(st1, st2)


@pytest.mark.parametrize("channels,seqs", [(1040, 6), (2048, 976), (2048, 978)])  # one channel per thread; either side of two million channels
def test_gdn_conv1d_rows(channels, seqs):
    torch.manual_seed(seqs)
    q_lens = ([1, 2, 3, 4, 1, 1] * seqs)[:seqs]
    meta = _state_meta(q_lens, [-1] + list(range(1, seqs)))
    x, w = torch.randn(sum(q_lens), channels, device=DEV).bfloat16(), (torch.randn(channels, 4, device=DEV) * 0.5).bfloat16()
    st1 = torch.randn(seqs, channels, 3, device=DEV).bfloat16()
    st2 = st1.clone()
    y1, y2 = cu().gdn_conv1d(x, w, st1, meta), R.gdn_conv1d(x, w, st2, meta)
    assert ((y1.float() - y2.float()).abs() <= 2 ** -7 * y2.float().abs() + 2 ** -9).all()  # as above
    assert torch.equal(st1, st2)


@pytest.mark.parametrize("m,k,bn,aligned", [(128, 64, 16, True), (200, 128, 16, True), (136, 320, 32, True), (256, 256, 48, True), (384, 1024, 128, True), (130, 768, 64, False), (300, 2048, 128, True)])
def test_int4_experts_of_ragged_rows(m, k, bn, aligned):
    """Weight rows and k around tiles of 128 and stages of 256, several token tiles and empty experts, scales that TMA can read or not."""
    torch.manual_seed(m + k)
    rows = [0, 1, bn, bn + 1, 2 * bn - 1, 0, 3]
    e, t = len(rows), sum(rows)
    x = torch.randn(t, k, device=DEV).bfloat16()
    packed = torch.randint(-(2 ** 31), 2 ** 31 - 1, (e, m, k // 8), dtype=torch.int32, device=DEV)
    buf = (torch.rand(e * m * k // 32 + 1, device=DEV) * 0.01 + 0.001).bfloat16()
    scales = (buf[:-1] if aligned else buf[1:]).view(e, m, k // 32)
    offsets = torch.tensor([0] + rows).cumsum(0).to(torch.int32).to(DEV)
    got, at = cu().grouped_gemm(x, offsets, packed, scales, bn), 0
    for i, n in enumerate(rows):
        a, w = x[at : at + n].double(), R.dequant_int4_g32(packed[i], scales[i]).double()
        # products of bf16 are exact; f32 sums of k terms, one rounding to bf16
        bound = 2 ** -8 * (a @ w.T).abs() + k * 2 ** -23 * (a.abs() @ w.abs().T)
        assert ((got[at : at + n].double() - a @ w.T).abs() <= bound).all()
        at += n
    assert cu().read_status(DEV) == 0


@pytest.mark.parametrize("where", ["k", "v", "f", "b", "q"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_kda_numbers_that_are_none_stay_behind_their_token(where, value):
    """Tokens in front of one that is not a number, and other heads and sequences, have the values that they have without it."""
    K = cu()
    torch.manual_seed(5)
    heads, dk, dv, lens, bad = 3, 128, 128, [400, 30, 450], 430 + 30  # the last sequence's token 30, in its second chunk
    meta, t = _state_meta(lens, [1, 2, 3]), sum(lens)
    x = {n: torch.randn(t, heads, dk, device=DEV).bfloat16() for n in "qkv"}
    x["f"], x["b"] = torch.randn(t, heads * dk, device=DEV).bfloat16(), torch.randn(t, heads, device=DEV).bfloat16()
    a_log, dt = torch.randn(heads, device=DEV) * 0.5, torch.randn(heads * dk, device=DEV) - 2
    s0 = torch.randn(4, heads, dk, dv, device=DEV)

    def run():
        s = s0.clone()
        return K.kda_recurrent(*(x[n] for n in "qkvfb"), a_log, dt, -5.0, s, meta), s

    want, ws = run()
    (x[where][bad, 1] if where in "qkv" else x[where][bad])[1 if where == "b" else 130 if where == "f" else 2] = value
    got, gs = run()
    others = [0, 2]
    assert torch.equal(got[:, others], want[:, others]) and torch.equal(gs[:, others], ws[:, others])
    assert torch.equal(got[:430], want[:430]) and torch.equal(gs[:3], ws[:3])
    # the chunk of the token may be summed in another order: f32, then one rounding to bf16
    assert (got[430:bad].float() - want[430:bad].float()).abs().max() <= 2 ** -8 * want.float().abs().max() + 1e-5
    if where in "kv" or value != value and where != "q":
        assert not torch.isfinite(got[bad:, 1].float()).all(-1).any() and not torch.isfinite(gs[3, 1]).all()
    else:  # an infinite gate is a decay or a step of its own, a query is no one else's
        assert torch.isfinite(gs).all() and torch.isfinite(got[bad + 1 :].float()).all()


@pytest.mark.parametrize("lower", [-5.0, -5.25, -5.5])
@pytest.mark.parametrize("shift", [6.0, -6.0, 0.0])  # decays near exp(lower), near one, both
def test_kda_prompts_of_strong_and_weak_decays(lower, shift):
    torch.manual_seed(int(shift) + 20)
    heads, dk, dv, q_lens = 2, 128, 128, [15, 16, 17, 31, 48, 400, 401]
    meta, t, n = _state_meta(q_lens, list(range(1, len(q_lens) + 1))), sum(q_lens), len(q_lens)
    q, k, v = (torch.randn(t, heads, dk, device=DEV).bfloat16() for _ in range(3))
    f, b = (torch.randn(t, heads * dk, device=DEV) * (8 if shift == 0 else 1) + shift).bfloat16(), torch.randn(t, heads, device=DEV).bfloat16()
    a_log, dt = torch.zeros(heads, device=DEV), torch.zeros(heads * dk, device=DEV)
    st1 = torch.randn(n + 1, heads, dk, dv, device=DEV)
    st2 = st1.double()
    o1 = cu().kda_recurrent(q, k, v, f, b, a_log, dt, lower, st1, meta)
    unit = lambda x: x * torch.rsqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    qd, kd = unit(q.double()) * dk ** -0.5, unit(k.double())
    dec, beta, at = torch.exp(lower * torch.sigmoid(f.double().view(t, heads, dk))), torch.sigmoid(b.double()), 0
    for s, m in enumerate(q_lens):
        S = st2[s + 1]
        for i in range(at, at + m):
            S = S * dec[i].unsqueeze(-1)
            d = (v[i].double() - torch.einsum("hkv,hk->hv", S, kd[i])) * beta[i].unsqueeze(-1)
            S = S + kd[i].unsqueeze(-1) * d.unsqueeze(1)
            want = torch.einsum("hkv,hk->hv", S, qd[i])
            # bf16 output; f32 sums of 128 channels and 16 tokens, 2^-23 a step
            assert (o1[i].double() - want).abs().max() <= 2 ** -8 * want.abs().max() + 1e-5
        st2[s + 1] = S
        at += m
    assert (st1.double() - st2).abs().max() < 2 ** -17 * st2.abs().max()
    if shift > 0:  # a state of a few tokens at most, each a product or two in f32: within its unit in the last place on average
        assert (st1.double() - st2)[1:].norm() <= 2 ** -23 * st2[1:].norm()


@pytest.mark.parametrize("n,m", [(5, 130), (59, 128), (60, 136), (117, 48), (118, 32)])  # around four of five SMs
@pytest.mark.parametrize("t", [1, 17, 64, 65, 129])
def test_products_per_head_where_token_tiles_narrow(t, n, m):
    g = torch.Generator().manual_seed(t * 1000 + m)
    k = 72
    x, w = torch.randn(t, n, k, generator=g).bfloat16(), torch.randn(n, m, k, generator=g).bfloat16()
    y = cu().multi_dense(x.to(DEV), w.to(DEV)).cpu().double()
    want, size = torch.einsum("tnk,nmk->tnm", x.double(), w.double()), torch.einsum("tnk,nmk->tnm", x.double().abs(), w.double().abs())
    # one rounding to bf16 of a sum of k products in f32
    assert ((y - want).abs() <= 2 ** -8 * want.abs() + k * 2 ** -23 * size).all()
