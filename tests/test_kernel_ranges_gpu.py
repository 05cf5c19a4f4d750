"""Kernels at the edges of the ranges that their launch rules draw: tile and segment edges, remainders, odd widths, the
smallest and largest sizes, against the PyTorch restatements."""
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


@pytest.mark.parametrize("routes,e0,e_local,total", [(1, 0, 1, 1), (31, 0, 3, 5), (512, 8, 64, 96), (513, 0, 384, 384), (8193, 16, 48, 384), (40007, 0, 512, 512)])
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
