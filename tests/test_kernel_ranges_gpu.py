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
