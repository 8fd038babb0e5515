"""One long context among short ones: how a launch spreads the contexts bounds what one CTA may meet, and the long context is
right whichever way it goes."""
import ctypes

import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native
from hipkittens_b200.synthetic import make_paged_inputs
from oracle.attn_oracle import paged_decode_oracle

# clusters of 2, 3, ... 16 CTAs of 4 warps that a GPU of 148 SMs may hold
HELD = [148, 94, 70, 56, 46, 41, 34, 30, 28, 24, 22, 20, 18, 16, 14]


def shape(S, H_KV, pages):
    held, warps = (ctypes.c_int * 17)(0, 0, *HELD), ctypes.c_int()
    return hk.capi().hk_selftest_decode_shape(S, H_KV, pages, 148, held, 6, ctypes.byref(warps)), warps.value


# us, one long context among others of 100 tokens: chunks / what the launch took without the bound
@pytest.mark.parametrize("S,H_KV,pages", [(8, 8, 500),    # 12.6 / 20.1
                                          (12, 8, 157),   # 10.9 / 16.7
                                          (32, 8, 125),   # 10.8 / 14.0
                                          (64, 1, 512)])  # 10.2 / 19.1
def test_tables_too_wide_for_one_cluster_take_chunks(native_built, S, H_KV, pages):
    assert shape(S, H_KV, pages)[0] == 0


def test_the_most_that_one_cta_may_meet(native_built):
    for S, H_KV in [(1, 8), (2, 8), (3, 8), (4, 8), (40, 1), (6, 8), (8, 8), (64, 1), (90, 1)]:  # clusters of 4-warp CTAs
        size = max(n + 2 for n, held in enumerate(HELD) if held >= S * H_KV)
        most = 44 if size == 16 else 64
        assert shape(S, H_KV, most * size) == (size, 4) and shape(S, H_KV, most * size + 1)[0] == 0
        assert shape(S, H_KV, 1) == (1, 4)  # no CTA without a page
    # CTAs of their own: (warps, the widest table); one wave also where the chunks need more than two
    for S, H_KV, by_width in [(12, 8, {48: 8, 96: 8, 97: 0, 160: 0}), (9, 16, {48: 8, 96: 8, 131: 0, 132: 8, 160: 8, 161: 0}),
                              (32, 8, {64: 4, 65: 8, 96: 8, 97: 0}), (37, 8, {64: 4, 65: 8, 97: 0}),
                              (19, 16, {64: 4, 65: 4, 80: 4, 81: 0}), (64, 16, {80: 4, 81: 0, 8192: 0})]:
        for pages, warps in by_width.items():
            assert shape(S, H_KV, pages) == ((1, warps) if warps else (0, 4)), (S, H_KV, pages)
    assert shape(1, 1, 257) == (16, 8) and shape(6, 1, 1024) == (16, 8) and shape(6, 1, 1025)[0] == 0
    # no warp has more than 32 pages, which are its lanes' ids
    for S in (1, 6, 7, 16, 40, 72, 100, 148, 149, 296, 297, 1000):
        for pages in range(1, 1100):
            cluster, warps = shape(S, 1, pages)
            assert cluster == 0 or pages <= 32 * warps * cluster
    assert shape(0, 1, 1)[0] < 0 and shape(1, 1, 8193)[0] < 0


# (S, H, H_KV, tokens of the long context, launches): on both sides of the lines for clusters, single CTAs of 8 and of 4 warps
@pytest.mark.gpu
@pytest.mark.parametrize("S,H,H_KV,top,launches", [
    (8, 16, 8, 2560, 1), (8, 16, 8, 8000, 2), (12, 16, 8, 1536, 1), (12, 16, 8, 1537, 2), (32, 24, 8, 1024, 1),
    (32, 24, 8, 1025, 1), (32, 24, 8, 1537, 2), (64, 8, 8, 1280, 1), (64, 8, 8, 1281, 2)])
def test_a_long_context_among_short_ones(S, H, H_KV, top, launches):
    dev = torch.device("cuda:0")
    lens = [1 + 7 * i for i in range(S)]
    lens[S // 2] = top
    q, kp, vp, bt, _ = make_paged_inputs(S, H, H_KV, 128, 16, S * 30 + (top + 15) // 16, 1, 1, seed=S)
    need = [(n + 15) // 16 for n in lens]
    ids = torch.randperm(kp.shape[0], generator=torch.Generator().manual_seed(top)).to(torch.int32)
    bt, at = torch.zeros(S, max(need), dtype=torch.int32), 0
    for i, n in enumerate(need):
        bt[i, :n] = ids[at:at + n]
        at += n
    ctx = torch.tensor(lens, dtype=torch.int32)
    args = [x.to(dev) for x in (q, kp, vp, bt, ctx)]
    o, lse = hk.paged_decode(*args)
    before = hk.kernel_launch_count()
    o2, lse2 = hk.paged_decode(*args)
    assert hk.kernel_launch_count() - before == launches
    assert _native.device_status(0) == 0 and torch.equal(o, o2) and torch.equal(lse, lse2)
    o_ref, l_ref = paged_decode_oracle(q, kp, vp, bt, ctx)
    assert float((o.cpu().float() - o_ref.float()).abs().max()) <= 2e-2
    assert float((lse.cpu() - l_ref).abs().max()) <= 1e-3
