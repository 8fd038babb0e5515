"""Paged decode over the ways in which a launch spreads the contexts (clusters of up to 16 CTAs of 4 or 8 warps, single
CTAs, chunks with a combining kernel), at lengths around their edges, against the CPU oracle."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native
from hipkittens_b200.synthetic import make_paged_inputs
from oracle.attn_oracle import paged_decode_oracle

pytestmark = pytest.mark.gpu

CASES = [
    # H, H_KV, launches, context lengths (the first is the table's width)
    (8, 8, 1, [3250]),                                     # clusters of 16 CTAs of 4 warps
    (8, 1, 1, [4097, 0, 64]),                              # 16 CTAs of 8 warps
    (16, 2, 1, [16384, 129, 8192]),                        # ... at its longest
    (8, 1, 2, [16400, 513, 100]),                          # a table beyond that: chunks
    (3, 1, 1, [100]),                                      # fewer pages than warps in a cluster of 16
    (32, 8, 1, [1000, 1, 16, 17, 64, 65, 1024]),           # clusters that leave some of their CTAs without a page
    (28, 4, 1, [2048, 2047, 33] + [5 * i for i in range(9)]),
    (16, 16, 1, [2560] + [1 + 300 * i for i in range(8)]),  # single CTAs of 8 warps, contexts of 0 to 160 pages
    (16, 16, 2, [2561] + [1 + 300 * i for i in range(8)]),
    (64, 16, 1, [1024] + [50 * i for i in range(18)]),     # single CTAs of 4 warps
]


@pytest.mark.parametrize("h,hkv,launches,lens", CASES)
def test_every_way_to_spread_a_context(h, hkv, launches, lens):
    dev = torch.device("cuda:0")
    top = max(lens)
    q, kp, vp, bt, _ = make_paged_inputs(len(lens), h, hkv, 128, 16, len(lens) * ((top + 15) // 16) + 3, top, top, seed=h)
    ctx = torch.tensor(lens, dtype=torch.int32)
    o = torch.full(q.shape, float("nan"), dtype=torch.bfloat16, device=dev)
    lse = torch.full((len(lens), h, 1, 1), float("nan"), device=dev)
    # the clusters leave the workspace alone, the chunks find it full of NaN
    ws = torch.full((hk.paged_decode_workspace_bytes(len(lens), h, 128, bt.shape[1]),), 255, dtype=torch.uint8, device=dev)
    args = [x.to(dev) for x in (q, kp, vp, bt, ctx)]
    hk.paged_decode(*args, out=o, lse=lse, workspace=ws)
    before = hk.kernel_launch_count()
    hk.paged_decode(*args, out=o, lse=lse, workspace=ws)
    assert hk.kernel_launch_count() - before == launches
    assert _native.device_status(0) == 0
    live = [i for i, n in enumerate(lens) if n > 0]
    o_ref, l_ref = paged_decode_oracle(q[live], kp, vp, bt[live], ctx[live])
    assert float((o.cpu()[live].float() - o_ref.float()).abs().max()) <= 2e-2
    assert float((lse.cpu()[live] - l_ref).abs().max()) <= 1e-3
    for i, n in enumerate(lens):
        if n == 0:  # defined output for an empty context
            assert not o[i].any() and bool(torch.isneginf(lse[i]).all())
