"""Decode over chunks, which a second kernel combines, and over clusters, in a chain of dependent launches and in a CUDA graph:
what both give is what the same calls give one by one."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native
from hipkittens_b200.synthetic import make_paged_inputs
from oracle.attn_oracle import paged_decode_oracle

pytestmark = pytest.mark.gpu


def launches(call):
    before = hk.kernel_launch_count()
    call()
    return hk.kernel_launch_count() - before


# a block table of more than 1024 pages has few units take chunks; the same contexts in a narrow one take clusters
@pytest.mark.parametrize("pages,kernels", [(1040, 2), (290, 1)])
def test_decode_steps_in_a_chain(pages, kernels):
    """The combine kernel merges partials of the split kernel before it while the append of the next step stands behind it; the
    workspace is one and the same, and every step's query is the result of the step before."""
    gen = torch.Generator("cuda").manual_seed(13)
    b, h, hkv = 3, 16, 2
    start0 = torch.tensor([700, 2100, 4500], dtype=torch.int32, device="cuda")
    pool0 = [torch.randn(b * 290, 16, hkv, 128, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]
    table = torch.zeros(b, pages, dtype=torch.int32, device="cuda")
    table[:, :290] = torch.randperm(b * 290, device="cuda", generator=gen).to(torch.int32).reshape(b, 290)
    workspace = torch.empty(hk.paged_decode_workspace_bytes(b, h, 128, pages), dtype=torch.uint8, device="cuda")
    angle = torch.rand(290 * 16, 64, device="cuda", generator=gen)
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
    q0 = torch.randn(b, 1, h, 128, device="cuda", generator=gen).to(torch.bfloat16)
    assert launches(lambda: hk.paged_decode(q0, *pool0, table, start0, workspace=workspace)) == kernels

    def chain(sync):
        k, v = (p.clone() for p in pool0)
        q, seen = q0, []
        for i in range(40):
            start = start0 + i
            hk.paged_kv_append_rotary(q[:, :, :hkv].contiguous(), q[:, :, hkv:2 * hkv].contiguous(), k, v, table, start,
                                      cos, sin)
            if sync:
                torch.cuda.synchronize()
            q, lse = hk.paged_decode(q, k, v, table, start + 1, workspace=workspace)
            if sync:
                torch.cuda.synchronize()
            seen += [q, lse]
        return seen

    for a, b_ in zip(chain(False), chain(True)):
        assert torch.equal(a, b_)
    assert _native.device_status(0) == 0


# (S, H, H_KV, longest context, pages of the table): few units with a wide table, more units than clusters hold, clusters
@pytest.mark.parametrize("S,H,H_KV,top,pages,kernels", [(3, 16, 2, 1500, 1100, 2), (20, 32, 8, 1700, 107, 2),
                                                        (3, 16, 2, 1500, 94, 1)])
def test_replays_from_a_cuda_graph(S, H, H_KV, top, pages, kernels):
    """The launches go onto the capturing stream, and a replay after the query, the lengths and the table have changed in place
    gives the same bits as an eager call."""
    dev = torch.device("cuda:0")
    q, kp, vp, bt, cl = make_paged_inputs(S, H, H_KV, 128, 16, S * 107, 100, top, seed=12)
    table = torch.zeros(S, pages, dtype=torch.int32)
    table[:, :bt.shape[1]] = bt
    q, kp, vp, table, cl = (t.to(dev) for t in (q, kp, vp, table, cl))
    ws = torch.empty(hk.paged_decode_workspace_bytes(S, H, 128, pages), dtype=torch.uint8, device=dev)
    o, lse = torch.empty_like(q), torch.empty((S, H, 1, 1), device=dev)

    def call(stream=None):
        hk.paged_decode(q, kp, vp, table, cl, out=o, lse=lse, workspace=ws, stream=stream)

    assert launches(call) == kernels
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call(side)
        call(side)  # the second one's split kernel stands behind the first one's combine
    for seed in (13, 14):
        q.copy_(torch.randn(q.shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16))
        cl.copy_(torch.flip(cl, (0,)))
        table.copy_(torch.flip(table, (0,)))
        o.fill_(float("nan"))
        lse.fill_(float("nan"))
        ws.fill_(255)
        graph.replay()
        torch.cuda.synchronize()
        got_o, got_lse = o.clone(), lse.clone()
        o_eager, lse_eager = hk.paged_decode(q, kp, vp, table, cl)
        assert _native.device_status(0) == 0
        assert torch.equal(got_o, o_eager) and torch.equal(got_lse, lse_eager)
    o_ref, l_ref = paged_decode_oracle(q.cpu(), kp.cpu(), vp.cpu(), table.cpu(), cl.cpu())
    assert float((got_o.float().cpu() - o_ref.float()).abs().max()) <= 2e-2
    assert float((got_lse.cpu() - l_ref).abs().max()) <= 1e-3


# context lengths around the chunk, the page and the empty context, in the chunks of 32 and of 64 pages
@pytest.mark.parametrize("S,H,H_KV,pages,lens", [
    (6, 8, 1, 1100, [512, 513, 511, 1024, 0, 16]), (5, 16, 2, 1100, [1, 15, 17, 496, 2048]),
    (16, 64, 16, 200, [1024, 1025, 1023, 2048, 0, 16] + [64 * i + 1 for i in range(10)])])
def test_chunk_and_page_boundaries(S, H, H_KV, pages, lens):
    dev = torch.device("cuda:0")
    top = max(lens)
    q, kp, vp, bt, _ = make_paged_inputs(S, H, H_KV, 128, 16, S * ((top + 15) // 16), top, top, seed=5)
    table = torch.zeros(S, pages, dtype=torch.int32)
    table[:, :bt.shape[1]] = bt
    ctx = torch.tensor(lens, dtype=torch.int32)
    args = [x.to(dev) for x in (q, kp, vp, table, ctx)]
    ws = torch.full((hk.paged_decode_workspace_bytes(S, H, 128, pages),), 255, dtype=torch.uint8, device=dev)
    o, lse = torch.full_like(args[0], float("nan")), torch.full((S, H, 1, 1), float("nan"), device=dev)
    assert launches(lambda: hk.paged_decode(*args, out=o, lse=lse, workspace=ws)) == 2
    assert _native.device_status(0) == 0
    live = [i for i, n in enumerate(lens) if n > 0]
    o_ref, l_ref = paged_decode_oracle(q[live], kp, vp, table[live], ctx[live])
    assert float((o.cpu()[live].float() - o_ref.float()).abs().max()) <= 2e-2
    assert float((lse.cpu()[live] - l_ref).abs().max()) <= 1e-3
    for i, n in enumerate(lens):
        if n == 0:
            assert not o[i].any() and bool(torch.isneginf(lse[i]).all())
