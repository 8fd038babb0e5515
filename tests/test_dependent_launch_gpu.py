"""Kernels are launched so that they may start under the tail of the one before them. A chain of calls that hand their
buffers on and overwrite them must give what the same calls give with a synchronisation after each."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native

pytestmark = pytest.mark.gpu


def _chain(n, d, steps, sync):
    gen = torch.Generator("cuda").manual_seed(11)

    def rand(*shape):
        return torch.randn(shape, device="cuda", generator=gen).to(torch.bfloat16)

    def call(fn, *args, **kwargs):
        r = fn(*args, **kwargs)
        if sync:
            torch.cuda.synchronize()
        return r

    q, k, v, d_o = rand(2, n, 4, d), rand(2, n, 2, d), rand(2, n, 2, d), rand(2, n, 4, d)
    angle = torch.rand(n, d // 2, device="cuda", generator=gen)
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
    kr, outs = torch.empty_like(k), [torch.empty_like(q), torch.empty_like(q)]
    lse = torch.empty(2, 4, 1, n, device="cuda")
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    pools = [torch.zeros(2 * n, 16, 2, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    table = torch.arange(2 * n, device="cuda", dtype=torch.int32).reshape(2, n)
    tokens, q1 = rand(2, 1, 2, 128), rand(2, 1, 8, 128)
    seen = []
    for i in range(steps):
        # every call reads what the one before it wrote, and overwrites what earlier ones read
        out, vi = outs[i % 2], v if i == 0 else outs[(i + 1) % 2][:, :, :2]
        call(hk.rotary_bnhd, k if i == 0 else kr, cos, sin, out=kr)
        call(hk.attn_fwd, q, kr, vi, causal=True, out=out, lse=lse)
        call(_native.attn_bwd_strided, q, kr, vi, out, d_o, lse, dq, dk, dv, causal=True)
        if d == 128:
            start = torch.full((2,), i, dtype=torch.int32, device="cuda")
            call(hk.paged_kv_append, tokens, tokens, *pools, table, start)
            o1, _ = call(hk.paged_decode, q1, *pools, table, start + 1)
            tokens = o1[:, :, :2].contiguous()
            seen.append(o1)
    return [*outs, lse, dq, dk, dv, kr, *pools, *seen]


@pytest.mark.parametrize("n,d", [(64, 64), (200, 128), (1000, 128)])
def test_back_to_back_calls_equal_synchronised_ones(n, d):
    for a, b in zip(_chain(n, d, 12, False), _chain(n, d, 12, True)):
        assert torch.equal(a, b)


def test_decode_steps_over_several_chunks():
    """Contexts that are cut into 2 to 9 chunks, so that the combine kernel merges partials of the split kernel before it
    while the append of the next step stands behind it; the workspace is one and the same."""
    gen = torch.Generator("cuda").manual_seed(13)
    b, h, hkv, pages = 3, 16, 2, 290
    start0 = torch.tensor([700, 2100, 4500], dtype=torch.int32, device="cuda")
    pool0 = [torch.randn(b * pages, 16, hkv, 128, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]
    table = torch.randperm(b * pages, device="cuda", generator=gen).to(torch.int32).reshape(b, pages)
    need = hk.paged_decode_workspace_bytes(b, h, 128, pages)
    workspace = torch.empty(need, dtype=torch.uint8, device="cuda")
    angle = torch.rand(pages * 16, 64, device="cuda", generator=gen)
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
    q0 = torch.randn(b, 1, h, 128, device="cuda", generator=gen).to(torch.bfloat16)

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


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("n,d", [(200, 64), (1000, 128)])
def test_three_call_backward_behind_its_forward(n, d, causal):
    """delta, the gradients and the shuffle each read what the kernel before them wrote, and the next pass overwrites it."""
    gen = torch.Generator("cuda").manual_seed(14)
    q, k, v, d_o = (torch.randn(2, n, x, d, device="cuda", generator=gen).to(torch.bfloat16) for x in (4, 2, 2, 4))

    def chain(sync):
        seen, x, o, lse = [], q, torch.empty_like(q), torch.empty(2, 4, 1, n, device="cuda")
        delta, dq_in = torch.empty_like(lse), torch.empty(2, 4, n, d, dtype=torch.bfloat16, device="cuda")
        dk, dv = torch.empty_like(k), torch.empty_like(v)
        for i in range(10):
            dq = torch.empty_like(q)
            for step in (lambda: hk.attn_fwd(x, k, v, causal=causal, out=o, lse=lse),
                         lambda: hk.attn_bwd_prep(o, d_o, delta=delta),
                         lambda: hk.attn_bwd(x, k, v, d_o, lse, delta, causal=causal, dq=dq_in, dk=dk, dv=dv,
                                             dq_layout=_native.HK_DQ_BHND),
                         lambda: hk.dq_shuffle(dq_in, dq)):
                step()
                if sync:
                    torch.cuda.synchronize()
            seen.append(dq)
            x = dq
        return [*seen, delta, dk, dv, o, lse]

    for a, b in zip(chain(False), chain(True)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("captured", [False, True])
def test_events_of_another_stream_are_waited_for(captured):
    """A dependent launch behind a wait for an event reads what that event stands for, in a stream and in a graph."""
    gen = torch.Generator("cuda").manual_seed(15)
    src = [torch.randn(1, 256, 4, 64, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(6)]
    cos, sin = (torch.randn(256, 32, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2))
    big = torch.randn(4096, 4096, device="cuda", generator=gen)
    side = torch.cuda.Stream()
    x, y = torch.zeros_like(src[0]), src[0].clone()
    outs = [torch.empty_like(x) for _ in src]

    def calls():
        main = torch.cuda.current_stream()
        for s, o in zip(src, outs):
            side.wait_stream(main)
            with torch.cuda.stream(side):
                torch.mm(big, big)  # some hundred microseconds
                x.copy_(s)
            hk.rotary_bnhd(y, cos, sin, out=y)  # the kernel before in the same stream is done long before that
            main.wait_stream(side)
            hk.rotary_bnhd(x, cos, sin, out=o)

    expected = [hk.rotary_bnhd(s, cos, sin) for s in src]
    torch.cuda.synchronize()
    if captured:
        torch.mm(big, big)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            calls()
        graph.replay()
        for o in outs:
            o.zero_()
        x.zero_()
        graph.replay()
    else:
        calls()
    torch.cuda.synchronize()
    for a, b in zip(outs, expected):
        assert torch.equal(a, b)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("d", [64, 128])
def test_long_forward_between_dependent_launches(d, causal):
    """A forward of more than 100 tiles per CTA is launched the ordinary way (most of them as code without the
    instructions of dependent launches): it still comes after what is before it, and before what follows."""
    n, h, hkv = 4096, 32, 8
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (h // 2) * (n // 128) ** 2 > 100 * sms
    gen = torch.Generator("cuda").manual_seed(12)
    q, k, v, d_o = (torch.randn(1, n, x, d, device="cuda", generator=gen).to(torch.bfloat16) for x in (h, hkv, hkv, h))
    angle = torch.rand(n, d // 2, device="cuda", generator=gen)
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)

    def chain(sync):
        x, seen = q.clone(), []
        for _ in range(4):
            for step in (lambda: hk.rotary_bnhd(x, cos, sin, out=x),
                         lambda: seen.extend(hk.attn_fwd(x, k, v, causal=causal)),
                         lambda: seen.append(hk.attn_bwd_prep(seen[-2], d_o)),
                         lambda: hk.rotary_bnhd(seen[-3], cos, sin, out=x)):
                step()
                if sync:
                    torch.cuda.synchronize()
        return seen

    for a, b in zip(chain(False), chain(True)):
        assert torch.equal(a, b)


def test_captured_chain_replays():
    """The dependent launches survive capture into a CUDA graph."""
    q, kv = torch.randn(2, 1, 300, 4, 64, device="cuda").to(torch.bfloat16)
    cos, sin = (torch.randn(300, 32, device="cuda").to(torch.bfloat16) for _ in range(2))
    rot, out, lse = torch.empty_like(q), torch.empty_like(q), torch.empty(1, 4, 1, 300, device="cuda")

    def calls():
        hk.rotary_bnhd(q, cos, sin, out=rot)
        hk.attn_fwd(rot, kv, kv, causal=True, out=out, lse=lse)

    calls()
    torch.cuda.synchronize()
    expected = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    out.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, expected)


def test_a_new_thread_launches_into_a_capture():
    """A thread without a CUDA context of its own may be the one that launches, also while a stream is being captured."""
    import threading

    q = torch.randn(1, 300, 4, 64, device="cuda").to(torch.bfloat16)
    out, lse = torch.empty_like(q), torch.empty(1, 4, 1, 300, device="cuda")
    expected, _ = hk.attn_fwd(q, q, q)
    torch.cuda.synchronize()
    codes = []
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # "global": calls that could disturb the capture are refused in every thread
        stream = torch.cuda.current_stream().cuda_stream
        t = threading.Thread(target=lambda: codes.append(_native.capi().hk_attn_fwd(
            q.data_ptr(), q.data_ptr(), q.data_ptr(), out.data_ptr(), lse.data_ptr(), 1, 300, 4, 4, 64, 0, 0.0, 0, stream)))
        t.start()
        t.join()
    assert codes == [0]
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, expected)
