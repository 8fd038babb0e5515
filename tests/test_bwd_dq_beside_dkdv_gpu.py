"""The dQ kernel runs beside the dK/dV kernel: whoever comes behind it waits for both, and dQ in the place of Q or dO is written
when nobody reads those any more. Results are those of the two kernels one after the other, bit for bit."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native

pytestmark = pytest.mark.gpu

# few dK/dV CTAs, most SMs taken, more than a round of them; both layouts of the kernels
SHAPES = [(1, 300, 8, 1, 128, True), (1, 512, 8, 8, 128, False), (2, 200, 6, 2, 64, False), (5, 300, 32, 8, 128, True),
          (3, 700, 16, 16, 64, True)]


def inputs(B, N, H, HK, D, causal):
    gen = torch.Generator(device="cuda").manual_seed(N)

    def rand(h):
        return torch.randn((B, N, h, D), generator=gen, device="cuda", dtype=torch.bfloat16)

    q, k, v, d_o = rand(H), rand(HK), rand(HK), rand(H)
    o, lse = hk.attn_fwd(q, k, v, causal=causal)
    return q, k, v, d_o, o, lse


def backward(q, k, v, o, d_o, lse, dq, causal):
    dk, dv = torch.empty_like(k), torch.empty_like(v)
    _native.attn_bwd_strided(q, k, v, o, d_o, lse, dq, dk, dv, causal=causal)
    return dq, dk, dv


@pytest.mark.parametrize("shape", SHAPES)
def test_dq_in_the_place_of_what_dkdv_reads(shape):
    causal = shape[-1]
    q, k, v, d_o, o, lse = inputs(*shape)
    ref = [t.clone() for t in backward(q, k, v, o, d_o, lse, torch.empty_like(q), causal)]
    for _ in range(5):
        q2, d2 = q.clone(), d_o.clone()
        for a, b in zip(backward(q2, k, v, o, d_o, lse, q2, causal), ref):
            assert torch.equal(a, b)
        for a, b in zip(backward(q, k, v, o, d2, lse, d2, causal), ref):
            assert torch.equal(a, b)
    assert _native.device_status(0) == 0


@pytest.mark.parametrize("shape", SHAPES)
def test_a_dependent_kernel_behind_it_finds_both_complete(shape):
    B, N, H, HK, D, causal = shape
    q, k, v, d_o, o, lse = inputs(*shape)
    ref = [t.clone() for t in backward(q, k, v, o, d_o, lse, torch.empty_like(q), causal)]
    ang = torch.arange(N, device="cuda")[:, None] / (1.0 + torch.arange(D // 2, device="cuda")[None])
    cos, sin = ang.cos().bfloat16(), ang.sin().bfloat16()
    want = [hk.rotary_bnhd(t, cos, sin) for t in ref]
    for _ in range(10):
        q2, k2 = q.clone(), k.clone()
        dq, dk, dv = backward(q2, k2, v, o, d_o, lse, torch.empty_like(q), causal)
        hk.rotary_bnhd(q2, cos, sin, out=q2)  # overwrites what both kernels read
        hk.rotary_bnhd(k2, cos, sin, out=k2)
        got = [hk.rotary_bnhd(t, cos, sin) for t in (dq, dk, dv)]
        for a, b in zip((dq, dk, dv, *got), (*ref, *want)):
            assert torch.equal(a, b)


def test_dq_of_few_queries_on_many_keys_is_served_once():
    """Groups of units of the causal dQ order: all units in one group here, two groups for the single batch elements."""
    gen = torch.Generator(device="cuda").manual_seed(3)

    def rand(n):
        return torch.randn((3, n, 8, 128), generator=gen, device="cuda", dtype=torch.bfloat16)

    q, d_o, k, v = rand(100), rand(100), rand(16384), rand(16384)
    o, lse = hk.attn_fwd(q, k, v, causal=True)
    got = backward(q, k, v, o, d_o, lse, torch.full_like(q, float("nan")), True)[0]
    assert bool(torch.isfinite(got).all())
    for i in range(3):
        one = [t[i:i + 1].contiguous() for t in (q, k, v, o, d_o, lse)]
        assert torch.equal(got[i:i + 1], backward(*one, torch.full_like(one[0], float("nan")), True)[0])


@pytest.mark.parametrize("shape", SHAPES)
def test_every_call_reads_its_own_statistics_and_lengths(shape):
    """L, delta and the key lengths of a call are written by the kernels just before its dK/dV kernel, into the buffers that
    the call before it read: back to back, every call gives what it gives when each of them is waited for."""
    B, N, H, HK, D, causal = shape
    gen = torch.Generator(device="cuda").manual_seed(N + 1)
    steps = []
    for i in range(8):
        q, k, v, d_o = (torch.randn((B, N, h, D), generator=gen, device="cuda", dtype=torch.bfloat16) * (1 + i % 3)
                        for h in (H, HK, HK, H))
        lens = torch.randint(1, N + 1, (B, 1), generator=gen, device="cuda")
        steps.append((q, k, v, d_o, torch.arange(N, device="cuda")[None] < lens))

    def chain(sync):
        o, lse, seen = torch.empty_like(steps[0][0]), torch.empty((B, H, 1, N), device="cuda"), []
        kv_lens = bad = None
        for q, k, v, d_o, mask in steps:
            del kv_lens, bad  # the next call's come to lie where they were
            kv_lens, bad = _native.key_padding_lens(mask)
            hk.attn_fwd(q, k, v, causal=causal, out=o, lse=lse, kv_lens=kv_lens)
            if sync:
                torch.cuda.synchronize()
            grads = [torch.empty_like(t) for t in (q, k, v)]
            _native.attn_bwd_strided(q, k, v, o, d_o, lse, *grads, causal=causal, kv_lens=kv_lens)
            if sync:
                torch.cuda.synchronize()
            seen += grads
        return seen

    for a, b in zip(chain(False), chain(True)):
        assert torch.equal(a, b)
    assert _native.device_status(0) == 0


@pytest.mark.parametrize("shape", [(1, 128, 8, 8, 128, False), (3, 100, 4, 4, 64, True), (40, 120, 8, 8, 128, True)])
def test_dq_in_the_place_of_a_single_key_tile(shape):
    """With one tile of queries and one of keys, and as many K/V heads as heads, a dQ tile may lie where the only K or V tile
    that its CTA reads lay."""
    causal = shape[-1]
    q, k, v, d_o, o, lse = inputs(*shape)
    ref = [t.clone() for t in backward(q, k, v, o, d_o, lse, torch.empty_like(q), causal)]
    for _ in range(5):
        k2, v2 = k.clone(), v.clone()
        for a, b in zip(backward(q, k2, v, o, d_o, lse, k2, causal), ref):
            assert torch.equal(a, b)
        for a, b in zip(backward(q, k, v2, o, d_o, lse, v2, causal), ref):
            assert torch.equal(a, b)
    assert _native.device_status(0) == 0
