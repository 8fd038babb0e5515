"""The backward over shards of the (batch, kv head) units against one call over all of them. With few key blocks, a shard's
blocks may be shared by another number of CTAs than the whole call's: dK and dV then agree but for the rounding of fp32 sums in
another order, everything else is the same bits."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native, shard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,H_KV,D,causal,world", [(2, 1024, 8, 2, 128, True, 4), (2, 700, 8, 4, 64, False, 3),
                                                       (4, 300, 16, 4, 128, True, 2)])
def test_shards_agree_with_the_whole_call(B, N, H, H_KV, D, causal, world):
    gen = torch.Generator(device="cuda").manual_seed(N)
    q, d_o = (torch.randn(B, N, H, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, N, H_KV, D, generator=gen, device="cuda").bfloat16() for _ in range(2))

    def grads(q, k, v, d_o):
        o, lse = hk.attn_fwd(q, k, v, causal=causal)
        out = [torch.empty_like(t) for t in (q, k, v)]
        _native.attn_bwd_strided(q, k, v, o, d_o, lse, *out, causal=causal)
        return out

    whole = grads(q, k, v, d_o)
    got = [torch.full_like(t, float("nan")) for t in whole]
    for rank in range(world):
        slices = shard.partition_units(B, H_KV, world, rank)
        for qs, ks, vs, members in shard.shard_tensors(q, k, v, H_KV, slices):
            shard.scatter_grads(*got, *grads(qs, ks, vs, shard.shard_like_q(d_o, H_KV, members)), members, H_KV)
    assert torch.equal(got[0], whole[0])
    for a, b in zip(got[1:], whole[1:]):
        a, b = a.float(), b.float()
        # a bf16 step (2^-7 at most) where the sums round to neighbours, and fp32 rounding of sums that nearly cancel
        assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-5 * b.abs().max()).all())
    assert _native.device_status(0) == 0
