"""How the causal dK/dV kernel deals its key blocks to CTAs: in pairs of equal cost or singly, by what either loses; and that
either way serves every block once."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200.attention import HipCrossAttention


def _in_pairs(b, n, nk, h, hkv, d, sms=148):
    return hk.capi().hk_selftest_dkdv_in_pairs(b, n, nk, h, hkv, d, sms)


# (B, N, H, H_KV, D) -> dealt in pairs; us of dK/dV and dQ in pairs and singly, as measured
@pytest.mark.parametrize("shape,pairs", [
    ((2, 384, 8, 2, 128), 0),       # fewer blocks than SMs
    ((24, 512, 16, 4, 128), 0),     # 151.8 / 129.8: pairs fill 0.65 of two rounds
    ((8, 4096, 16, 4, 128), 0),     # 1556 / 1519: 0.865 full, 256 MB of Q and dO over 32 units
    ((12, 8192, 4, 4, 64), 0),      # 1552 / 1507: 0.943 full, 96 MB
    ((12, 1536, 16, 4, 128), 1),    # 366.4 / 372.5: 0.973 full
    ((32, 3072, 16, 4, 128), 1),    # 3478 / 3744: 0.943 full, 768 MB
    ((48, 2048, 16, 4, 128), 1),    # 2467 / 2680
    ((24, 4096, 4, 4, 128), 1),     # 1180 / 1247: 0.943 full, 192 MB
    ((24, 4096, 16, 4, 64), 1),     # 3163 / 3285: 0.943 full, 384 MB
    ((48, 1024, 16, 4, 128), 1),    # 750.7 / 771.4: 0.865 full, 384 MB over 192 units
])
def test_the_dealing_that_measured_faster(native_built, shape, pairs):
    b, n, h, hkv, d = shape
    assert _in_pairs(b, n, n, h, hkv, d) == pairs


def test_edges_of_the_rule(native_built):
    # three blocks: every second CTA would be given nothing but middle blocks. 76 us in pairs, 64 us singly with 192 units, D128
    assert _in_pairs(148, 384, 384, 1, 1, 128) == 0 and _in_pairs(256, 384, 384, 8, 1, 128) == 0
    # with more blocks the odd one matters less
    assert _in_pairs(148, 128 * 11, 128 * 11, 1, 1, 64) == 1
    # one round of pairs, full, 5 % idle, and one more pair than a round
    assert [_in_pairs(1, 200, 256 * k, 2, 1, 64) for k in (148, 141, 140, 149)] == [1, 1, 0, 0]
    assert _in_pairs(0, 1, 1, 1, 1, 64) < 0 and _in_pairs(1, 1, 1, 3, 2, 64) < 0 and _in_pairs(1, 1, 1, 1, 1, 96) < 0


def _rand(*shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


# (b in pairs, other dealt singly, n, nk, h, hkv, d): odd numbers of blocks, whose middle block is a pair of its own, over
# one and several rounds of pairs; pairs because of what the units in flight read, with an even and an odd number
@pytest.mark.gpu
@pytest.mark.parametrize("b,other,n,nk,h,hkv,d", [
    (4, 1, 200, 128 * 73, 2, 1, 64), (8, 1, 200, 128 * 73, 2, 1, 64), (2, 1, 200, 128 * 73 - 5, 4, 2, 64),
    (74, 3, 130, 128 * 11, 2, 2, 128), (48, 1, 2048, 2048, 16, 4, 128), (29, 1, 2944, 2944, 16, 4, 64)])
def test_pairs_and_single_blocks_give_the_same_gradients(b, other, n, nk, h, hkv, d):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _in_pairs(b, n, nk, h, hkv, d, sms) == 1 and _in_pairs(other, n, nk, h, hkv, d, sms) == 0
    q, kv, d_o = _rand(1, n, h, d, seed=6), _rand(1, nk, 2, hkv, d, seed=7), _rand(1, n, h, d, seed=8)

    def grads(copies):
        qd = q.expand(copies, -1, -1, -1).contiguous().requires_grad_()
        kvd = kv.expand(copies, -1, -1, -1, -1).contiguous().requires_grad_()
        HipCrossAttention(causal=True)(qd, kvd).backward(d_o.expand(copies, -1, -1, -1).contiguous())
        return kvd.grad

    got, ref = grads(b), grads(other)[:1]
    assert bool(torch.isfinite(got).all())
    assert bool((ref.float().abs().amax(dim=(2, 3, 4)) > 0).all())  # every key is seen, so no block stays unwritten
    for i in range(b):
        assert torch.equal(got[i:i + 1], ref)
