"""The modules' packed path: q, k, v read as views of a packed projection in both directions, its gradient written in
place, key lengths taken from the mask on the device."""
import pytest
import torch

from hipkittens_b200 import _native
from hipkittens_b200.attention import HipAttnFunction, HipCrossAttention, HipSelfAttention

pytestmark = pytest.mark.gpu


def _rand(*shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,n,nk,h,hkv,d", [(1, 1, 1, 1, 1, 64), (2, 129, 129, 4, 2, 128), (3, 200, 333, 6, 2, 64),
                                            (1, 256, 256, 8, 8, 128), (2, 300, 130, 2, 1, 64)])
def test_packed_gradient_is_the_gradient_of_the_parts(b, n, nk, h, hkv, d, causal):
    """Same kernels on the same values: O and every gradient are bit-identical to the contiguous call's."""
    q, kv, d_o = _rand(b, n, h, d, seed=1), _rand(b, nk, 2, hkv, d, seed=2), _rand(b, n, h, d, seed=3)
    qp, kvp = q.clone().requires_grad_(), kv.clone().requires_grad_()
    out = HipCrossAttention(causal=causal)(qp, kvp)
    out.backward(d_o)
    parts = [t.clone(memory_format=torch.contiguous_format).requires_grad_()
             for t in (q, kv[:, :, 0], kv[:, :, 1])]
    ref = HipAttnFunction.apply(*parts, causal)
    ref.backward(d_o)
    assert torch.equal(out, ref) and torch.equal(qp.grad, parts[0].grad)
    assert kvp.grad.is_contiguous()
    assert torch.equal(kvp.grad[:, :, 0], parts[1].grad) and torch.equal(kvp.grad[:, :, 1], parts[2].grad)
    if n == nk and h == hkv:
        qkv = torch.stack([q, kv[:, :, 0], kv[:, :, 1]], dim=2).detach().requires_grad_()
        HipSelfAttention(causal=causal)(qkv).backward(d_o)
        for i in range(3):
            assert torch.equal(qkv.grad[:, :, i], parts[i].grad)


@pytest.mark.parametrize("order", [(0, 1, 2, 3, 4), (4, 3, 2, 1, 0), (1, 0, 3, 4, 2)])
def test_saved_tensor_hooks_may_change_the_layout(order):
    """What a hook gives back for the projection, or for q, k and v, is the same numbers in a layout of its own choice."""
    def unpack(t):
        if t.dtype != torch.bfloat16 or t.dim() != 5:
            return t  # O and L
        return t.permute(order).contiguous().permute([order.index(i) for i in range(5)])

    qkv, d_o = _rand(2, 160, 3, 2, 64, seed=9), _rand(2, 160, 2, 64, seed=10)
    grads = []
    for hook in (lambda t: t, unpack):
        x = qkv.clone().requires_grad_()
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, hook):
            HipSelfAttention(causal=True)(x).backward(d_o)
        grads.append(x.grad)
    assert torch.equal(*grads)


@pytest.mark.parametrize("order", [(3, 2, 1, 0), (1, 0, 3, 2)])
def test_saved_tensor_hooks_may_change_the_layout_of_parts(order):
    q, k, v, d_o = (_rand(2, 160, h, 64, seed=s) for s, h in ((11, 6), (12, 2), (13, 2), (14, 6)))
    saved = []

    def unpack(t):
        if t.dtype != torch.bfloat16 or t.data_ptr() == saved[3]:
            return t  # L and O
        return t.permute(order).contiguous().permute([order.index(i) for i in range(4)])

    def pack(t):
        saved.append(t.data_ptr())
        return t

    grads = []
    for hook in (lambda t: t, unpack):
        saved.clear()
        leaves = [t.clone().requires_grad_() for t in (q, k, v)]
        with torch.autograd.graph.saved_tensors_hooks(pack, hook):
            HipAttnFunction.apply(*leaves, True).backward(d_o)
        grads.append([t.grad for t in leaves])
    for a, b in zip(*grads):
        assert torch.equal(a, b)


def test_offloaded_saved_tensors():
    qkv, d_o = _rand(2, 160, 3, 2, 64, seed=15), _rand(2, 160, 2, 64, seed=16)
    a, b = qkv.clone().requires_grad_(), qkv.clone().requires_grad_()
    HipSelfAttention()(a).backward(d_o)
    with torch.autograd.graph.save_on_cpu():
        HipSelfAttention()(b).backward(d_o)
    assert torch.equal(a.grad, b.grad)


def test_float16_projection_takes_the_converting_path():
    qkv = _rand(2, 160, 3, 2, 64, seed=4).half().requires_grad_()
    out = HipSelfAttention()(qkv)
    d_o = _rand(2, 160, 2, 64, seed=5).half()
    out.backward(d_o)
    ref = qkv.detach().to(torch.bfloat16).requires_grad_()
    HipSelfAttention()(ref).backward(d_o.to(torch.bfloat16))
    assert out.dtype == torch.float16 and qkv.grad.dtype == torch.float16
    assert torch.equal(qkv.grad, ref.grad.half())


# key blocks against 148 SMs: one round of single blocks and its edge, several rounds of them, pairs that fill 95 %
@pytest.mark.parametrize("b,nk,hkv", [(1, 128 * 148, 1), (1, 128 * 148 + 1, 1), (4, 128 * 37, 1), (2, 128 * 37, 2),
                                      (3, 128 * 100, 1), (2, 128 * 148, 1), (4, 128 * 74, 1)])
def test_causal_key_blocks_dealt_singly_and_in_pairs(b, nk, hkv):
    """Every key block is served exactly once however the blocks are dealt: a batch element's dK and dV are bit-identical
    to those of a call with another number of batch elements."""
    n = 200
    q, kv, d_o = _rand(1, n, 2 * hkv, 64, seed=6), _rand(1, nk, 2, hkv, 64, seed=7), _rand(1, n, 2 * hkv, 64, seed=8)

    def grads(copies):
        qd = q.expand(copies, -1, -1, -1).contiguous().requires_grad_()
        kvd = kv.expand(copies, -1, -1, -1, -1).contiguous().requires_grad_()
        HipCrossAttention(causal=True)(qd, kvd).backward(d_o.expand(copies, -1, -1, -1).contiguous())
        return kvd.grad

    got, other = grads(b), grads(b + 1)[:1]
    assert bool(torch.isfinite(got).all()) and float(got.float().abs().max()) > 0
    for i in range(b):
        assert torch.equal(got[i:i + 1], other)


@pytest.mark.parametrize("b,n", [(1, 1), (3, 255), (2, 256), (5, 1000)])
def test_key_padding_lens(b, n):
    gen = torch.Generator().manual_seed(n)
    lens = torch.randint(1, n + 1, (b,), generator=gen)
    mask = torch.arange(n)[None] < lens[:, None]
    got, bad = _native.key_padding_lens(mask.cuda())
    assert got.cpu().tolist() == lens.tolist() and int(bad) == 0
    wide = torch.zeros(b, 2 * n, dtype=torch.bool)  # a mask that is a strided view
    wide[:, ::2] = mask
    got, bad = _native.key_padding_lens(wide.cuda()[:, ::2])
    assert got.cpu().tolist() == lens.tolist() and int(bad) == 0
    empty = mask.clone()
    empty[b - 1] = False
    assert int(_native.key_padding_lens(empty.cuda())[1]) != 0
    if n > 2:
        hole = mask.clone()
        hole[0] = True
        hole[0, n // 2] = False
        assert int(_native.key_padding_lens(hole.cuda())[1]) != 0


def test_a_refused_mask_leaves_the_next_call_alone():
    """The verdict on a mask is a flag of its own per call, read behind the forward: refused and accepted masks in turn."""
    qkv = _rand(2, 300, 3, 4, 64, seed=11)
    good = torch.arange(300)[None].cuda() < torch.tensor([[300], [120]]).cuda()
    bad = good.clone()
    bad[1, 5] = False
    module = HipSelfAttention()
    ref = module(qkv, key_padding_mask=good)
    for _ in range(3):
        with pytest.raises(ValueError):
            module(qkv, key_padding_mask=bad)
        assert torch.equal(module(qkv, key_padding_mask=good), ref)


@pytest.mark.parametrize("default", ["cuda", "cuda:0"])
def test_a_mask_under_a_default_device(default):
    """The verdict's flag lies in host memory wherever tensors are made by default."""
    qkv = torch.randn(2, 80, 3, 2, 64, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda().requires_grad_()
    mask = (torch.arange(80)[None] < torch.tensor([80, 33])[:, None]).cuda()
    module = HipSelfAttention(causal=True)
    ref = module(qkv, key_padding_mask=mask)
    with torch.device(default):
        out = module(qkv, key_padding_mask=mask)
        out.backward(torch.ones_like(out))
        with pytest.raises(ValueError):
            module(qkv, key_padding_mask=~mask)
    assert torch.equal(out, ref) and bool(torch.isfinite(qkv.grad).all())
