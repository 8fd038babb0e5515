"""Key lengths may be any int32 view [B]: the kernels index them densely, so other strides are made dense on the way."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native
from hipkittens_b200.attention import HipAttnFunction


def _views(device):
    """name -> (view [3], what it says)"""
    return {
        "every_second": (torch.tensor([7, 130, 200, 1, 129, 2], dtype=torch.int32, device=device)[::2], [7, 200, 129]),
        "expanded": (torch.tensor([77], dtype=torch.int32, device=device).expand(3), [77, 77, 77]),
        "column": (torch.tensor([[5, 0], [200, 0], [64, 0]], dtype=torch.int32, device=device)[:, 0], [5, 200, 64]),
    }


@pytest.mark.parametrize("name", ["every_second", "expanded", "column"])
def test_views_become_dense(name):
    view, values = _views("cpu")[name]
    assert not view.is_contiguous()
    dense = _native._dense_lens(view, 3, view.device, None)
    assert dense.is_contiguous() and dense.tolist() == values
    assert _native._dense_lens(dense, 3, view.device, None) is dense  # and what is dense is not copied
    with pytest.raises(RuntimeError, match="int32 tensor"):
        _native._dense_lens(view, 2, view.device, None)


@pytest.mark.gpu
@pytest.mark.parametrize("other_stream", [False, True])
@pytest.mark.parametrize("name", ["every_second", "expanded", "column"])
def test_every_entry_masks_by_what_the_view_says(name, other_stream):
    gen = torch.Generator("cuda").manual_seed(11)
    q, kv, d_o = (torch.randn(s, device="cuda", generator=gen).to(torch.bfloat16)
                  for s in ((3, 200, 4, 64), (3, 200, 2, 2, 64), (3, 200, 4, 64)))
    k, v = (t.contiguous() for t in kv.unbind(2))
    view, values = _views("cuda")[name]
    dense = torch.tensor(values, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream() if other_stream else None
    torch.cuda.synchronize()

    def grads(lens):
        out, lse = hk.attn_fwd(q, k, v, kv_lens=lens, stream=stream)
        delta = hk.attn_bwd_prep(out, d_o, stream=stream)
        three = hk.attn_bwd(q, k, v, d_o, lse, delta, kv_lens=lens, stream=stream)
        torch.cuda.synchronize()
        packed = [torch.empty_like(q), *torch.empty_like(kv).unbind(2)]
        _native.attn_bwd_strided(q, *kv.unbind(2), out, d_o, lse, *packed, kv_lens=lens)
        leaf = q.clone().requires_grad_()
        through = HipAttnFunction.apply(leaf, k, v, False, None, lens)
        through.backward(d_o)
        return (out, lse, *three, *packed, through.detach(), leaf.grad)

    for got, ref in zip(grads(view), grads(dense)):
        assert torch.equal(got, ref)
