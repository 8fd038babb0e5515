"""Host-side mirror of the reference's attention call site (forward and backward).

``HipAttnFunction`` / ``HipSelfAttention`` / ``HipCrossAttention`` follow
``training/llama/llama/models/attentions/hipkittens.py:17-61,122-202``: inputs and outputs are BNHD, O [B,N,H,D] bf16
and L [B,H,1,N] fp32 are allocated here, O is returned in the input dtype and (q, k, v, O, L) are saved for the backward
pass. Like the reference's ``tk_kernel_fwd.dispatch_fwd`` and its three backward calls (hipkittens.py:64-119), forward
and backward each return when the device is done and raise if a kernel reported a failure; they synchronise once for
that, not after each kernel. A ``key_padding_mask`` is looked at on the device, and its verdict is read behind the forward's
synchronisation: a mask that cannot be honoured raises after the kernels have run on clamped lengths.

Differences: bf16 tensors are read through strided TMA descriptors and gradients written through strides, so there are
no ``.contiguous()`` copies of q, k and v (hipkittens.py:37-39) in either direction, and the modules' packed
qkv / kv gradient is written in place instead of being stacked from its parts afterwards; dQ is written in its final
layout, without the zero fill and the shuffle pass (``dispatch_prep`` / ``dispatch_bwd_combined`` /
``dispatch_dq_shuffle`` stay available in the compiled modules); a right-padded ``key_padding_mask``
(True = keep, as in ``base.py:88-103``) is honoured through per-batch key lengths, also together with ``causal``
and with more keys than queries (``base.py:104-116``), where the reference's modules accept the argument and ignore
it (hipkittens.py:147-162); and causality and the softmax scale are honoured here (they are baked into the reference's compiled module, and its modules
ignore the ``causal`` and ``softmax_scale`` they are constructed with, hipkittens.py:147-162).
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch.autograd import Function

from ._native import attn_bwd_strided, attn_fwd, device_status, key_padding_lens


def _tma_viewable(t: torch.Tensor) -> bool:
    """bf16, last dimension contiguous, other strides positive multiples of 8 elements (16 bytes)."""
    return (t.dtype == torch.bfloat16 and t.dim() == 4 and t.stride(3) == 1
            and all(st > 0 and st % 8 == 0 for st in t.stride()[:3]))


def _packed_viewable(t: torch.Tensor) -> bool:
    """The same for the q, k, v slices of a packed projection [B, S, 2 or 3, H, D]."""
    return (t.dtype == torch.bfloat16 and t.dim() == 5 and t.stride(4) == 1
            and all(t.stride(i) > 0 and t.stride(i) % 8 == 0 for i in (0, 1, 3)))


def _check_qkv(q, k, v):
    B, N, H, D = q.shape
    HKV, NK = k.shape[2], k.shape[1]
    assert k.shape == (B, NK, HKV, D), f"K shape mismatch: expected ({B}, {NK}, {HKV}, {D}), got {k.shape}"
    assert v.shape == (B, NK, HKV, D), f"V shape mismatch: expected ({B}, {NK}, {HKV}, {D}), got {v.shape}"
    assert q.is_cuda and k.is_cuda and v.is_cuda, "All tensors must be on CUDA device"
    assert q.device == k.device == v.device, "All tensors must be on same device"
    assert H % HKV == 0, f"H ({H}) must be divisible by HKV ({HKV}) for GQA"


def _blocking_status(dev, what):
    status = device_status(dev.index)  # blocks on the device like the reference's dispatch_* calls do
    if status != 0:
        raise RuntimeError(f"attention {what} failed on the device (status {status})")


def _forward(q, k, v, causal, softmax_scale, kv_lens):
    O, L = attn_fwd(q, k, v, causal=causal, softmax_scale=softmax_scale, kv_lens=kv_lens)
    _blocking_status(q.device, "forward")
    return O, L


def _backward(ctx, q, k, v, O, L, dO_bnhd, dQ, dK, dV):
    assert dO_bnhd.shape == O.shape, f"dO shape mismatch: expected {tuple(O.shape)}, got {dO_bnhd.shape}"
    assert dO_bnhd.is_cuda and dO_bnhd.device == O.device, "dO must be on correct CUDA device"
    dO = dO_bnhd.to(torch.bfloat16).contiguous()
    rest = dict(causal=ctx.causal, softmax_scale=ctx.softmax_scale, kv_lens=ctx.kv_lens)
    try:
        attn_bwd_strided(q, k, v, O, dO, L, dQ, dK, dV, **rest)
    except RuntimeError:
        # saved-tensor hooks may have given q, k or v back in a layout that the kernels cannot read (looked for only here,
        # where the call was refused: the look takes 4 us)
        dense = [t if _tma_viewable(t) else t.contiguous() for t in (q, k, v)]
        if all(a is b for a, b in zip(dense, (q, k, v))):
            raise
        attn_bwd_strided(*dense, O, dO, L, dQ, dK, dV, **rest)
    _blocking_status(O.device, "backward")


class HipAttnFunction(Function):
    @staticmethod
    def forward(ctx, q_bnhd: torch.Tensor, k_bnhd: torch.Tensor, v_bnhd: torch.Tensor, causal: bool = True,
                softmax_scale=None, kv_lens=None):
        _check_qkv(q_bnhd, k_bnhd, v_bnhd)
        if all(_tma_viewable(t) for t in (q_bnhd, k_bnhd, v_bnhd)):
            q, k, v = q_bnhd, k_bnhd, v_bnhd
        else:
            q, k, v = (t.to(torch.bfloat16).contiguous() for t in (q_bnhd, k_bnhd, v_bnhd))
        O, L = _forward(q, k, v, bool(causal), softmax_scale, kv_lens)
        ctx.save_for_backward(q, k, v, O, L)
        ctx.causal = bool(causal)
        ctx.softmax_scale = softmax_scale
        ctx.kv_lens = kv_lens
        return O.to(q_bnhd.dtype)

    @staticmethod
    def backward(ctx, dO_bnhd: torch.Tensor):
        q, k, v, O, L = ctx.saved_tensors
        dQ, dK, dV = (torch.empty(t.shape, dtype=torch.bfloat16, device=t.device) for t in (q, k, v))
        _backward(ctx, q, k, v, O, L, dO_bnhd, dQ, dK, dV)
        return dQ.to(dO_bnhd.dtype), dK.to(dO_bnhd.dtype), dV.to(dO_bnhd.dtype), None, None, None


class _PackedAttnFunction(Function):
    """``HipAttnFunction`` on the modules' packed bf16 projections: `packed` [B,S,2,H_KV,D] with a `q` of its own, or
    [B,S,3,H,D] with q = None. q, k and v are read as strided views and the packed gradient is written in place (as
    ``unbind`` outputs the three gradients would be stacked by a copy of them all)."""

    @staticmethod
    def forward(ctx, q, packed, causal, softmax_scale, kv_lens):
        qkv = packed.unbind(dim=2) if q is None else (q, *packed.unbind(dim=2))
        _check_qkv(*qkv)
        O, L = _forward(*qkv, causal, softmax_scale, kv_lens)
        ctx.save_for_backward(*([packed] if q is None else [q, packed]), O, L)
        ctx.causal = causal
        ctx.softmax_scale = softmax_scale
        ctx.kv_lens = kv_lens
        return O

    @staticmethod
    def backward(ctx, dO_bnhd):
        *q, packed, O, L = ctx.saved_tensors
        d_packed = torch.empty(packed.shape, dtype=torch.bfloat16, device=packed.device)
        d_q = [torch.empty(t.shape, dtype=torch.bfloat16, device=t.device) for t in q]
        _backward(ctx, *q, *packed.unbind(dim=2), O, L, dO_bnhd, *d_q, *d_packed.unbind(dim=2))
        return d_q[0] if q else None, d_packed, None, None, None


def _attend(q, packed, causal, softmax_scale, key_padding_mask):
    """Attention of q (None: the first of the packed tensors) over a packed projection [B, S, 2 or 3, H, D]."""
    if key_padding_mask is None:
        out = _apply(q, packed, causal, softmax_scale, None)
    else:
        kv_lens, bad = _lens_from_key_padding_mask(key_padding_mask, packed)
        try:
            out = _apply(q, packed, causal, softmax_scale, kv_lens)
        except BaseException:
            torch.cuda.synchronize(packed.device)  # the flag may still be written: it is given back only then
            raise
        # whatever the mask, the kernels clamp the lengths
        if bad.item() != 0:
            raise ValueError(_BAD_MASK)
    return out.to((packed if q is None else q).dtype).contiguous()


def _apply(q, packed, causal, softmax_scale, kv_lens):
    if _packed_viewable(packed) and (q is None or _tma_viewable(q)):
        return _PackedAttnFunction.apply(q, packed, bool(causal), softmax_scale, kv_lens)
    views = packed.unbind(dim=2) if q is None else (q, *packed.unbind(dim=2))
    return HipAttnFunction.apply(*views, causal, softmax_scale, kv_lens)


_BAD_MASK = "only right-padded key_padding_mask (a kept prefix of at least one key per row) is supported"


def _lens_from_key_padding_mask(mask: torch.Tensor, packed: torch.Tensor):
    """(B, S) bool, True = keep (base.py:88-89) -> int32 key lengths, for masks that keep a prefix of each row
    (right padding, what padded batches have), and a flag that becomes non-zero if a row is anything else, which
    cannot be expressed as lengths and is refused."""
    if mask.dim() != 2 or mask.shape[1] != packed.shape[1] or mask.dtype != torch.bool:
        raise ValueError("key_padding_mask must be a bool tensor (batch, seqlen), True = keep")
    assert packed.is_cuda, "All tensors must be on CUDA device"
    if mask.device != packed.device:
        raise RuntimeError("key_padding_mask must be on the device of q, k and v")
    # pinned memory (of the CPU, whatever the default device is), which the forward's synchronisation makes readable: a flag
    # on the device cost a fill, a copy and a synchronisation of its own
    return key_padding_lens(mask, torch.zeros((), dtype=torch.int32, device="cpu", pin_memory=True))


class HipSelfAttention(nn.Module):
    """qkv [B, S, 3, H, D] -> [B, S, H, D] (hipkittens.py:122-162). Same constructor as the reference;
    `causal` and `softmax_scale` take effect here, dropout is not applied (the reference builds an
    nn.Dropout but never calls it, hipkittens.py:141,158-161)."""

    def __init__(self, causal=False, softmax_scale=None, attention_dropout=0.0, deterministic=False):
        super().__init__()
        self.causal = causal
        self.softmax_scale = softmax_scale
        self.drop = nn.Dropout(attention_dropout)
        self.deterministic = deterministic

    def forward(self, qkv, causal=None, key_padding_mask=None):
        assert qkv.dtype in [torch.float16, torch.bfloat16]
        assert qkv.is_cuda
        causal = self.causal if causal is None else causal
        return _attend(None, qkv, causal, self.softmax_scale, key_padding_mask)


class HipCrossAttention(nn.Module):
    """q [B, Sq, H, D], kv [B, Sk, 2, H_KV, D] -> [B, Sq, H, D] (hipkittens.py:165-202). Sq may differ from Sk and
    `causal` may be combined with a right-padded `key_padding_mask`, with the reference math path's alignment of the
    causal mask to the last query and the last kept key (base.py:104-116)."""

    def __init__(self, causal=False, softmax_scale=None, attention_dropout=0.0, deterministic=False):
        super().__init__()
        self.causal = causal
        self.softmax_scale = softmax_scale
        self.drop = nn.Dropout(attention_dropout)
        self.deterministic = deterministic

    def forward(self, q, kv, causal=None, key_padding_mask=None):
        batch_size = q.shape[0]
        causal = self.causal if causal is None else causal
        assert kv.shape[0] == batch_size and kv.shape[4] == q.shape[3]
        return _attend(q, kv, causal, self.softmax_scale, key_padding_mask)
