"""Tensors without storage (what torch.func's transforms hand to a function) are refused by every front end with the Python
checks' own error, whether the native code is in front of them or not. Nothing is launched. On the CPU the tensors are
fakes that call themselves CUDA tensors, which is as far as a call gets that does not use its data."""
import contextlib
import types

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import hipkittens_b200 as hk
from hipkittens_b200 import _native


class _Nothing:
    """A front end that leaves every call to the Python code."""

    def __getattr__(self, name):
        return lambda *args: None


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16, device="cuda")


def _i32(*shape):
    return torch.zeros(shape, dtype=torch.int32, device="cuda")


def _calls():
    """name -> (tensors, the call on them)"""
    q, k, v = _bf16(2, 64, 4, 128), _bf16(2, 64, 2, 128), _bf16(2, 64, 2, 128)
    lse = torch.zeros(2, 4, 1, 64, device="cuda")
    paged = _bf16(9, 16, 2, 128), _bf16(9, 16, 2, 128), _i32(2, 4), _i32(2)
    cos, sin = _bf16(64, 64), _bf16(64, 64)
    return {
        "attn_fwd": ((q, k, v), hk.attn_fwd),
        "attn_fwd_out": ((q, k, v, _bf16(2, 64, 4, 128)), lambda q, k, v, out: hk.attn_fwd(q, k, v, out=out)),
        "attn_fwd_lens": ((q, k, v, _i32(2)), lambda q, k, v, lens: hk.attn_fwd(q, k, v, kv_lens=lens)),
        "attn_bwd_strided": ((q, k, v, q, q, lse, q, k, v), _native.attn_bwd_strided),
        "rotary_bnhd": ((q, cos, sin), hk.rotary_bnhd),
        "paged_decode": ((_bf16(2, 1, 4, 128), *paged), hk.paged_decode),
        "attn_fwd_paged": ((_bf16(2, 3, 4, 128), *paged), hk.attn_fwd_paged),
        "paged_kv_append": ((_bf16(2, 3, 2, 128), _bf16(2, 3, 2, 128), *paged), hk.paged_kv_append),
        "paged_kv_append_rotary": ((_bf16(2, 3, 2, 128), _bf16(2, 3, 2, 128), *paged, cos, sin), hk.paged_kv_append_rotary),
    }


@pytest.mark.parametrize("where", ["cpu", pytest.param("gpu", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("transform", ["vmap", "grad", "vmap_first", "grad_first"])
@pytest.mark.parametrize("name", ["attn_fwd", "attn_fwd_out", "attn_fwd_lens", "attn_bwd_strided", "rotary_bnhd",
                                  "paged_decode", "attn_fwd_paged", "paged_kv_append", "paged_kv_append_rotary"])
def test_a_tensor_without_storage_is_refused(native_built, monkeypatch, name, transform, where):
    if where == "cpu":
        monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=0))
    with FakeTensorMode() if where == "cpu" else contextlib.nullcontext():
        tensors, call = _calls()[name]
        # the tensors that the transform wraps: all that it can, or the first alone
        wrapped = [i for i, t in enumerate(tensors) if t.is_floating_point() or transform == "vmap"]
        if transform.endswith("first"):
            wrapped = [0]
        if transform.startswith("vmap"):
            stacked = [torch.stack([t, t]) if i in wrapped else t for i, t in enumerate(tensors)]
            in_dims = tuple(0 if i in wrapped else None for i in range(len(tensors)))
            run = lambda: torch.func.vmap(call, in_dims=in_dims)(*stacked)  # noqa: E731
        else:
            run = lambda: torch.func.grad(call, argnums=tuple(wrapped))(*tensors)  # noqa: E731
        launches = hk.kernel_launch_count()
        with pytest.raises(RuntimeError, match="doesn't have storage") as native:
            run()
        monkeypatch.setattr(_native, "_front_module", _Nothing())
        with pytest.raises(RuntimeError, match="doesn't have storage") as python:
            run()
    assert str(native.value) == str(python.value)
    assert hk.kernel_launch_count() == launches
