"""The native front ends and the Python checks behind them accept the same calls and give the same results."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(shape, device="cuda", generator=torch.Generator("cuda").manual_seed(7)).to(torch.bfloat16)


class _Nothing:
    """A front end that leaves every call to the Python code."""

    def __getattr__(self, name):
        return lambda *args: None


def _both(monkeypatch, call):
    got = call()
    with monkeypatch.context() as m:
        m.setattr(_native, "_front_module", _Nothing())
        ref = call()
    for a, b in zip(got if isinstance(got, tuple) else (got,), ref if isinstance(ref, tuple) else (ref,)):
        assert (a is None and b is None) or (a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b))
    return got


@pytest.mark.parametrize("layout", ["contiguous", "packed", "head_major"])
@pytest.mark.parametrize("n,nk", [(130, 130), (40, 200)])
def test_attn_fwd(monkeypatch, layout, n, nk):
    q, kv = _rand(2, n, 4, 64), _rand(2, nk, 2, 2, 64)
    k, v = kv.unbind(2)
    if layout == "contiguous":
        k, v = k.contiguous(), v.contiguous()
    if layout == "head_major":
        q, k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v))
    for lens in (None, torch.tensor([nk, 7], dtype=torch.int32, device="cuda")):
        for scale in (None, 0.3, 1):
            _both(monkeypatch, lambda: hk.attn_fwd(q, k, v, causal=True, softmax_scale=scale, kv_lens=lens))
    out, lse = torch.empty_like(q, memory_format=torch.contiguous_format), torch.empty(2, 4, 1, n, device="cuda")
    r = hk.attn_fwd(q, k, v, out=out, lse=lse)
    assert r[0] is out and r[1] is lse


def test_paged_entries(monkeypatch):
    pools = [_rand(9, 16, 2, 128) for _ in range(2)]
    table = torch.randperm(9, device="cuda").to(torch.int32)[:8].reshape(2, 4).contiguous()
    lens = torch.tensor([50, 64], dtype=torch.int32, device="cuda")
    new, start = _rand(2, 3, 2, 128), (lens - 3).to(torch.int32)
    cos, sin = _rand(64, 64), _rand(64, 64)

    def append(fn, *extra):
        k, v = (p.clone() for p in pools)
        fn(new, new, k, v, table, start, *extra)
        return k, v

    _both(monkeypatch, lambda: append(hk.paged_kv_append))
    _both(monkeypatch, lambda: append(hk.paged_kv_append_rotary, cos, sin))
    _both(monkeypatch, lambda: hk.paged_decode(_rand(2, 1, 8, 128), *pools, table, lens))
    _both(monkeypatch, lambda: hk.attn_fwd_paged(_rand(2, 3, 8, 128), *pools, table, lens))
    _both(monkeypatch, lambda: hk.rotary_bnhd(_rand(2, 60, 4, 128), cos, sin, pos_offset=4))


def test_what_was_refused_stays_refused(monkeypatch):
    q, k = _rand(2, 64, 4, 64), _rand(2, 64, 2, 64)
    lse = torch.empty(2, 4, 1, 64, device="cuda")
    calls = [
        lambda: hk.attn_fwd(q.float(), k, k),
        lambda: hk.attn_fwd(q, k, k[:, :32]),
        lambda: hk.attn_fwd(q, k.cpu(), k),
        lambda: hk.attn_fwd(q[..., ::2], k[..., ::2], k[..., ::2]),
        lambda: hk.attn_fwd(q, k, k, out=torch.empty_like(q).float()),
        lambda: hk.attn_fwd(q, k, k, lse=lse[:, :2]),
        lambda: hk.attn_fwd(q[:, :, :3].contiguous(), k, k),
        lambda: hk.attn_fwd(q, k, k, kv_lens=torch.tensor([1, 2], device="cuda")),
        lambda: hk.attn_fwd(*(t[..., :48].contiguous() for t in (q, k, k))),
        lambda: hk.rotary_bnhd(q, k[0, :32, 0], k[0, :32, 0]),
        lambda: hk.rotary_bnhd(q, k[0, :, 0].contiguous(), k[0, :, 0].contiguous(), pos_offset=-1),
    ]
    for call in calls:
        with pytest.raises(RuntimeError) as native:
            call()
        with monkeypatch.context() as m:
            m.setattr(_native, "_front_module", _Nothing())
            with pytest.raises(RuntimeError) as python:
                call()
        assert str(native.value) == str(python.value)


def test_shim_reads_tensors_and_their_subclasses_alike():
    q, k, v = _rand(1, 128, 2, 64), _rand(1, 128, 2, 64), _rand(1, 128, 2, 64)
    tk = hk.load_tk_kernel(False)
    outs = []
    named = type("Tensor", (torch.Tensor,), {})  # the class name is what the shims ask for
    for wrap in (lambda t: t, lambda t: t.as_subclass(named)):
        out, lse = torch.empty_like(q), torch.empty(1, 2, 1, 128, device="cuda")
        tk.dispatch_micro(*(wrap(t) for t in (q, k, v)), out, lse)
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(*outs)
    with pytest.raises(RuntimeError, match="Tensor must be contiguous"):
        tk.dispatch_micro(q[:, :, ::2], k, v, out, lse)
    with pytest.raises(RuntimeError, match="Tensor must be on CUDA device"):
        tk.dispatch_micro(q.cpu(), k, v, out, lse)
    with pytest.raises(RuntimeError, match="Tensor.ndim <= 4"):
        tk.dispatch_micro(q[None], k, v, out, lse)
    with pytest.raises(RuntimeError, match="torch.bfloat16"):
        tk.dispatch_micro(q.half(), k, v, out, lse)
