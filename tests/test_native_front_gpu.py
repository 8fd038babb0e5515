"""The native front ends and the Python checks behind them accept the same calls and give the same results."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native

pytestmark = pytest.mark.gpu


_gen = None


@pytest.fixture(autouse=True)
def _seeded():
    """One generator per test, so that no two tensors of a test are alike: an argument taken for another shows."""
    global _gen
    _gen = torch.Generator("cuda").manual_seed(7)


def _rand(*shape):
    return torch.randn(shape, device="cuda", generator=_gen).to(torch.bfloat16)


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
    k_new, v_new, start = _rand(2, 3, 2, 128), _rand(2, 3, 2, 128), (lens - 3).to(torch.int32)
    cos, sin = _rand(64, 64), _rand(64, 64)
    q1, q3, x = _rand(2, 1, 8, 128), _rand(2, 3, 8, 128), _rand(2, 60, 4, 128)

    def append(fn, *extra):
        k, v = (p.clone() for p in pools)
        fn(k_new, v_new, k, v, table, start, *extra)
        return k, v

    _both(monkeypatch, lambda: append(hk.paged_kv_append))
    _both(monkeypatch, lambda: append(hk.paged_kv_append_rotary, cos, sin))
    for scale in (None, 0.3):
        _both(monkeypatch, lambda: hk.paged_decode(q1, *pools, table, lens, softmax_scale=scale))
        _both(monkeypatch, lambda: hk.attn_fwd_paged(q3, *pools, table, lens, causal=True, softmax_scale=scale))
    _both(monkeypatch, lambda: hk.rotary_bnhd(x, cos, sin, pos_offset=4))
    need = hk.paged_decode_workspace_bytes(2, 8, 128, 4)
    out, lse = torch.empty_like(q1), torch.empty(2, 8, 1, 1, device="cuda")
    r = _both(monkeypatch, lambda: hk.paged_decode(q1, *pools, table, lens, out=out, lse=lse,
                                                   workspace=torch.empty(max(need, 256), dtype=torch.uint8, device="cuda")))
    assert r[0] is out and r[1] is lse


@pytest.mark.parametrize("causal", [False, True])
def test_attn_bwd_strided(monkeypatch, causal):
    q, kv, d_o = _rand(2, 130, 4, 64), _rand(2, 200, 2, 2, 64), _rand(2, 130, 4, 64)
    k, v = kv.unbind(2)
    for lens in (None, torch.tensor([200, 140], dtype=torch.int32, device="cuda")):
        for scale in (None, 0.3, 1):
            o, lse = hk.attn_fwd(q, k, v, causal=causal, softmax_scale=scale, kv_lens=lens)

            def grads():
                dq, dkv = torch.full_like(q, 7), torch.full_like(kv, 7)
                _native.attn_bwd_strided(q, k, v, o, d_o, lse, dq, *dkv.unbind(2), causal=causal, softmax_scale=scale,
                                         kv_lens=lens)
                return dq, dkv

            dq, dkv = _both(monkeypatch, grads)
            delta = hk.attn_bwd_prep(o, d_o)
            ref = hk.attn_bwd(q, k.contiguous(), v.contiguous(), d_o, lse, delta, causal=causal, softmax_scale=scale,
                              kv_lens=lens)
            for got, want in zip((dq, dkv[:, :, 0], dkv[:, :, 1]), ref):
                assert torch.equal(got, want)


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
    q1, pool = _rand(2, 1, 4, 128), _rand(9, 16, 2, 128)
    table, lens = torch.zeros(2, 4, dtype=torch.int32, device="cuda"), torch.ones(2, dtype=torch.int32, device="cuda")
    new, tab = _rand(2, 1, 2, 128), _rand(64, 64)
    calls += [
        lambda: hk.paged_decode(q1.float(), pool, pool, table, lens),
        lambda: hk.paged_decode(q1, pool, pool[:8], table, lens),
        lambda: hk.paged_decode(q1, pool, pool, table.long(), lens),
        lambda: hk.paged_decode(q1, pool, pool, table, lens[:1]),
        lambda: hk.paged_decode(q1, pool, pool, table, lens.cpu()),
        lambda: hk.paged_decode(q1, pool, pool, table[:, ::2], lens),
        lambda: hk.paged_decode(q1[:, :, :3].contiguous(), pool, pool, table, lens),
        lambda: hk.paged_decode(q1, pool, pool, table, lens, workspace=torch.empty(16, dtype=torch.uint8, device="cuda")),
        lambda: hk.attn_fwd_paged(q1, pool, pool[..., :64].contiguous(), table, lens),
        lambda: hk.attn_fwd_paged(q1, pool, pool, table, lens, out=q1.float()),
        lambda: hk.paged_kv_append(new, new.float(), pool, pool, table, lens),
        lambda: hk.paged_kv_append(new, new, pool, pool, table, lens.float()),
        lambda: hk.paged_kv_append_rotary(new, new, pool, pool, table, lens, tab, tab[:32]),
        lambda: _native.attn_bwd_strided(q, k, k, q, q[:, :32], lse, q.clone(), k.clone(), k.clone()),
        lambda: _native.attn_bwd_strided(q, k, k, q, q, lse[:, :2], q.clone(), k.clone(), k.clone()),
        lambda: _native.attn_bwd_strided(q, k, k, q, q, lse, q.float(), k.clone(), k.clone()),
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
