"""Key blocks that are shared by the CTAs of a cluster (few K/V heads): gradients against fp32 autograd, at shares that are
uneven or empty, blocks that nobody sees, key lengths, cross lengths and strided outputs; the same bits from run to run."""
import pytest
import torch

import hipkittens_b200 as hk
from hipkittens_b200 import _native
from hipkittens_b200.attention import HipCrossAttention

pytestmark = pytest.mark.gpu


def rand(*shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


def reference(q, k, v, d_o, causal, lens):
    """Gradients of softmax attention in fp64; rows that see no key give nothing."""
    B, N, H, D = q.shape
    NK, G = k.shape[1], H // k.shape[2]
    leaves = [t.double().requires_grad_() for t in (q, k, v)]
    kk, vv = (t.repeat_interleave(G, dim=2) for t in leaves[1:])
    s = torch.einsum("bnhd,bmhd->bhnm", leaves[0], kk) * D ** -0.5
    length = torch.tensor(lens or [NK] * B, device="cuda")
    col, row = torch.arange(NK, device="cuda"), torch.arange(N, device="cuda")
    keep = (col[None, None] < length[:, None, None]).expand(B, N, NK)
    if causal:
        keep = keep & (col[None, None] <= row[None, :, None] + (length - N)[:, None, None])
    p = torch.softmax(s.masked_fill(~keep[:, None], -1e30), dim=-1) * keep[:, None]
    torch.einsum("bhnm,bmhd->bnhd", p, vv).backward(d_o.double())
    return [t.grad for t in leaves]


# the cluster has 8 CTAs where blocks are few and long, 4 or 2 otherwise
@pytest.mark.parametrize("B,N,NK,H,HK,D,causal,lens", [
    (1, 1024, 1024, 8, 1, 128, True, None),
    (1, 1000, 1000, 8, 1, 64, True, None),
    (1, 520, 520, 7, 1, 128, False, None),          # 35 pairs over 8 CTAs
    (2, 300, 300, 5, 1, 64, False, None),
    (2, 900, 900, 4, 2, 128, False, None),
    (3, 1024, 640, 8, 1, 128, True, None),          # queries that see no key
    (1, 384, 2000, 8, 1, 128, True, None),          # more keys than queries: blocks of very different length
    (3, 640, 640, 8, 1, 128, False, [640, 1, 300]),  # blocks of padding
    (3, 512, 512, 8, 1, 64, True, [512, 130, 7]),   # blocks with fewer pairs than CTAs
])
def test_gradients(B, N, NK, H, HK, D, causal, lens):
    q, k, v, d_o = rand(B, N, H, D, seed=1), rand(B, NK, HK, D, seed=2), rand(B, NK, HK, D, seed=3), rand(B, N, H, D, seed=4)
    kv_lens = torch.tensor(lens, dtype=torch.int32, device="cuda") if lens else None
    o, lse = hk.attn_fwd(q, k, v, causal=causal, kv_lens=kv_lens)
    runs = []
    for _ in range(2):
        dq, d_kv = torch.empty_like(q), torch.full((B, NK, 2, HK, D), float("nan"), dtype=torch.bfloat16, device="cuda")
        _native.attn_bwd_strided(q, k, v, o, d_o, lse, dq, d_kv[:, :, 0], d_kv[:, :, 1], causal=causal, kv_lens=kv_lens)
        assert _native.device_status(0) == 0
        runs.append((dq, d_kv[:, :, 0], d_kv[:, :, 1]))
    for a, b, ref in zip(*runs, reference(q, k, v, d_o, causal, lens)):
        assert torch.equal(a, b)
        # bf16 rounding of P, dS and the result, as for the kernels that do not split
        assert float((a.double() - ref).norm() / ref.norm()) <= 5e-3
    if lens:
        for b, n in enumerate(lens):
            assert not runs[0][1][b, n:].any() and not runs[0][2][b, n:].any()


def test_the_clusters_are_taken(monkeypatch):
    """The split kernel is another instantiation, which the profiler's kernel names show."""
    q, kv = rand(1, 1024, 8, 128, seed=5).requires_grad_(), rand(1, 1024, 2, 1, 128, seed=6).requires_grad_()
    out = HipCrossAttention(causal=True)(q, kv)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out.backward(torch.ones_like(out))
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages()]
    if any("attn_bwd" in n for n in names):  # a box without the profiler's interface gives no kernels
        assert any("attn_bwd_dkdv_kernel<128, true, true>" in n for n in names), names
