"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values. `prepare` makes what a user's program holds before the call (inputs drawn from the
seed, caller-owned outputs and workspaces, the module), `run` is one pass through the public entry points:

    forward    tk_kernel.dispatch_micro(q, k, v, out, lse): the harness's call, outputs owned by the caller
    prefill    an inference prompt: rotary_bnhd of q and of k, then causal attn_fwd
    backward   the three calls dispatch_prep, dispatch_bwd_combined, dispatch_dq_shuffle
    train_self HipSelfAttention on a packed qkv projection, forward and loss.backward()
    train_cross HipCrossAttention on q and a packed kv (grouped heads), forward and loss.backward()
    decode     one decode step of one layer: append of the new token's rotated K and of V (optional), then paged_decode
    chunk      chunked prefill: append of the chunk with the rotary embedding of K, then attn_fwd_paged
"""
import math

import torch

import hipkittens_b200 as hk
from hipkittens_b200.attention import HipCrossAttention, HipSelfAttention

PAGE = 16


def listed():
    return [
        # the smallest call of the test configurations: one 256-token sequence; what counts is latency and host work
        dict(name="forward_small_d64", kind="forward", b=1, n=256, h=8, hkv=2, d=64, causal=False),
        # the reference README's default shape, the headline workload of bench.py
        dict(name="forward_gqa_d128", kind="forward", b=16, n=2048, h=64, hkv=8, d=128, causal=False),
        # long-context causal forward, bench.py's second workload
        dict(name="forward_causal_long_d128", kind="forward", b=4, n=8192, h=64, hkv=8, d=128, causal=True),
        # small head dimension, as many K/V heads as heads: bench.py's third workload
        dict(name="forward_mha_d64", kind="forward", b=16, n=4096, h=16, hkv=16, d=64, causal=False),
        # one user's prompt of an odd length in front of a decode loop
        dict(name="prefill_one_prompt", kind="prefill", b=1, n=1511, h=32, hkv=8, d=128, causal=True),
        # a short training step: gradients of a small model, where launches and host work count
        dict(name="train_small_d128", kind="train_cross", b=2, n=384, h=8, hkv=2, d=128, causal=True, padded=False),
        # BERT-style fine-tuning: a batch of right-padded sequences with a key_padding_mask
        dict(name="train_padded_d64", kind="train_self", b=16, n=512, h=16, hkv=16, d=64, causal=False, padded=True),
        # a Llama-style training step with grouped heads
        dict(name="train_causal_gqa_d128", kind="train_cross", b=4, n=4096, h=32, hkv=8, d=128, causal=True, padded=False),
        # the backward harness at the default shape, through the three calls of the training call site
        dict(name="backward_gqa_d128", kind="backward", b=16, n=2048, h=64, hkv=8, d=128, causal=False),
        # a full serving batch: bench.py's paged decode, 64 sequences in a 40 000-page pool
        dict(name="decode_batch64", kind="decode", b=64, lo=512, hi=8192, h=64, hkv=8, d=128, append=False, pool=40000),
        # one interactive user: a single sequence, append and attention of one token
        dict(name="decode_single", kind="decode", b=1, lo=3000, hi=3500, h=32, hkv=8, d=128, append=True, pool=4096),
        # chunked prefill of a few sequences against what they have cached
        dict(name="chunk_prefill", kind="chunk", b=4, t=512, lo=2048, hi=8192, h=64, hkv=8, d=128, pool=4096),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _max_cost():
    works = [work(c) for c in listed()]
    return max(w["flops"] for w in works), max(w["bytes"] for w in works)


def draw(rng):
    """One more case of the listed ranges: every kind, both head dimensions, any length, group sizes 1 to 8."""
    max_flops, max_bytes = _max_cost()
    while True:
        kind = rng.choice(["forward", "prefill", "backward", "train_self", "train_cross", "decode", "chunk"])
        d = 128 if kind in ("decode", "chunk") else rng.choice([64, 128])
        hkv = rng.choice([1, 2, 4, 8, 8, 16])
        g = rng.choice([1, 1, 2, 3, 4, 4, 8])
        if kind == "train_self":
            hkv, g = rng.choice([8, 12, 16]), 1
        h = hkv * g
        if kind in ("decode", "chunk"):
            b = _log_int(rng, 1, 64 if kind == "decode" else 16)
            hi = _log_int(rng, 256, 16384)
            lo = max(1, int(hi * rng.uniform(0.1, 0.95)))
            case = dict(kind=kind, b=b, lo=lo, hi=hi, h=h, hkv=hkv, d=d)
            if kind == "decode":
                case["append"] = rng.random() < 0.5
            else:
                case["t"] = min(lo, _log_int(rng, 16, 2048))
            case["pool"] = b * ((hi + PAGE - 1) // PAGE) + rng.randrange(1, 200)
        else:
            n = _log_int(rng, 128, 8192)
            if rng.random() < 0.5:
                n = (n + 127) // 128 * 128
            b = _log_int(rng, 1, 16)
            case = dict(kind=kind, b=b, n=n, h=h, hkv=hkv, d=d, causal=True if kind == "prefill" else rng.random() < 0.5)
            if kind.startswith("train"):
                case["padded"] = not case["causal"] and rng.random() < 0.5
        w = work(case)
        if w["flops"] <= max_flops and w["bytes"] <= max_bytes:
            return case


def _tables(rows, d, dev):
    """cos and sin of the rotary embedding, bf16 [rows, d / 2] (the reference harness's get_cos_sin)."""
    inv = 10000.0 ** (-torch.arange(0, d, 2, dtype=torch.float32, device=dev) / d)
    ang = torch.arange(rows, dtype=torch.float32, device=dev)[:, None] * inv[None]
    return ang.cos().to(torch.bfloat16), ang.sin().to(torch.bfloat16)


def _lens(case):
    """Context lengths of the paged kinds: fixed by the case (the work of a case does not depend on the seed), spread
    evenly over [lo, hi]."""
    b, lo, hi = case["b"], case["lo"], case["hi"]
    if b == 1:
        return [(lo + hi) // 2]
    lens = [lo + (hi - lo) * i // (b - 1) for i in range(b)]
    return [lens[(i * 29 + 7) % b] for i in range(b)] if math.gcd(29, b) == 1 else lens


def _padded_lens(case):
    n, b = case["n"], case["b"]
    return [max(1, n - (n * 7 // 8) * ((i * 5) % b) // b) for i in range(b)]


def prepare(case, seed):
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(seed)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device=dev, dtype=torch.bfloat16)

    kind, b, h, hkv, d = case["kind"], case["b"], case["h"], case["hkv"], case["d"]
    st = {"case": case}
    if kind in ("decode", "chunk"):
        lens = _lens(case)
        t = case.get("t", 1)
        pages = [(x + PAGE - 1) // PAGE for x in lens]
        perm = torch.randperm(case["pool"], generator=gen, device=dev).to(torch.int32)
        table = torch.zeros((b, max(pages)), dtype=torch.int32, device=dev)
        at = 0
        for s, c in enumerate(pages):
            table[s, :c] = perm[at:at + c]
            at += c
        st.update(
            q=rand(b, t, h, d), k_pages=rand(case["pool"], PAGE, hkv, d), v_pages=rand(case["pool"], PAGE, hkv, d),
            table=table, ctx=torch.tensor(lens, dtype=torch.int32, device=dev),
            out=torch.empty((b, t, h, d), dtype=torch.bfloat16, device=dev),
            lse=torch.empty((b, h, 1, t), dtype=torch.float32, device=dev))
        if kind == "decode":
            need = hk.paged_decode_workspace_bytes(b, h, d, table.shape[1])
            st["workspace"] = torch.empty(max(need, 256), dtype=torch.uint8, device=dev)
        if kind == "chunk" or case["append"]:
            st["k_new"], st["v_new"] = rand(b, t, hkv, d), rand(b, t, hkv, d)
            st["start"] = torch.tensor([x - t for x in lens], dtype=torch.int32, device=dev)
            st["cos"], st["sin"] = _tables(max(lens), d, dev)
        return st
    n, causal = case["n"], case["causal"]
    if kind in ("train_self", "train_cross"):
        if kind == "train_self":
            st["x"] = (rand(b, n, 3, h, d).requires_grad_(),)
            st["module"] = HipSelfAttention(causal=causal)
        else:
            st["x"] = (rand(b, n, h, d).requires_grad_(), rand(b, n, 2, hkv, d).requires_grad_())
            st["module"] = HipCrossAttention(causal=causal)
        st["d_o"] = rand(b, n, h, d)
        st["mask"] = None
        if case["padded"]:
            lens = torch.tensor(_padded_lens(case), device=dev)
            st["mask"] = torch.arange(n, device=dev)[None] < lens[:, None]
        return st
    st.update(q=rand(b, n, h, d), k=rand(b, n, hkv, d), v=rand(b, n, hkv, d))
    if kind == "prefill":
        st["cos"], st["sin"] = _tables(n, d, dev)
        return st
    st["out"] = torch.empty((b, n, h, d), dtype=torch.bfloat16, device=dev)
    st["lse"] = torch.empty((b, h, 1, n), dtype=torch.float32, device=dev)
    if kind == "forward":
        st["tk"] = hk.load_tk_kernel(causal)
    else:
        hk.attn_fwd(st["q"], st["k"], st["v"], causal=causal, out=st["out"], lse=st["lse"])
        st["d_o"] = rand(b, n, h, d)
        st["bkwd"], st["prep"] = hk.load_tk_kernel_bkwd(causal), hk.load_tk_kernel_bkwd_prep(causal)
        st["delta"] = torch.empty((b, h, 1, n), dtype=torch.float32, device=dev)
        st["dq_in"] = torch.empty((b, h, n, d), dtype=torch.bfloat16, device=dev)
        st["dq"] = torch.empty((b, n, h, d), dtype=torch.bfloat16, device=dev)
        st["dk"] = torch.empty((b, n, hkv, d), dtype=torch.bfloat16, device=dev)
        st["dv"] = torch.empty((b, n, hkv, d), dtype=torch.bfloat16, device=dev)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "forward":
        st["tk"].dispatch_micro(st["q"], st["k"], st["v"], st["out"], st["lse"])
        return st["out"], st["lse"]
    if kind == "prefill":
        q = hk.rotary_bnhd(st["q"], st["cos"], st["sin"])
        k = hk.rotary_bnhd(st["k"], st["cos"], st["sin"])
        out, lse = hk.attn_fwd(q, k, st["v"], causal=True)
        return out, lse, q, k
    if kind == "backward":
        st["prep"].dispatch_prep(st["out"], st["d_o"], st["delta"])
        st["bkwd"].dispatch_bwd_combined(st["q"], st["k"], st["v"], st["d_o"], st["dq_in"], st["dk"], st["dv"],
                                         st["lse"], st["delta"])
        st["prep"].dispatch_dq_shuffle(st["dq_in"], st["dq"])
        return st["dq"], st["dk"], st["dv"], st["delta"]
    if kind in ("train_self", "train_cross"):
        for x in st["x"]:
            x.grad = None
        out = st["module"](*st["x"], key_padding_mask=st["mask"])
        out.backward(st["d_o"])
        return (out.detach(),) + tuple(x.grad for x in st["x"])
    if kind == "decode":
        if case["append"]:
            hk.paged_kv_append_rotary(st["k_new"], st["v_new"], st["k_pages"], st["v_pages"], st["table"], st["start"],
                                      st["cos"], st["sin"])
        hk.paged_decode(st["q"], st["k_pages"], st["v_pages"], st["table"], st["ctx"], out=st["out"], lse=st["lse"],
                        workspace=st["workspace"])
    else:
        hk.paged_kv_append_rotary(st["k_new"], st["v_new"], st["k_pages"], st["v_pages"], st["table"], st["start"],
                                  st["cos"], st["sin"])
        hk.attn_fwd_paged(st["q"], st["k_pages"], st["v_pages"], st["table"], st["ctx"], causal=True, out=st["out"],
                          lse=st["lse"])
    if "k_new" in st:
        return st["out"], st["lse"], st["k_pages"], st["v_pages"]
    return st["out"], st["lse"]


def work(case):
    """Two products of the forward, five of the backward, over the (query, key) pairs that the masks leave; every input
    once and every output once."""
    kind, b, h, hkv, d = case["kind"], case["b"], case["h"], case["hkv"], case["d"]
    if kind in ("decode", "chunk"):
        lens, t = _lens(case), case.get("t", 1)
        pairs = sum(t * (x - t) + t * (t + 1) // 2 for x in lens)
        kv = 2 * sum(lens) * hkv * d * 2
        rows = b * t
        new = 2 * (2 * rows * hkv * d * 2) if "t" in case or case["append"] else 0  # read, and written into the pages
        return {"flops": 4.0 * pairs * h * d, "bytes": float(kv + new + rows * h * (4 * d + 4))}
    n = case["n"]
    if case.get("padded"):
        pairs = n * sum(_padded_lens(case))
    else:
        pairs = b * (n * (n + 1) // 2 if case["causal"] else n * n)
    q_bytes, kv_bytes, row_bytes = 2 * b * n * h * d, 2 * b * n * hkv * d, 4 * b * n * h
    fwd = 4.0 * pairs * h * d
    if kind == "forward":
        return {"flops": fwd, "bytes": float(2 * q_bytes + 2 * kv_bytes + row_bytes)}
    if kind == "prefill":
        return {"flops": fwd, "bytes": float(2 * q_bytes + 3 * kv_bytes + row_bytes + q_bytes)}
    if kind == "backward":  # q, o, dO, lse and k, v in; delta, dQ, dK, dV out
        return {"flops": 2.5 * fwd, "bytes": float(4 * q_bytes + 4 * kv_bytes + 2 * row_bytes)}
    # training: q, k, v, dO in, O and the three gradients out
    return {"flops": 3.5 * fwd, "bytes": float(4 * q_bytes + 4 * kv_bytes)}


def tolerance(case):
    """Four times what each kind differs by from the same path in 64 bits: rel 2.3e-3 for O (its rounding to bf16 and
    that of P) and 2.6e-3 for the gradients; the largest single difference, over the rms, 0.026 for O and 0.13 for
    causal gradients, whose first rows are far larger than the rms."""
    return {"rel": 1e-2, "max": 0.1 if case["kind"] in ("forward", "prefill", "decode", "chunk") else 0.5}
