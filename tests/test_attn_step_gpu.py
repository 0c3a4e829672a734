"""Attention of single-token steps (csrc/attn_step.cu) against 64 bits: every head size and group of query heads it is built for, stores
that wrap around, windows and blocks, contexts of one key up to several tiles and clusters, and every term of its epilogue."""
import math
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


@pytest.mark.parametrize("D,H,G,pos,cap,window,chunk,extra", [
    (128, 4, 4, [0, 15, 16, 700], 300, 300, 0, ""),
    (128, 8, 2, [5, 299, 300, 1000], 256, 256, 0, "gate"),
    (128, 16, 2, [40, 41], 1 << 10, 1 << 30, 0, "sink gate_head cap"),
    (128, 2, 1, [63, 64, 65, 130], 64, 1 << 30, 64, "vrot"),
    (64, 4, 2, [1, 2000], 512, 100, 0, "vrot_halves gate"),
    (64, 12, 4, [33, 90, 17], 128, 128, 0, "sink"),
    (256, 16, 1, [3, 500, 1500], 2048, 1 << 30, 0, "gate_head"),
    (256, 6, 2, [129] * 70, 200, 90, 0, "cap vrot"),
])
def test_against_64_bits(D, H, G, pos, cap, window, chunk, extra):
    from llark_b200 import ops

    torch.manual_seed(D + H + len(pos))
    n, dev, extra = len(pos), "cuda", extra.split()
    ints = lambda v: torch.tensor(v, device=dev, dtype=torch.int32)  # noqa: E731
    slots = torch.randperm(n + 2)[:n].tolist()
    st = types.SimpleNamespace(n_tok=n, n_seq=n, max_len=1, tok_seq=ints(range(n)), cu=ints(range(n + 1)), pos0=ints(pos), slot=ints(slots))
    q, k, v = (torch.randn(*s, device=dev).to(BF16) for s in ((n, H * D), (n + 2, cap, G * D), (n + 2, cap, G * D)))
    scale = torch.rand(H, device=dev) / math.sqrt(D) + 0.02
    sink = torch.randn(H, device=dev) if "sink" in extra else None
    per_head = "gate_head" in extra
    gate = torch.randn(n, H if per_head else H * D, device=dev) if per_head or "gate" in extra else None
    softcap = 3.0 if "cap" in extra else 0.0
    vrot = "vrot" in extra or "vrot_halves" in extra
    vfreq = torch.rand(D // 2, device=dev) if vrot else None
    out = ops.seq_swa_attn(q, None, None, k, v, gate, gate.stride(0) if gate is not None else 0, scale, st, H, G, D, D, window, cap,
                           from_ring_only=True, sink=sink, gate_per_head=per_head, chunk=chunk, softcap=softcap, vfreq=vfreq,
                           v_interleaved="vrot" in extra, out_scale=0.7).view(n, H, D)
    for b, p in enumerate(pos):
        lo = p // chunk * chunk if chunk else max(0, p - window + 1)
        at = torch.arange(lo, p + 1, device=dev) % cap
        kb, vb = (t[slots[b], at].view(-1, G, D).repeat_interleave(H // G, 1).to(F64) for t in (k, v))
        s = torch.einsum("hd,jhd->hj", q[b].view(H, D).to(F64), kb) * scale.to(F64)[:, None]
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if sink is not None:
            s = torch.cat([s, sink.to(F64)[:, None]], 1)
        w = torch.softmax(s, 1)[:, :kb.shape[0]]
        o = torch.einsum("hj,jhd->hd", w, vb) * 0.7
        if vrot:
            a = float(p) * vfreq  # the angle is an fp32 product by definition
            c, si = a.to(F64).cos(), a.to(F64).sin()
            u, x = (o[:, 0::2], o[:, 1::2]) if "vrot" in extra else (o[:, :D // 2], o[:, D // 2:])
            y = torch.stack([u * c + x * si, x * c - u * si], -1)
            o = y.flatten(-2) if "vrot" in extra else y.transpose(-1, -2).reshape(H, D)
        if gate is not None:
            o = o * torch.sigmoid((gate[b].view(H, -1)).to(F64))
        # one rounding to eight bits (2^-8 of a value at most); everything before it is fp32
        assert ((out[b].to(F64) - o).norm() / o.norm()).item() < 2.0 ** -8, b


def test_cache_rows_off_16_byte_boundaries_and_empty_rows():
    from llark_b200 import ops

    torch.manual_seed(3)
    B, S, NH = 3, 96, 2
    q = torch.randn(B * NH * 128 + 1, device="cuda").to(BF16)[1:].view(B, NH * 128)  # two bytes off
    k, v = (torch.randn(B, S, NH * 128, device="cuda").to(BF16) for _ in range(2))
    lens = torch.tensor([0, 1, 96], device="cuda", dtype=torch.int32)
    got, want = ops.attn_decode(q, k, v, lens, NH, 128), ops.attn_decode(q.clone(), k, v, lens, NH, 128)
    assert want[0].abs().max().item() == 0
    assert ((got - want).float().norm() / want.float().norm()).item() < 2.0 ** -7


@pytest.mark.parametrize("B,S,NH,pos", [(1, 64, 2, 0), (3, 300, 4, 16), (2, 2000, 2, 1777), (40, 128, 16, 127)])
def test_packed_projection_is_that_of_the_stores(B, S, NH, pos):
    """The form that takes the new key and value from the packed projection stores them and gives what the stored ones give."""
    from llark_b200 import ops

    torch.manual_seed(pos + B)
    H = NH * 128
    qkv = torch.randn(B, 3 * H + 8, device="cuda").to(BF16)[:, :3 * H]
    k, v = (torch.randn(B, S, H, device="cuda").to(BF16) for _ in range(2))
    want_k, want_v = k.clone(), v.clone()
    want_k[:, pos], want_v[:, pos] = qkv[:, H:2 * H], qkv[:, 2 * H:]
    got = ops.attn_decode_packed(qkv, k, v, pos, NH, 128)
    assert torch.equal(k, want_k) and torch.equal(v, want_v)
    lens = torch.full((B,), pos + 1, device="cuda", dtype=torch.int32)
    assert torch.equal(got, ops.attn_decode(qkv[:, :H].contiguous(), want_k, want_v, lens, NH, 128))


@pytest.mark.parametrize("D,H,G", [(128, 4, 1), (64, 4, 4), (256, 4, 2)])
def test_scores_that_are_not_numbers_reach_the_result(D, H, G):
    """A query that is NaN beside a sink, and sixteen keys that are NaN, all that one warp takes at a time: NaN for the heads that read
    them; scores of minus infinity weigh nothing; other requests and heads as without."""
    from llark_b200 import ops

    torch.manual_seed(D)
    n, cap, nan, inf, dev = 4, 200, float("nan"), float("inf"), "cuda"
    ints = lambda v: torch.tensor(v, device=dev, dtype=torch.int32)  # noqa: E731
    st = types.SimpleNamespace(n_tok=n, n_seq=n, max_len=1, tok_seq=ints(range(n)), cu=ints(range(n + 1)), pos0=ints([70] * n), slot=ints(range(n)))
    q, k, v = (torch.randn(*s, device=dev).to(BF16) for s in ((n, H, D), (n, cap, G, D), (n, cap, G, D)))
    scale, sink = torch.full((H,), 0.1, device=dev), torch.randn(H, device=dev)

    def run(q, k):
        return ops.seq_swa_attn(q.view(n, H * D), None, None, k.view(n, cap, G * D), v.view(n, cap, G * D), None, 0, scale, st, H, G, D, D, cap,
                                cap, from_ring_only=True, sink=sink).view(n, H, D)

    want = run(q, k)
    q2, k2 = q.clone(), k.clone()
    q2[0, 1, 3] = nan
    k2[1, 16:32, 0, :] = nan
    q2[3, :, 0], k2[3, :, :, 0] = 1.0, 0.0
    k2[3, :50, :, 0] = -inf
    got = run(q2, k2)
    heads = torch.arange(H, device=dev)
    assert torch.equal(got[0].isnan().all(1), heads == 1) and torch.equal(got[0].isnan().any(1), heads == 1)
    assert torch.equal(got[1].isnan().all(1), heads < H // G) and torch.equal(got[1].isnan().any(1), heads < H // G)
    keep = torch.ones(n, H, dtype=torch.bool, device=dev)
    keep[0, 1], keep[1, :H // G], keep[3] = False, False, False
    assert torch.equal(got[keep], want[keep])
    s = torch.einsum("hd,jhd->hj", q2[3].to(F64), k2[3, 50:71].repeat_interleave(H // G, 1).to(F64)) * 0.1
    w = torch.softmax(torch.cat([s, sink.to(F64)[:, None]], 1), 1)[:, :-1]
    ref = torch.einsum("hj,jhd->hd", w, v[3, 50:71].repeat_interleave(H // G, 1).to(F64))
    assert ((got[3].to(F64) - ref).norm() / ref.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("B,H,I,pos", [(1, 256, 512, 0), (9, 256, 520, 5), (33, 512, 1000, 17), (64, 256, 264, 31)])
def test_layers_of_a_decode_step_in_one_call(B, H, I, pos):
    """The layers issued by one call against the single ops of the same step: the same launches, so the same bits, in x and in the caches."""
    from llark_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B + H)
    r = lambda *s, std=1.0: (std * torch.randn(*s, device="cuda", generator=g)).to(torch.bfloat16)  # noqa: E731
    L, NH, s_max = 3, H // 128, 40
    cos, sin = r(s_max, 128), r(s_max, 128)
    w = [dict(norm1=r(H), qkv=r(3 * H, H, std=H ** -0.5), o=r(H, H, std=H ** -0.5), norm2=r(H), gate_up=r(2 * I, H, std=H ** -0.5),
              down=r(H, I, std=I ** -0.5), k=r(B, s_max, H), v=r(B, s_max, H)) for _ in range(L)]
    x0 = r(B, H)
    rstd = torch.empty(B, device="cuda", dtype=torch.float32)
    caches = [(a["k"].clone(), a["v"].clone()) for a in w]
    x = x0
    for a, (k, v) in zip(w, caches):
        qkv = ops.gemm(ops.rmsnorm_fwd(x, a["norm1"], 1e-5, rstd=rstd), a["qkv"], rope=(cos[pos:], sin[pos:], 1, 2 * H))
        mid = ops.gemm(ops.attn_decode_packed(qkv, k, v, pos, NH, 128), a["o"], residual=x)
        act = ops.gemm(ops.rmsnorm_fwd(mid, a["norm2"], 1e-5, rstd=rstd), a["gate_up"], swiglu=True)
        x = ops.gemm(act, a["down"], residual=mid)
    table = (ops.DecodeLayer * L)(*[ops.DecodeLayer(**{n: t.data_ptr() for n, t in a.items()}) for a in w])
    got = x0.clone()
    ops.decode_layers(table, got, cos[pos:], sin[pos:], pos, s_max, I, NH, 1e-5, rstd)
    assert torch.equal(got, x)
    assert all(torch.equal(a["k"], k) and torch.equal(a["v"], v) for a, (k, v) in zip(w, caches))
