"""Sliding-window attention of prompts with heads of 128 (csrc/seq_swa_tc.cu) against 64 bits: packed requests of unlike lengths, keys
from the step and from rings that wrap around, windows and blocks, tiles that a row does not see, and every term of the epilogue."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F64 = torch.bfloat16, torch.float64


@pytest.mark.parametrize("H,G,lens,pos,cap,window,chunk,extra", [
    (4, 2, [65, 1, 130], [0, 0, 0], 64, 64, 0, ""),
    (4, 1, [128, 127, 129], [0, 1, 700], 256, 100, 0, "gate"),
    (2, 2, [300, 200], [5, 1000], 1024, 1024, 0, "sink gate_head"),
    (6, 2, [257, 66], [200, 64], 256, 1 << 30, 64, "slice"),
    (3, 3, [500], [33], 1024, 1 << 30, 192, "sink gate"),
    (2, 1, [1400], [0], 1, 1, 0, "slice"),
])
def test_against_64_bits(H, G, lens, pos, cap, window, chunk, extra):
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    torch.manual_seed(H + sum(lens))
    n, D, dev, extra, nan = sum(lens), 128, "cuda", extra.split(), float("nan")
    slots = torch.randperm(len(lens) + 2)[:len(lens)].tolist()
    st = StepLayout(lens, pos, slots, dev)
    q, k, v = (torch.randn(n, x * D, device=dev).to(BF16) for x in (H, G, G))
    kring, vring = (torch.full((len(lens) + 2, cap, G * D), nan, device=dev, dtype=BF16) for _ in range(2))
    ks, vs = [], []  # all keys and values of each request, by position
    for b, (ln, p) in enumerate(zip(lens, pos)):
        old_k, old_v = (torch.randn(p, G * D, device=dev).to(BF16) for _ in range(2))
        at = torch.arange(max(0, p - cap), p, device=dev)
        kring[slots[b], at % cap], vring[slots[b], at % cap] = old_k[at], old_v[at]
        a = st.cu_host[b]
        ks.append(torch.cat([old_k, k[a:a + ln]]))
        vs.append(torch.cat([old_v, v[a:a + ln]]))
    scale = (torch.rand(H, device=dev) + 0.3) / math.sqrt(D)
    scale[0] *= 20  # large scores: maxima that move by more than 2^8 between tiles
    sink = torch.randn(H, device=dev) if "sink" in extra else None
    per_head = "gate_head" in extra
    gate = torch.randn(n, H if per_head else H * D, device=dev) if per_head or "gate" in extra else None
    wide = torch.zeros(n, H * D + 8, device=dev, dtype=BF16)
    out = wide[:, 8:] if "slice" in extra else None
    o = ops.seq_swa_attn(q, k, v, kring, vring, gate, gate.stride(0) if gate is not None else 0, scale, st, H, G, D, D, window, cap,
                         from_ring_only=False, sink=sink, gate_per_head=per_head, chunk=chunk, out=out, out_scale=0.7)
    for b, (ln, p) in enumerate(zip(lens, pos)):
        a = st.cu_host[b]
        qp, kp = torch.arange(p, p + ln, device=dev)[:, None], torch.arange(p + ln, device=dev)
        seen = (kp <= qp) & ((kp >= qp // chunk * chunk) if chunk else (kp > qp - window))
        kb, vb = (t[b].view(-1, G, D).repeat_interleave(H // G, 1).to(F64) for t in (ks, vs))
        s = torch.einsum("ihd,jhd->hij", q[a:a + ln].view(ln, H, D).to(F64), kb) * scale.to(F64)[:, None, None]
        s = s.masked_fill(~seen, -math.inf)
        s = torch.cat([s, (sink.to(F64)[:, None, None].expand(H, ln, 1) if sink is not None else torch.full_like(s[..., :1], -math.inf))], 2)
        w = torch.softmax(s, 2)[..., :-1]
        f = torch.sigmoid(gate[a:a + ln].to(F64)).view(ln, H, -1) * 0.7 if gate is not None else 0.7
        want = torch.einsum("hij,jhd->ihd", w, vb) * f
        # Probabilities and results are rounded to the eight significant bits of bf16: 2^-8 of a term at most (half of the spacing
        # 2^-7 above 1). The scores are fp32 sums of 128 exact products.
        ds = torch.einsum("ihd,jhd->hij", q[a:a + ln].view(ln, H, D).to(F64).abs(), kb.abs()).amax(2).T * scale.to(F64) * 2.0 ** -20
        bound = torch.einsum("hij,jhd->ihd", w, vb.abs()) * f * (2.0 ** -8 + 2 * ds[..., None]) + want.abs() * 2.0 ** -8 + 1e-6
        err = (o[a:a + ln].view(ln, H, D).to(F64) - want).abs()
        assert (err <= 1.05 * bound).all(), (b, (err / bound).max().item())
    assert out is None or wide[:, :8].abs().max().item() == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("pos,window,chunk", [(0, 1 << 30, 0), (90, 100, 0), (64, 1 << 30, 128)])
def test_values_that_are_not_finite_reach_the_rows_that_see_them_only(pos, window, chunk, bad):
    """A value row that is infinite or NaN, of the step and of the ring: queries in front of it and behind its window, in the same tile of
    the products, are as without it."""
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    torch.manual_seed(pos)
    H, G, D, n, cap, dev = 2, 1, 128, 300, 512, "cuda"
    st = StepLayout([n], [pos], [0], dev)
    q, k, v = (torch.randn(n, x * D, device=dev).to(BF16) for x in (H, G, G))
    kring, vring = (torch.randn(1, cap, G * D, device=dev).to(BF16) for _ in range(2))
    scale = torch.full((H,), 0.1, device=dev)

    def run(v, vring):
        return ops.seq_swa_attn(q, k, v, kring, vring, None, 0, scale, st, H, G, D, D, window, cap, from_ring_only=False, chunk=chunk).view(n, H, D)

    want = run(v, vring)
    v2, vring2 = v.clone(), vring.clone()
    at = [pos + 37, pos + 200] + ([pos - 8] if pos else [])  # positions; channels 5, 40 and 70
    v2[37, 5], v2[200, 40] = bad, -bad
    if pos:
        vring2[0, pos - 8, 70] = bad
    got = run(v2, vring2)
    qp = torch.arange(pos, pos + n, device=dev)
    hit = torch.zeros(n, D, dtype=torch.bool, device=dev)
    for p, c in zip(at, (5, 40, 70)):
        hit[:, c] = (qp >= p) & ((qp // chunk == p // chunk) if chunk else (qp - p < window))
    hit = hit[:, None].expand(n, H, D)
    assert not got[hit].isfinite().any() and got[~hit].isfinite().all()
    if bad == float("inf"):
        assert got[hit].isinf().all()
    # beside them either the products' result or, in tiles that hold one, sums of FMAs: P is rounded to eight bits in the former
    assert ((got[~hit].float() - want[~hit].float()).norm() / want[~hit].float().norm()).item() < 2.0 ** -7
