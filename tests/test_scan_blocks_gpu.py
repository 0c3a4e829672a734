"""The block walk of matrix recurrences (csrc/seq_chunk.cu) against 64 bits and against the token-by-token kernels: requests of one token,
around a block of 16, several passes of its workspace, decays from nothing left to nothing lost, states that were there before, both
head sizes and all three sources."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
F32, F64 = torch.float32, torch.float64


@pytest.fixture(autouse=True)
def walk(monkeypatch):
    """The walk at the sizes where it can go wrong, whether or not it is the faster one there."""
    from llark_b200 import ops

    monkeypatch.setattr(ops, "walk_pays", lambda *a: True)


def _layout(lens, slots, dev="cuda"):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ints = lambda v: torch.tensor(v, device=dev, dtype=torch.int32)  # noqa: E731
    return types.SimpleNamespace(n_tok=cu[-1], n_seq=len(lens), max_len=max(lens), cu=ints(cu), slot=ints(slots), lens_dev=ints(lens),
                                 device=dev, cu_host=cu)


def _walk(q, d, z, p, v, S, correct):
    """One request in 64 bits: vectors [T, H, D], values [T, H, E], state [H, D, E]."""
    out = []
    for t in range(q.shape[0]):
        u = v[t] - (torch.einsum("hde,hd->he", S, z[t]) if correct else 0)
        S = d[t][..., None] * S + p[t][..., None] * u[:, None]
        out.append(torch.einsum("hde,hd->he", S, q[t]))
    return torch.stack(out), S


@pytest.mark.parametrize("kind", ["hgrn2", "scalar", "channel", "state"])
@pytest.mark.parametrize("lens,H,D,E,bytes_", [([16], 1, 128, 128, None), ([1, 17, 40], 5, 128, 64, None), ([33, 15, 2], 3, 64, 96, None),
                                               ([200, 70], 2, 128, 128, 1)])
def test_against_64_bits(kind, lens, H, D, E, bytes_, monkeypatch):
    from llark_b200 import ops

    if bytes_:
        monkeypatch.setattr(ops, "SCAN_BLOCK_BYTES", bytes_)  # a workspace of one block per request: a pass per 16 tokens
    torch.manual_seed(sum(lens) + H + D)
    dev, n = "cuda", sum(lens)
    slots = torch.randperm(len(lens) + 1)[:len(lens)].tolist()
    st = _layout(lens, slots)
    S0 = torch.randn(len(lens) + 1, H, D, E, device=dev)
    state = S0.clone()
    # decays of every kind: channels that keep next to nothing, that keep nearly everything, and anything between
    x = torch.randn(n, H, D, device=dev) * 3 + torch.linspace(-12, 8, D, device=dev)
    if kind == "hgrn2":
        ld = 2 * H * D + H * E
        src = torch.randn(n, ld, device=dev)
        src[:, H * D:2 * H * D] = x.reshape(n, -1)
        lower = torch.rand(H * D, device=dev) * (torch.rand(H * D, device=dev) > 0.3)
        o = ops.seq_glr_scan(src, 0, H * D, 2 * H * D, lower, state, st, H, D, E)
        s = src.to(F64)
        q = torch.nn.functional.silu(s[:, :H * D]).view(n, H, D)
        lo = lower.to(F64)
        d = (lo + (1 - lo) * torch.sigmoid(s[:, H * D:2 * H * D])).view(n, H, D)
        z, p, v = None, 1 - d, s[:, 2 * H * D:].reshape(n, H, E)
    else:
        rule = {"scalar": ops.DELTA_GATED_SCALAR, "channel": ops.DELTA_GATED, "state": ops.DELTA_STATE_SPACE}[kind]
        G = 1 if H % 2 else H // 2  # heads share keys
        wide = torch.randn(n, 2 * G * D + H * E + 4, device=dev)  # column slices, as the mixers hand them over
        q, k, v = wide[:, :G * D], wide[:, G * D:2 * G * D] + 0.3, wide[:, 2 * G * D + 4:]
        dec = x.reshape(n, -1) if kind == "channel" else x[:, :, 5].contiguous()
        mix, rate_log, bias = torch.randn(n, H, device=dev), torch.randn(H, device=dev), torch.randn(dec.shape[1], device=dev)
        args = (rule, q, k, v, dec, None if kind == "state" else mix)
        o = ops.seq_delta_rule(*args, state, st, H, G, D, E, dec_bias=bias, rate_log=rate_log)
        monkeypatch.setattr(ops, "SCAN_BLOCK_MIN_LEN", 1 << 30)
        old_state = S0.clone()
        old = ops.seq_delta_rule(*args, old_state, st, H, G, D, E, dec_bias=bias, rate_log=rate_log)
        q, k = (t.to(F64).reshape(n, G, D).repeat_interleave(H // G, 1) for t in (q, k))
        v = v.to(F64).reshape(n, H, E)
        step = torch.nn.functional.softplus(dec.to(F64) + bias.to(F64))
        step = step.view(n, H, D) if kind == "channel" else step[:, :, None]
        d = torch.exp(-torch.exp(rate_log.to(F64))[:, None] * step).expand(n, H, D)
        if kind == "state":
            z, p = None, step * k
        else:
            unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            q, k = unit(q) / D ** 0.5, unit(k)
            z, p = k * d, torch.sigmoid(mix.to(F64))[:, :, None] * k
    for b, ln in enumerate(lens):
        at = slice(st.cu_host[b], st.cu_host[b] + ln)
        want, S = _walk(q[at], d[at], z[at] if z is not None else None, p[at], v[at], S0[slots[b]].to(F64), kind in ("scalar", "channel"))
        rel = lambda a, w: ((a.to(F64) - w).norm() / w.norm()).item()  # noqa: E731
        eo, es = rel(o.view(n, H, E)[at], want), rel(state[slots[b]], S)
        # 2^-21 of a product from the split, sums of up to 128 + 16 of them: 2e-6 of the terms' norm at most
        assert eo < 2e-6 and es < 2e-6, (b, eo, es)
        if kind != "hgrn2":
            assert eo < max(2 * rel(old.view(n, H, E)[at], want), 1e-6) and es < max(2 * rel(old_state[slots[b]], S), 1e-6)
    rest = [s for s in range(len(lens) + 1) if s not in slots]
    assert torch.equal(state[rest], S0[rest])  # nobody else's state was touched


@pytest.mark.parametrize("kind", ["hgrn2", "scalar", "channel", "state"])
@pytest.mark.parametrize("lens,H", [([300, 100], 4), ([70, 33], 40), ([70, 33], 80)])  # up to two CTAs per SM, more, 64 columns per CTA
def test_as_exact_as_fp32_sums(kind, lens, H):
    """Decays, keys and values as a layer's projections give them: the split operands are rounded and the chains in the truncating adders
    are two products long. Measured 1.2 to 1.6e-7 of the outputs, the token-by-token FMAs 0.7 to 1.4e-7, operands that
    are cut 4.5e-7: 2^-22."""
    from llark_b200 import ops

    torch.manual_seed(11)
    D, E, dev = 128, 128, "cuda"
    n, st = sum(lens), _layout(lens, [0, 1])
    state = torch.zeros(2, H, D, E, device=dev)
    q, k, v = (torch.nn.functional.silu(torch.randn(n, H * D, device=dev)) for _ in range(3))
    z = None
    if kind == "hgrn2":
        src, lower = torch.randn(n, 3 * H * D, device=dev), torch.rand(H * D, device=dev) * 0.9
        src[:, H * D:2 * H * D] += 1.0
        o = ops.seq_glr_scan(src, 0, H * D, 2 * H * D, lower, state, st, H, D, E)
        s, lo = src.to(F64), lower.to(F64)
        q = torch.nn.functional.silu(s[:, :H * D]).view(n, H, D)
        d = (lo + (1 - lo) * torch.sigmoid(s[:, H * D:2 * H * D])).view(n, H, D)
        p, v = 1 - d, s[:, 2 * H * D:].reshape(n, H, E)
    else:
        rule = {"scalar": ops.DELTA_GATED_SCALAR, "channel": ops.DELTA_GATED, "state": ops.DELTA_STATE_SPACE}[kind]
        if kind == "state":
            q, k = q / 11, k / 11
        dec, mix = torch.randn(n, H * D if kind == "channel" else H, device=dev), torch.randn(n, H, device=dev)
        rate, bias = torch.randn(H, device=dev) * 0.5 - 1, torch.randn(dec.shape[1], device=dev) - 1
        o = ops.seq_delta_rule(rule, q, k, v, dec, None if kind == "state" else mix, state, st, H, H, D, E, dec_bias=bias, rate_log=rate)
        q, k, v = (t.to(F64).view(n, H, D) for t in (q, k, v))
        step = torch.nn.functional.softplus(dec.to(F64) + bias.to(F64))
        step = step.view(n, H, D) if kind == "channel" else step[:, :, None]
        d = torch.exp(-torch.exp(rate.to(F64))[:, None] * step).expand(n, H, D)
        if kind == "state":
            p = step * k
        else:
            q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, z, p = q / D ** 0.5, k * d, torch.sigmoid(mix.to(F64))[:, :, None] * k
    for b, ln in enumerate(lens):
        at = slice(st.cu_host[b], st.cu_host[b] + ln)
        want, _ = _walk(q[at], d[at], z[at] if z is not None else None, p[at], v[at], torch.zeros(H, D, E, device=dev, dtype=F64), z is not None)
        assert ((o.view(n, H, E)[at].to(F64) - want).norm() / want.norm()).item() < 2.0 ** -22


@pytest.mark.parametrize("kind", ["hgrn2", "scalar", "channel", "state"])
@pytest.mark.parametrize("what,value", [("v", float("nan")), ("v", float("inf")), ("k", float("nan")), ("q", -float("inf")),
                                        ("d", float("nan")), ("state", float("inf"))])
def test_numbers_that_are_not_finite_stay_behind_their_token(kind, what, value, monkeypatch):
    """An infinity or a NaN in one token of a block: nothing changes in front of it, and behind it results are those of the token-by-token
    kernels, infinite or NaN where they are."""
    from llark_b200 import ops

    torch.manual_seed(7)
    lens, H, D, E, dev = [40, 21], 2, 64, 32, "cuda"
    n, st = sum(lens), _layout(lens, [1, 0])
    S0 = torch.randn(2, H, D, E, device=dev)
    t, h = 27, 1  # token 11 of the first request's second block
    if what == "state":
        S0[1, h, 3, 9] = value
    if kind == "hgrn2":
        src = torch.randn(n, 2 * H * D + H * E, device=dev)
        at = {"v": 2 * H * D + h * E + 9, "k": None, "q": h * D + 3, "d": H * D + h * D + 3, "state": None}[what]
        if what == "k":
            pytest.skip("HGRN2 has no keys of its own")
        if at is not None:
            src[t, at] = value
        run = lambda s: ops.seq_glr_scan(src, 0, H * D, 2 * H * D, None, s, st, H, D, E)  # noqa: E731
    else:
        rule = {"scalar": ops.DELTA_GATED_SCALAR, "channel": ops.DELTA_GATED, "state": ops.DELTA_STATE_SPACE}[kind]
        q, k, v = (torch.randn(n, H * x, device=dev) for x in (D, D, E))
        dec, mix = torch.randn(n, H * D if kind == "channel" else H, device=dev), torch.randn(n, H, device=dev)
        bias, rate = torch.zeros(dec.shape[1], device=dev), torch.zeros(H, device=dev)
        if what != "state":
            {"v": v, "k": k, "q": q, "d": dec}[what][t, {"v": h * E + 9, "d": h * D + 3 if kind == "channel" else h}.get(what, h * D + 3)] = value
        run = lambda s: ops.seq_delta_rule(rule, q, k, v, dec, None if kind == "state" else mix, s, st, H, H, D, E, dec_bias=bias,  # noqa: E731
                                           rate_log=rate)
    s1, s2 = S0.clone(), S0.clone()
    o1 = run(s1)
    monkeypatch.setattr(ops, "SCAN_BLOCK_MIN_LEN", 1 << 30)
    o2 = run(s2)
    for a, b in ((o1, o2), (s1, s2)):
        assert not b.isfinite().all() or what == "q"
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        assert torch.equal(a[a.isinf()], b[b.isinf()])
        ok = b.isfinite()
        assert ((a[ok] - b[ok]).norm() / b[ok].norm()).item() < 2e-6  # as above


@pytest.mark.parametrize("lens,most", [([40], 9), ([1, 17, 300, 2], 8), ([1] * 1500 + [500] + [30] * 700, 2400)])
def test_the_plan_of_a_pass(lens, most):
    """The device's lists against the step: more requests than one sweep of the kernel takes, requests that end in an earlier pass."""
    from llark_b200 import ops

    st = _layout(lens, list(range(len(lens))))
    blocks = [-(-n // 16) for n in lens]
    for (done, each, n, m), (lists, n_, m_) in zip(ops.scan_passes(st.cu_host, most), ops._scan_tables(st, most)):
        requests, table = lists[:4 * n].view(n, 4), lists[4 * n:].view(m, 2)
        assert (n_, m_) == (n, m)
        want_r, want_b = [], []
        for b, x in enumerate(blocks):
            k = min(max(x - done, 0), each)
            if k:
                want_r.append([b, len(want_b), k, done])
                want_b += [[b, done + i] for i in range(k)]
        assert requests.tolist() == want_r and table.tolist() == want_b and (n, m) == (len(want_r), len(want_b))


@pytest.mark.parametrize("kind", ["hgrn2", "scalar", "channel", "state"])
def test_full_fp32_is_the_token_by_token_scan(kind, monkeypatch):
    from llark_b200 import ops

    torch.manual_seed(3)
    lens, H, D, E, dev = [40, 3], 2, 64, 32, "cuda"
    n, st = sum(lens), _layout(lens, [0, 1])
    S0, x = torch.randn(2, H, D, E, device=dev), torch.randn(n, 3 * H * D + 2 * H, device=dev)
    one = torch.ones(H * D, device=dev)

    def run(**kw):
        s = S0.clone()
        if kind == "hgrn2":
            return ops.seq_glr_scan(x, 0, H * D, 2 * H * D, None, s, st, H, D, E, **kw), s
        rule = {"scalar": ops.DELTA_GATED_SCALAR, "channel": ops.DELTA_GATED, "state": ops.DELTA_STATE_SPACE}[kind]
        wide = kind == "channel"
        dec, bias = (x[:, H * D:2 * H * D].contiguous(), one) if wide else (x[:, -H:], one[:H])
        return ops.seq_delta_rule(rule, x[:, :H * D].contiguous(), x[:, H * D:2 * H * D].contiguous(), x[:, 2 * H * D:2 * H * D + H * E].contiguous(),
                                  dec, None if kind == "state" else x[:, -2 * H:-H], s, st, H, H, D, E, dec_bias=bias, rate_log=one[:H], **kw), s

    got = run(full_fp32=True)
    walk = run()
    monkeypatch.setattr(ops, "SCAN_BLOCK_MIN_LEN", 1 << 30)
    want = run()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert not torch.equal(walk[0], want[0])  # the other form, at fp32 accuracy


def test_a_capture_writes_its_own_lists():
    """A step that a stream capture meets first, replayed, and the same step launched directly afterwards: the lists of the capture exist
    in its replays only and must not be kept with the step."""
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    torch.manual_seed(5)
    H, D, E, lens = 2, 64, 32, [50, 20]
    src, S0 = torch.randn(sum(lens), 3 * H * D, device="cuda"), torch.randn(2, H, D, E, device="cuda")
    run = lambda st, s: ops.seq_glr_scan(src, 0, H * D, 2 * H * D, None, s, st, H, D, E)  # noqa: E731
    want_s = S0.clone()
    want = run(StepLayout(lens, [0, 0], [0, 1], "cuda"), want_s)
    st, state = StepLayout(lens, [0, 0], [0, 1], "cuda"), S0.clone()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got = run(st, state)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(state, want_s)
    again = S0.clone()
    assert torch.equal(run(st, again), want) and torch.equal(again, want_s)
    del graph


@pytest.mark.parametrize("kind", ["hgrn2", "scalar", "state"])
def test_a_request_that_is_nan_from_a_token_on(kind, monkeypatch):
    """Every projection NaN from a token in the middle of a block on, over several blocks and passes: NaN from there, nothing before, and the
    other request as alone."""
    from llark_b200 import ops

    torch.manual_seed(2)
    lens, H, D, E, dev, bad = [150, 60], 2, 64, 32, "cuda", 37
    n, st = sum(lens), _layout(lens, [1, 0])
    src, mix, one = torch.randn(n, 3 * H * D, device=dev), torch.randn(n, H, device=dev), torch.ones(H, device=dev)
    S0 = torch.randn(2, H, D, E, device=dev)
    monkeypatch.setattr(ops, "SCAN_BLOCK_BYTES", 6 * H * ops.lib().llark_seq_chunk_block_bytes(D, 1))

    def run():
        s = S0.clone()
        if kind == "hgrn2":
            return ops.seq_glr_scan(src, 0, H * D, 2 * H * D, None, s, st, H, D, E), s
        rule = ops.DELTA_GATED_SCALAR if kind == "scalar" else ops.DELTA_STATE_SPACE
        return ops.seq_delta_rule(rule, src[:, :H * D], src[:, H * D:2 * H * D], src[:, 2 * H * D:], mix, None if kind == "state" else mix, s, st,
                                  H, H, D, E, dec_bias=one, rate_log=one), s

    want_o, want_s = run()
    assert want_o.isfinite().all() and want_s.isfinite().all()
    src[bad:lens[0]], mix[bad:lens[0]] = float("nan"), float("nan")
    got_o, got_s = run()
    assert got_o[bad:lens[0]].isnan().all() and got_s[1].isnan().all()
    keep = torch.ones(n, dtype=torch.bool, device=dev)
    keep[bad:lens[0]] = False
    assert torch.equal(got_s[0], want_s[0]) and torch.equal(got_o[lens[0]:], want_o[lens[0]:])
    # the block of the first bad token is summed by FMAs, everything in front of it by the same products
    assert torch.equal(got_o[:bad // 16 * 16], want_o[:bad // 16 * 16])
    assert ((got_o[keep] - want_o[keep]).norm() / want_o[keep].norm()).item() < 2e-6
