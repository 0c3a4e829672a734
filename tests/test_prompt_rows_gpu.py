"""Row-wise kernels of prompts that request several rows at once: against plain formulas in 64 bits, at ragged counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ULP = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8}


def _near(got, want, scale):
    """A dozen fp32 roundings of terms whose absolute sum is `scale`, and the result's own."""
    assert ((got.double() - want).abs() <= 16 * 2.0 ** -24 * scale + ULP[got.dtype] * want.abs() + 1e-30).all()


def _rand(seed, *shape):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


# (tokens, heads, entries): below the limit, at it, a count that ends inside a warp's four heads; heads that leave lanes idle
@pytest.mark.parametrize("n,H,E", [(591, 16, 128), (592, 16, 128), (3159, 3, 128), (9473, 1, 128), (1201, 8, 96), (9475, 1, 4)])
@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
def test_head_norms(n, H, E, act):
    from llark_b200 import ops

    x, w, wide = _rand(1, n, H * E), _rand(2, H * E), _rand(3, n, H * E + 8)
    xd = x.double().view(n, H, E)
    unit = xd / (xd.square().mean(-1, keepdim=True) + 1e-5).sqrt()
    if E == 128:
        want = (unit * w[:E].double()).view(n, -1)
        _near(ops.seq_head_rmsnorm(x, w[:E].contiguous(), E, 1e-5, act), want, want.abs())
    gate = wide[:, 4:4 + H * E]
    g = gate.double()
    for per_head, silu in ((False, True), (True, False)):
        ww = (w if per_head else w[:E]).contiguous()
        want = (unit * (ww.double().view(H, E) if per_head else ww.double())).view(n, -1) * torch.sigmoid(g) * (g if silu else 1)
        _near(ops.seq_head_norm_gate(x, ww, H, E, 1e-5, act, gate=gate, gate_silu=silu, w_per_head=per_head), want, want.abs())
    want = unit.view(n, -1)
    _near(ops.seq_head_norm_gate(x, None, H, E, 1e-5, act), want, want.abs())


# requests that start and end inside a run of 8 or 16 rows, at its first and last row, and ones shorter than the taps
@pytest.mark.parametrize("lens", [[64], [65], [1, 2, 3, 58, 16, 8, 200], [16, 16, 15, 17, 300], [3, 61, 128]])
@pytest.mark.parametrize("taps,C", [(2, 4), (3, 132), (4, 260), (4, 512)])
def test_convolutions(lens, taps, C):
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    n, k = sum(lens), taps - 1
    st = StepLayout(lens, [0] * len(lens), list(range(len(lens)))[::-1], torch.device("cuda"))
    wide, w = _rand(4, n, C + 4), _rand(5, C * taps + 1)[1 if C == 260 else 0:][:C * taps].view(C, taps)
    old = _rand(6, len(lens), k, C)
    x = wide[:, :C]
    rows = []
    for b, (lo, hi) in enumerate(zip(st.cu_host, st.cu_host[1:])):
        padded = torch.cat([old[st.slots_host[b]], x[lo:hi]]).double()
        rows.append(torch.stack([padded[j:j + hi - lo] * w[:, j].double() for j in range(taps)]))
    terms = torch.cat(rows, 1)
    y, reach = terms.sum(0), terms.abs().sum(0)
    carry = old.clone()
    got = ops.seq_conv_act(x, w, carry, st, silu=False)
    _near(got, y, reach)
    _near(ops.seq_conv_act(x, w, old.clone(), st, silu=True), y * torch.sigmoid(y), 2 * reach)
    tail = old.clone()
    _near(ops.seq_short_conv(x.contiguous(), w, tail, st, torch.float32), y + x.double(), reach + x.double().abs())
    assert torch.equal(carry, tail)
