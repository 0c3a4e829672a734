"""Steps of one token per request: the fused launches against the launches they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(n):
    from llark_b200.state_cache import StepLayout

    return StepLayout([1] * n, [5] * n, [(3 * b + 1) % (2 * n + 3) for b in range(n)] if n % 3 else list(range(n, 0, -1)), torch.device("cuda"))


def _rand(*shape):
    return torch.randn(shape, device="cuda", generator=_rand.g)


_rand.g = None


@pytest.fixture(autouse=True)
def _seed():
    _rand.g = torch.Generator(device="cuda").manual_seed(11)


@pytest.mark.parametrize("n,H,D,low,act", [(1, 1, 64, True, torch.bfloat16), (8, 16, 128, True, torch.bfloat16), (5, 3, 128, False, torch.float32),
                                           (130, 2, 64, False, torch.float32)])
def test_a_gated_recurrence_s_step_is_the_scan_and_the_norm(n, H, D, low, act):
    """The state's numbers are the scan's; the read-out adds the same D products in another order: within D ulp of their absolute sum, which the
    norm scales by |w| / rms (its sum of squares moves by as much, relatively), and an ulp of the result's type."""
    from llark_b200 import ops

    E, st = 128, _step(n)
    src = _rand(n, H * (2 * D + E) + 4)
    lower = torch.rand(H * D, device="cuda", generator=_rand.g) if low else None
    s0, norm = _rand(2 * n + 3, H, D, E), _rand(E)
    sa, sb = s0.clone(), s0.clone()
    at = (src, 0, H * D, 2 * H * D, lower)
    raw = ops.seq_glr_scan(*at, sa, st, H, D, E)
    want = ops.seq_head_rmsnorm(raw, norm, E, 1e-5, torch.float32).double()
    got = ops.seq_glr_step(*at, sb, st, H, D, E, norm, 1e-5, act)
    assert torch.equal(sa, sb) and not torch.equal(sa, s0)
    q = src[:, :H * D].double()
    q = (q * q.sigmoid()).view(n, H, D, 1)
    reach = (q.abs() * sa[st.slot.long()].double().abs()).sum(2)
    rms = raw.double().view(n, H, E).square().mean(-1, keepdim=True).add(1e-5).sqrt()
    moved = 2 * D * 2.0 ** -24 * (reach / rms + reach.square().mean(-1, keepdim=True).sqrt() / rms * (raw.double().view(n, H, E) / rms).abs())
    bound = (moved * norm.double().abs()).view(n, -1) + want.abs() * (2.0 ** -8 if act == torch.bfloat16 else 2.0 ** -22)
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("n,C,taps,act", [(1, 4, 1, torch.float32), (3, 132, 2, torch.bfloat16), (8, 2048, 4, torch.bfloat16), (150, 2052, 6, torch.float32)])
def test_the_norm_and_the_next_convolution_are_those_of_two_launches(n, C, taps, act):
    from llark_b200 import ops

    st = _step(n)
    x, y, w, cw = _rand(n, C), _rand(n, C), _rand(C), _rand(C, taps)
    t0 = _rand(2 * n + 3, max(taps - 1, 1), C)
    ta, tb = t0.clone(), t0.clone()
    xa = ops.seq_add_rmsnorm(x, y, w, 1e-5)
    ha = ops.seq_short_conv(xa, cw, ta, st, act)
    xb, hb = ops.seq_add_rmsnorm_conv(x, y, w, 1e-5, cw, tb, st, act)
    assert torch.equal(xa, xb) and torch.equal(ha, hb) and torch.equal(ta, tb) and (taps == 1 or not torch.equal(t0, tb))


@pytest.mark.parametrize("stores", [1, 3, 16, 17])
def test_a_new_request_s_slot_is_zero_in_every_store_and_no_other_is_touched(stores):
    from llark_b200.state_cache import StateCache

    c = StateCache("cuda", n_slots=5)
    shapes = [(3 + 2 * i, 5) for i in range(stores)]
    zeroed = [c.add_store(s, torch.float32, zero_on_alloc=True) for s in shapes for _ in range(2)]
    half, kept = c.add_store((7,), torch.bfloat16, zero_on_alloc=stores == 3), c.add_store((64,), torch.bfloat16, zero_on_alloc=False)
    first = c.alloc()
    for h in zeroed + [half, kept]:
        c.view(h).fill_(1.5)
    second = c.alloc()
    for h in zeroed + ([half] if stores == 3 else []):
        v = c.view(h)
        assert (v[second] == 0).all() and v.float().sum().item() == 1.5 * (v.numel() - v[second].numel())
    assert (c.view(kept) == 1.5).all() and first != second
