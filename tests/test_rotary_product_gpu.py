"""q, k and v of a window layer's prompts from one product, against the product in fp32 and the rotation of its rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _near(got, pin, want, reach):
    """The sums are the same chains of products (tiles and operands are); the rotation rounds each of its two products and their sum, and the
    angles' cosines and sines are the same numbers: 2 ulp of fp32 of the pair's absolute sum, then one rounding to bf16 on either side."""
    bound = 3 * 2.0 ** -24 * reach + 2.0 ** -8 * want.float().abs() + 2.0 ** -24
    assert ((got.float() - want.float()).abs() <= bound).all()


# (rows of the requests, H, G, D, E, n_rot, K, bias): tiles cut by rows, by q | k | v inside a tile, heads of 32, 64, 96 and 128, nothing turned
@pytest.mark.parametrize("lens,H,G,D,E,n_rot,K,bias", [([65], 2, 1, 64, 64, 64, 64, False), ([1, 80, 3], 4, 2, 128, 128, 128, 256, True),
                                                       ([257, 300], 6, 2, 32, 96, 32, 136, False), ([130], 5, 1, 128, 64, 64, 512, True),
                                                       ([511, 2], 4, 2, 96, 64, 32, 72, False), ([700, 1, 900], 8, 8, 128, 128, 0, 1024, False)])
def test_a_product_that_turns_its_pairs(lens, H, G, D, E, n_rot, K, bias):
    from llark_b200 import ops
    from llark_b200.mixers import rotary_frequencies
    from llark_b200.state_cache import StepLayout

    g = torch.Generator(device="cuda").manual_seed(n_rot + K)
    r = lambda *s: torch.randn(s, device="cuda", generator=g)  # noqa: E731
    N, n = (H + G) * D + G * E, sum(lens)
    a, w, b = r(n, K).to(BF), (r(N, K) * K ** -0.5).to(BF), r(N) if bias else None
    st = StepLayout(lens, [7 * i for i in range(len(lens))], list(range(len(lens))), torch.device("cuda"))
    freq = rotary_frequencies(n_rot, 10000.0)[0].to(device="cuda", dtype=torch.float32) if n_rot else None
    assert ops.linear_qkv_rotary_takes(a, w, H, G, D, E, n_rot)
    pin = ops.linear(a, w, bias=b, out_dtype=torch.float32)
    want = ops.seq_qkv_rotary(pin, 0, H * D, (H + G) * D, H, G, D, E, 1e-5, BF, st, qk_freq=freq, qk_interleaved=True)
    got = ops.linear_qkv_rotary(a, w, st, H, G, D, E, bias=b, freq=freq)
    pair = pin.view(n, -1, 2).abs().sum(2, keepdim=True).expand(-1, -1, 2).reshape(n, N)
    for x, y, p in zip(got, want, pair.split([H * D, G * D, G * E], 1)):
        assert x.shape == y.shape
        _near(x, pin, y, p)
    assert torch.equal(got[2], want[2])


def test_what_it_does_not_take():
    from llark_b200 import ops

    a, w = torch.zeros(100, 64, device="cuda", dtype=BF), torch.zeros(256, 64, device="cuda", dtype=BF)
    takes = ops.linear_qkv_rotary_takes
    assert takes(a, w, 2, 1, 64, 64, 64) and not takes(a[:64], w, 2, 1, 64, 64, 64) and not takes(a.float(), w.float(), 2, 1, 64, 64, 64)
    assert not takes(a, w, 2, 1, 64, 64, 24) and not takes(a, w[:248], 2, 1, 64, 56, 64) and not takes(a, w, 1, 1, 96, 64, 32)
    assert not takes(torch.zeros(6404, device="cuda", dtype=BF)[4:].view(100, 64), w, 2, 1, 64, 64, 64)
    two = ops.lib().llark_gemm_get_mode()
    ops.lib().llark_gemm_set_mode(0)
    try:
        assert not takes(a, w, 2, 1, 64, 64, 64)
    finally:
        ops.lib().llark_gemm_set_mode(two)


def test_a_stream_makes_its_own_table_of_angles():
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    st, freq = StepLayout([3, 70], [0, 5], [0, 1], torch.device("cuda")), torch.rand(32, device="cuda")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        there = ops.seq_rotary_table(freq, st)
    here = ops.seq_rotary_table(freq, st)
    torch.cuda.synchronize()
    assert here is not there and here is ops.seq_rotary_table(freq, st) and torch.equal(here, there)


def test_a_stream_makes_its_own_lists_of_a_step():
    """The lists of the block walk and of the scans' chunks, as the tables above: a stream does not read what another one may still be writing."""
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    st = StepLayout([3, 170], [0, 5], [0, 1], torch.device("cuda"))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for make in (lambda: ops._scan_tables(st, 8), lambda: st.chunks(64)):
        with torch.cuda.stream(side):
            there = make()
        here = make()
        torch.cuda.synchronize()
        assert here is not there and here is make()
        values = lambda c: [t for t, _, _ in c] if isinstance(c, list) else [c.row0, c.n, c.index, c.minus1, c.last_slot, c.inner, c.seq_item0]  # noqa: E731
        assert all(torch.equal(a, b) for a, b in zip(values(here), values(there), strict=True))


def test_tables_of_a_step_are_those_of_their_frequencies():
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    st, freq = StepLayout([3, 70], [0, 5], [0, 1], torch.device("cuda")), torch.rand(32, device="cuda")
    wide, narrow = ops.seq_rotary_table(freq, st), ops.seq_rotary_table(freq[:16], st)  # the same address
    assert narrow.shape == (73, 16, 2) and torch.equal(narrow, wide[:, :16])


def test_what_a_capture_writes_is_not_kept_for_later_calls():
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    n, H, D, E = 73, 2, 64, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    src = torch.randn(n, H * (2 * D + E), device="cuda", generator=g)
    freq, powers = torch.rand(32, device="cuda", generator=g), ops.decay_powers([0.9, 0.99], torch.device("cuda"))

    def scan(st):
        return ops.seq_decay_scan(src, 0, H * D, 2 * H * D, powers, torch.zeros(2, H, D, E, device="cuda"), st, H, D, E, freq=freq)

    layout = lambda: StepLayout([3, 70], [0, 5], [0, 1], torch.device("cuda"))  # noqa: E731
    want, st = scan(layout()), layout()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        got = scan(st)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # the stream of the capture, which has not been replayed
        assert torch.equal(scan(st), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
