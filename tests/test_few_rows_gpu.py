"""Products with few rows (csrc/skinny.cu) at the edges of their tiles: tokens 1 / 8 | 9 / 16 | 17 / 32 | 33 / 64 (the kernels' groups),
weight rows that fill no tile, K of one slice, of a ragged last slice and of a cluster of eight, every epilogue, and the routed form
with empty and full experts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def _rel(a, b):
    return ((a.to(F64) - b).norm() / b.norm()).item()


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(64, 64), (72, 136), (1000, 2048), (4096, 4096), (333, 8)])
def test_products_and_epilogues(M, N, K):
    from llark_b200 import ops

    torch.manual_seed(M + N + K)
    x, w = (torch.randn(M, K, device="cuda") * 0.5).to(BF16), (torch.randn(N, K, device="cuda") * 0.5).to(BF16)
    b = torch.randn(N, device="cuda")
    z = x.to(F64) @ w.to(F64).t()
    # fp32 results: products of bf16 numbers are exact, so only the order and the cut of K fp32 additions shows: at most
    # K * 2^-24 relative to the terms' norm, sqrt(K) of it in practice; the tensor cores' truncating adders measure 2e-6
    taken = ops.LINEAR_STATS["rows"]
    assert _rel(ops.linear(x, w, bias=b, out_dtype=F32), z + b.to(F64)) < (5e-7 if M <= 8 else 5e-6)
    # bf16 results: one rounding to eight bits, at most 2^-8 of a value
    assert _rel(ops.linear(x, w, act="relu2"), torch.relu(z) ** 2) < 2.0 ** -8
    assert ops.LINEAR_STATS["rows"] == taken + 2
    if N % 2 == 0:
        v = z + b.to(F64)
        assert _rel(ops.linear(x, w, bias=b, act="relu_glu"), torch.relu(v[:, 0::2]) * v[:, 1::2]) < 2.0 ** -8
        g, u = z[:, 0::2].clamp(max=7.0), z[:, 1::2].clamp(-7.0, 7.0)
        assert _rel(ops.linear(x, w, act="clamp_glu", act_limit=7.0), g * torch.sigmoid(1.702 * g) * (u + 1)) < 2.0 ** -8
    if N % 8 == 0:
        r = torch.randn(M, N, device="cuda").to(BF16)
        assert _rel(ops.gemm(x, w, residual=r, bias=b.to(BF16)), z + r.to(F64) + b.to(BF16).to(F64)) < 2.0 ** -8


@pytest.mark.parametrize("M", [1, 5, 16, 33, 64])
def test_rotation_in_the_epilogue_is_that_of_the_op(M):
    from llark_b200 import ops

    torch.manual_seed(M)
    H, K = 512, 1024
    x, w = (torch.randn(M, K, device="cuda") * 0.5).to(BF16), (torch.randn(3 * H, K, device="cuda") * 0.1).to(BF16)
    cos, sin = torch.randn(16, 128, device="cuda").to(BF16), torch.randn(16, 128, device="cuda").to(BF16)
    for S in (1, 7):
        want = ops.gemm(x, w)
        ops.rope_(want, cos, sin, S, H // 128, 128)  # rotates the q and the k heads of the packed projection
        assert torch.equal(ops.gemm(x, w, rope=(cos, sin, S, 2 * H)), want)


@pytest.mark.parametrize("T,C,ff,E,top,kind", [(1, 64, 64, 4, 2, "silu"), (9, 136, 72, 8, 3, "silu"), (70, 256, 128, 2, 1, "clamp"),
                                                (33, 128, 200, 16, 4, "relu2"), (300, 512, 256, 8, 4, "silu")])
def test_routed_experts(T, C, ff, E, top, kind):
    from llark_b200 import ops

    torch.manual_seed(T + C)
    up = ff if kind == "relu2" else 2 * ff
    wu, wd = torch.randn(E, up, C, device="cuda").mul(C ** -0.5).to(BF16), torch.randn(E, C, ff, device="cuda").mul(ff ** -0.5).to(BF16)
    x = torch.randn(T, C, device="cuda").to(BF16)
    hot = max(top, E // 2)  # the other experts get nothing
    ids = torch.stack([torch.randperm(hot, device="cuda")[:top] for _ in range(T)]).to(torch.int32)
    wts = torch.rand(T, top, device="cuda") if kind == "clamp" else None
    z, pos = ops.seq_moe_experts(x, ids, wu, wd, gated=kind != "relu2", in_wts=wts, limit=7.0 if kind == "clamp" else None)
    got = z[pos.long()].view(T, top, C)
    want = torch.empty(T, top, C, device="cuda", dtype=F64)
    for t in range(T):
        for k in range(top):
            e = int(ids[t, k])
            u = wu[e].to(F64) @ x[t].to(F64)
            if kind == "clamp":
                u = u * wts[t, k].to(F64)
                g, v = u[0::2].clamp(max=7.0), u[1::2].clamp(-7.0, 7.0)
                h = g * torch.sigmoid(ops.GLU_SLOPE * g) * (v + 1)
            elif kind == "silu":
                h = torch.nn.functional.silu(u[:ff]) * u[ff:]
            else:
                h = torch.relu(u) ** 2
            want[t, k] = wd[e].to(F64) @ h
    assert _rel(got, want) < 2.0 ** -8  # the units are rounded to eight bits between the two products


@pytest.mark.parametrize("M,N,K", [(1, 704, 256), (8, 1024, 512), (9, 208, 72), (40, 2816, 1024)])
def test_gate_and_up_in_the_epilogue_are_those_of_the_op(M, N, K):
    from llark_b200 import ops

    torch.manual_seed(M + N)
    x, w = (torch.randn(M, K, device="cuda") * 0.5).to(BF16), (torch.randn(N, K, device="cuda") * 0.2).to(BF16)
    got = ops.gemm(x, w, swiglu=True)
    # the halves' tiles cut K as the plain product's do, up to how many CTAs share a row: the sums may differ in their last bits
    assert _rel(got, ops.swiglu_fwd(ops.gemm(x, w)).to(F64)) < 2.0 ** -8


@pytest.mark.parametrize("M", [9, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(40, 4096), (56, 72), (24, 11008)])
def test_narrow_products_and_paired_fp32_results_are_as_exact_as_fmas(M, N, K):
    """Rows above eight: chains of one slice of K in the tensor cores' truncating adders, everything else in fp32. An fp32 FMA chain of
    these lengths measures 4e-7 to 1.1e-6, short chains 1 to 1.3e-7, one chain over K 2e-7 to 1.4e-6: 2^-22."""
    from llark_b200 import ops

    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device="cuda").to(BF16), torch.randn(N, K, device="cuda").to(BF16)
    z = x.to(F64) @ w.to(F64).t()
    assert _rel(ops.linear(x, w, out_dtype=F32), z) < 2.0 ** -22
    wide = torch.randn(8 * N, K, device="cuda").to(BF16)
    u = x.to(F64) @ wide.to(F64).t()
    assert _rel(ops.linear(x, wide, act="relu_glu", out_dtype=F32), torch.relu(u[:, 0::2]) * u[:, 1::2]) < 2.0 ** -21  # a product of two


@pytest.mark.parametrize("T,C,ff,E,top", [(1, 128, 1024, 32, 4), (32, 256, 2048, 8, 4), (100, 72, 4096, 8, 4), (500, 64, 8192, 4, 2)])
def test_the_experts_second_product_is_as_exact_as_fmas(T, C, ff, E, top):
    """llark_seq_moe_down alone, whose sums are handed on in fp32: FMAs measured 0.7e-7 to 1e-6, short chains 1 to 2.2e-7, one chain over K
    1 to 9e-6: 2^-21."""
    from llark_b200 import ops
    from llark_b200._lib import lib

    torch.manual_seed(T)
    n, L, p = T * top, lib(), ops._p
    ids = torch.stack([torch.randperm(E, device="cuda")[:top] for _ in range(T)]).to(torch.int32)
    most = (n + L.llark_seq_moe_tile_rows() - 1) // L.llark_seq_moe_tile_rows() + E
    perm, pos, tiles, meta, seg = (torch.zeros(k, device="cuda", dtype=torch.int32) for k in (n, n, 3 * most, 2, E + 1))
    assert L.llark_seq_moe_sort(p(ids), n, E, E, p(perm), p(pos), p(tiles), p(meta), p(seg), None, ops._stream()) == 0
    act, wd = torch.randn(n, ff, device="cuda").to(BF16), torch.randn(E, C, ff, device="cuda").to(BF16)
    z = torch.empty(n, C, device="cuda")
    assert L.llark_seq_moe_down(p(act), p(wd), p(z), p(tiles), p(meta), most, n, C, ff, 0, ops._stream()) == 0
    want, e = torch.empty(n, C, device="cuda", dtype=F64), ids.view(-1).long()
    for k in range(E):
        at = pos.long()[(e == k).nonzero().view(-1)]
        want[at] = act[at].to(F64) @ wd[k].to(F64).t()
    assert _rel(z, want) < 2.0 ** -21


@pytest.mark.parametrize("M", [1, 8, 9, 33, 64])
def test_products_that_begin_early_see_what_was_written_before(M):
    """Kernels launched behind each other without a wait: tokens, residuals and weights written by the launch in front, buffers written
    again while the launch in front may still read them; eagerly and as a captured graph, against the same launches one at a time."""
    from llark_b200 import ops

    torch.manual_seed(M)
    K = 1024
    ws = [(torch.randn(K, K, device="cuda") * K ** -0.5).to(BF16) for _ in range(4)]
    gamma = torch.ones(K, device="cuda", dtype=BF16)
    w, x, y, n, rstd = ws[0].clone(), *(torch.empty(M, K, device="cuda", dtype=BF16) for _ in range(3)), torch.empty(M, device="cuda")
    x0 = torch.randn(M, K, device="cuda").to(BF16)

    def walk(wait):
        x.copy_(x0)
        wait()
        for step in range(12):
            w.copy_(ws[step % 4])  # the weights of the product right behind
            wait()
            ops.gemm(x, w, out=y)
            wait()
            ops.rmsnorm_fwd(y, gamma, 1e-5, y=n, rstd=rstd)
            wait()
            ops.gemm(n, ws[(step + 1) % 4], residual=x, out=y)  # y has been read
            wait()
            ops.gemm(y, ws[(step + 2) % 4], out=x)
            wait()
        return x.clone()

    want = walk(torch.cuda.synchronize)
    assert want.isfinite().all()
    for _ in range(20):
        assert torch.equal(walk(lambda: None), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = walk(lambda: None)
    for _ in range(5):
        graph.replay()
        assert torch.equal(got, want)


@pytest.mark.parametrize("M", [9, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(22016, 520), (9000, 1032), (2176, 4104)])
def test_tiles_of_fewer_rows_and_clusters(M, N, K):
    """Matrices that are cut into tiles of 64 to 128 rows and clusters of one to eight, the last tile and the last slice of K ragged."""
    from llark_b200 import ops

    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device="cuda").to(BF16), (torch.randn(N, K, device="cuda") * K ** -0.5).to(BF16)
    z = x.to(F64) @ w.to(F64).t()
    # fp32 results: only the order and the cut of the sums shows, 5e-6 as above; bf16: one rounding, 2^-8 of a value; gate times up
    # rounds its two sums, the gate's function and the result: four of 2^-9 each at most
    assert _rel(ops.linear(x, w, out_dtype=F32), z) < 5e-6
    assert _rel(ops.linear(x, w, act="relu_glu"), torch.relu(z[:, 0::2]) * z[:, 1::2]) < 2.0 ** -8
    if N % 16 == 0:  # rows of the result on 16-byte boundaries
        g, u = z[:, :N // 2], z[:, N // 2:]
        assert _rel(ops.gemm(x, w, swiglu=True), torch.nn.functional.silu(g) * u) < 2.0 ** -7


@pytest.mark.parametrize("M", [9, 32, 33])
@pytest.mark.parametrize("N,K", [(1024, 512), (6144, 1024), (2048, 2048), (4224, 2048), (2560, 2560)])
def test_chains_over_k_are_short(M, N, K):
    """A chain of n products of 16 channels in the tensor cores' adders, which cut, loses about n / 4 of 2^-24 (2.3e-7 over 256 channels, 4.7e-7 over
    512); these sizes are cut into chains of 256 or 320. Half as much again is allowed; a chain twice as long is not."""
    from llark_b200 import ops

    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device="cuda").to(BF16), (torch.randn(N, K, device="cuda") * K ** -0.5).to(BF16)
    chain = 320 if K == 2560 else 256
    assert _rel(ops.linear(x, w, out_dtype=F32), x.to(F64) @ w.to(F64).t()) < 1.5 * chain / 16 / 4 * 2.0 ** -24


@pytest.mark.parametrize("n", [1, 8, 40])
def test_one_token_kernels_that_begin_early_see_what_was_written_before(n):
    """The recurrence's step and the norm with the next convolution between products, each input written by the launch in front and each buffer
    written again while the launch in front may still read it: against the same launches one at a time."""
    from llark_b200 import ops
    from llark_b200.state_cache import StepLayout

    torch.manual_seed(n)
    H, D, E, C, taps = 4, 128, 128, 512, 4
    wide = [(torch.randn(3 * C, C, device="cuda") * C ** -0.5).to(BF16) for _ in range(2)]
    square = [(torch.randn(C, C, device="cuda") * C ** -0.5).to(BF16) for _ in range(2)]
    norm, row_norm, cw = torch.rand(E, device="cuda"), torch.rand(C, device="cuda"), torch.randn(C, taps, device="cuda") / 2
    s0, t0, x0 = torch.randn(n, H, D, E, device="cuda"), torch.randn(n, taps - 1, C, device="cuda"), torch.randn(n, C, device="cuda")
    src, y = torch.empty(n, 3 * C, device="cuda"), torch.empty(n, C, device="cuda")
    w, low = norm.clone(), torch.empty(H * D, device="cuda")

    def walk(wait):
        state, tail, x = s0.clone(), t0.clone(), x0.clone()
        st = StepLayout([1] * n, [0] * n, list(range(n))[::-1], torch.device("cuda"))
        wait()
        h = x.to(BF16)
        wait()
        for step in range(12):
            ops.linear(h, wide[step % 2], out=src)
            wait()
            low.fill_(0.1 * (step % 3))
            wait()
            w.copy_(norm if step % 2 else 2 * norm)  # what the step right behind reads
            wait()
            o = ops.seq_glr_step(src, 0, H * D, 2 * H * D, low, state, st, H, D, E, w, 1e-5, BF16)
            wait()
            ops.linear(o, square[step % 2], out=y)
            wait()
            x, h = ops.seq_add_rmsnorm_conv(x, y, row_norm, 1e-5, cw, tail, st, BF16)
            wait()
        return x, h, state, tail

    want = walk(torch.cuda.synchronize)
    assert all(v.float().isfinite().all() for v in want)
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(walk(lambda: None), want))


@pytest.mark.parametrize("M", [9, 33, 64])
def test_rows_that_lie_in_each_other(M):
    """One row for all tokens, and rows that begin 8 entries after each other, as tokens and as weights: the same as of copies of them."""
    from llark_b200 import ops

    torch.manual_seed(M)
    K = N = 512
    long, w, r = torch.randn(K + 8 * N, device="cuda").to(BF16), (torch.randn(N, K, device="cuda") * K ** -0.5).to(BF16), torch.randn(M, N, device="cuda").to(BF16)
    cos, sin = (torch.rand(5, 128, device="cuda").to(BF16) for _ in range(2))
    for x, v in ((long[:K].expand(M, K), w), (long.as_strided((M, K), (8, 1)), w), (w[:M], (long * K ** -0.5).as_strided((N, K), (8, 1)))):
        z = x.to(F64) @ v.to(F64).t()
        assert _rel(ops.gemm(x, v, out_dtype=F32), z) < 5e-6  # fp32 sums in any order, as above
        assert _rel(ops.gemm(x, v, residual=r), z + r.to(F64)) < 2.0 ** -8  # one rounding of the result
        want = ops.gemm(x.contiguous(), v.contiguous(), rope=(cos, sin, 5, 256))
        # the same sums but for their order, which moves a rounding to bf16 here and there: sums, products and result are rounded
        assert _rel(ops.gemm(x, v, rope=(cos, sin, 5, 256)), want.to(F64)) < 2.0 ** -8
