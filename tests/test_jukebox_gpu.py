"""GPU parity of the Jukebox front-end mirror (llark_b200/jukebox) against oracle/jukebox_oracle.py (CPU
restatement; network parity UNPINNED upstream, see its header) and against the reference's own windowed_average
golden (tests/golden/pool_ref.pt). Tolerances: fp32 SIMT kernels 1e-4 rel; TF32 tensor-core GEMM path 5e-3 rel;
bf16 mode 4e-2 rel; VQ codes equal except at near-ties (reported margin < 1e-4)."""
import math
import os

import numpy as np
import pytest
import torch

from llark_b200.testing import check_close  # noqa: E402

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return ((a - b).norm() / (b.norm() + 1e-30)).item()


def _cfgs():
    from oracle import jukebox_oracle as jo
    from llark_b200.jukebox.model import JukeboxConfig

    ocfg = jo.tiny_cfg()
    keys = ("sample_length", "downs_t", "width", "depth", "emb_width", "l_bins", "dilation_growth_rate", "n_ctx",
            "prior_width", "prior_depth", "heads", "m_attn", "m_mlp", "blocks", "ln_eps")
    return jo, ocfg, JukeboxConfig(**{k: getattr(ocfg, k) for k in keys})


def test_conv_encoder_and_vq_match_oracle():
    jo, ocfg, cfg = _cfgs()
    from llark_b200.jukebox.model import JukeboxVQVAE

    vq = jo.init_vqvae_params(ocfg, seed=0)
    g = torch.Generator().manual_seed(5)
    audio = torch.rand(3, ocfg.sample_length, generator=g) * 2 - 1
    lat_o = jo.encoder_top(audio[:, None, :], vq, ocfg)
    codes_o, dist = jo.vq_nearest(lat_o, vq["codebook"])
    m = JukeboxVQVAE(cfg, vq)
    lat = m.encode_top_latents(audio[:, None, :].cuda().contiguous())
    assert lat.shape == lat_o.shape
    check_close("test_conv_encoder_and_vq_match_oracle:_rel_lat_lat_o_", _rel(lat, lat_o), 1e-4)
    codes = m.encode(audio[:, :, None].cuda())[-1].cpu()
    assert codes.dtype == torch.int64 and codes.shape == codes_o.shape
    neq = (codes != codes_o).flatten().nonzero().flatten()
    if len(neq):  # only near-ties may differ (different fp32 summation order)
        d = dist[neq]
        top2 = d.topk(2, largest=False).values
        margin = (top2[:, 1] - top2[:, 0]) / top2[:, 1].abs().clamp_min(1e-6)
        assert margin.max().item() < 1e-4, margin.max().item()
    assert len(neq) <= 0.002 * codes.numel()
    # codes computed from the ORACLE's latents must be bit-exact except ties
    from llark_b200 import ops

    codes2 = ops.jb_vq_encode(lat_o.cuda().contiguous(), vq["codebook"].cuda()).cpu()
    assert (codes2 != codes_o).float().mean().item() < 1e-3


@pytest.mark.parametrize("precision,tol", [("3xtf32", 2e-5), ("tf32", 5e-3), ("bf16", 1.5e-2)])
def test_prior_forward_matches_oracle(precision, tol):
    jo, ocfg, cfg = _cfgs()
    from llark_b200.jukebox.model import JukeboxTopPrior

    pp = jo.init_prior_params(ocfg, seed=1)
    g = torch.Generator().manual_seed(9)
    codes = torch.randint(0, ocfg.l_bins, (2, ocfg.n_ctx), generator=g)
    ref = jo.prior_forward(codes, pp, ocfg)
    tp = JukeboxTopPrior(cfg, pp, precision=precision)
    tp.prior.only_encode = True
    out = tp.prior.forward(codes.cuda(), x_cond=None, y_cond=None, encoder_kv=None, fp16=False)
    assert out.shape == ref.shape and out.dtype == torch.float32
    check_close(f"test_prior_forward_matches_oracle:{precision}", _rel(out, ref), tol)
    with pytest.raises(NotImplementedError):
        tp.prior.forward(codes.cuda(), fp16=True)


@pytest.mark.parametrize("pattern", [0, 1, 2])
def test_sparse_attention_real_head_shape(pattern):
    """8 heads x 150, block 64, T = 2048 (32 blocks): the prior's real head geometry."""
    from oracle import jukebox_oracle as jo
    from llark_b200 import ops

    cfg = jo.JukeboxCfg(n_ctx=2048, blocks=32, prior_width=4800)
    g = torch.Generator().manual_seed(pattern)
    qkv = torch.randn(1, 2048, 3 * cfg.attn_width, generator=g)
    ref = jo.factored_attention(qkv, cfg, pattern)
    q = qkv.view(2048, -1).cuda().contiguous()
    out = ops.jb_sparse_attn(q, 1, 2048, 8, 150, 64, pattern, exact=True)  # fp32 SIMT kernel
    check_close("test_sparse_attention_real_head_shape:_rel_out_view_1_2048_1_ref_", _rel(out.view(1, 2048, -1), ref), 1e-4)
    # tensor-core kernel: operands rounded to TF32 (10-bit mantissa), fp32 accumulate -> 2e-3; bf16 output adds 2^-9
    out_tc = ops.jb_sparse_attn(q, 1, 2048, 8, 150, 64, pattern)
    assert out_tc.dtype == torch.float32 and _rel(out_tc.view(1, 2048, -1), ref) < 2e-3
    out_bf = ops.jb_sparse_attn(q, 1, 2048, 8, 150, 64, pattern, out_dtype=torch.bfloat16)
    if pattern == 1:
        # 32 blocks -> 32-row groups: outside the tensor-core kernel's envelope (64 / 128 rows), so the wrapper ran the
        # fp32 SIMT kernel and hands back fp32 for the caller to cast
        assert out_bf.dtype == torch.float32 and torch.equal(out_bf, out)
    else:
        assert out_bf.dtype == torch.bfloat16 and _rel(out_bf.view(1, 2048, -1), ref) < 5e-3
        assert torch.equal(out_bf, out_tc.to(torch.bfloat16))


@pytest.mark.parametrize("pattern", [0, 1, 2])
def test_sparse_attention_tc_full_geometry(pattern):
    """T = 8192, 128 blocks of 64 (the real prior): pattern 1 gathers 128-row groups with stride 64."""
    from llark_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(10 + pattern)
    qkv = torch.randn(2 * 8192, 3600, device="cuda", generator=g)
    ref = ops.jb_sparse_attn(qkv, 2, 8192, 8, 150, 64, pattern, exact=True)
    got = ops.jb_sparse_attn(qkv, 2, 8192, 8, 150, 64, pattern)
    check_close("test_sparse_attention_tc_full_geometry:_rel_got_ref_", _rel(got, ref), 2e-3)


@pytest.mark.parametrize("N", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("T,W", [(1, 4), (7, 260), (1800, 4800)])  # the last: additive tables beyond what stays in L2
def test_prior_input_rows(N, T, W):
    """One, two or four clips a block, the last block's clips short: (token + position) + condition, y_cond at step 0, the same bits."""
    from llark_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(N + T)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    codes, emb = torch.randint(0, 40, (N, T), device="cuda", generator=g), r(40, W)
    y, pos, xc = r(W), r(T, W), r(T, W)
    rows = torch.cat([y.expand(N, 1, W), emb[codes[:, :-1]]], 1)
    assert torch.equal(ops.jb_embed_tokens(codes, emb, y, pos, xc).view(N, T, W), (rows + pos) + xc)


def test_pool_matches_reference_golden():
    from llark_b200.jukebox import main as jm

    ref = torch.load(os.path.join(GOLD, "pool_ref.pt"), weights_only=False)
    assert abs(jm.ACTS_SAMPLE_RATE - ref["acts_sample_rate"]) < 1e-9
    g = torch.Generator().manual_seed(ref["seed"])
    acts = torch.randn(ref["T_valid"], 4800, generator=g)
    pooled = jm.windowed_average(acts.cuda(), ref["frame_len"]).squeeze(0).cpu()
    assert tuple(pooled.shape) == ref["shape"]
    assert torch.allclose(pooled[:, :64], ref["pooled_head"], atol=1e-6)
    assert abs(pooled.double().sum().item() - ref["pooled_sum"]) < 1e-3
    # the batched launch (embed_batch): every clip pooled as the per-clip call pools it, odd widths / tails included
    for N, T, W, valid, frame in ((3, 700, 4800, 700, 34), (2, 64, 50, 61, 7), (1, 40, 4, 40, 1)):
        a = torch.randn(N, T, W, generator=torch.Generator().manual_seed(T)).cuda()
        got = jm.pool_batch(a, valid, frame)
        n = valid // frame
        want = a[:, : n * frame].reshape(N, n, frame, W).double().mean(2)
        assert got.shape == (N, n, W) and torch.allclose(got.double(), want, atol=1e-6)


def test_get_acts_from_file_end_to_end_tiny():
    jo, ocfg, cfg = _cfgs()
    from llark_b200.jukebox import main as jm

    vq, pp = jo.init_vqvae_params(ocfg, 0), jo.init_prior_params(ocfg, 1)
    hps, vqvae, top_prior = jm.load_model("5b", state=(vq, pp), cfg=cfg)
    g = torch.Generator().manual_seed(3)
    n = int(ocfg.sample_length * 0.8)  # shorter than the window: padded, activations truncated proportionally
    stereo = (torch.rand(2, n, generator=g) * 2 - 1).numpy().astype(np.float32)
    acts = jm.get_acts_from_file(stereo, hps, vqvae, top_prior, meanpool=True, pool_frames_per_second=10)
    ref = jo.get_acts(torch.from_numpy(stereo), vq, pp, ocfg, meanpool=True, pool_frames_per_second=10)
    assert acts.shape == tuple(ref.shape)
    # codes may differ at near-ties, which changes whole token embeddings: compare with a loose norm bound and
    # require most frames to agree tightly
    per_frame = ((torch.from_numpy(acts) - ref).norm(dim=1) / ref.norm(dim=1))
    assert (per_frame < 2e-2).float().mean().item() > 0.9
    with pytest.raises(AssertionError):
        jm.get_z(np.zeros(10, dtype=np.float32), vqvae)
    full = jm.get_acts_from_file(stereo, hps, vqvae, top_prior, meanpool=True, pool_frames_per_second=0)
    assert full.shape == (ocfg.prior_width,)


def test_label_conditioning_on_gpu_matches_oracle_and_feeds_the_prior():
    """J4 on the GPU: get_cond through llark_jb_label_cond (bins on the host, table arithmetic in the kernel) is bit-equal
    to the oracle's LabelConditioner, embed_batch / get_acts_from_file use it (no ready-made x_cond / y_cond constants in
    the state), and the whole front end still agrees with the oracle run on those conditioning tensors."""
    jo, ocfg, cfg = _cfgs()
    from types import SimpleNamespace

    from llark_b200.jukebox import main as jm

    vq, pp = jo.init_vqvae_params(ocfg, 0), jo.init_prior_params(ocfg, 1)
    pp.pop("x_cond"), pp.pop("y_cond")
    tables = jo.init_label_params(ocfg, jo.LabelCfg(), seed=5)
    hps, vqvae, top_prior = jm.load_model("5b", state=(vq, {**pp, **tables}), cfg=cfg)
    assert top_prior.has_label_conditioner
    x_cond, y_cond = jm.get_cond(SimpleNamespace(sr=44100, n_samples=8), top_prior)
    want_x, want_y = jo.get_cond(tables, ocfg, jo.LabelCfg())
    assert torch.equal(x_cond.cpu(), want_x) and torch.equal(y_cond.cpu(), want_y)
    g = torch.Generator().manual_seed(3)
    wav = (torch.rand(2, ocfg.sample_length, generator=g) * 2 - 1)
    got = jm.embed_batch(wav, vqvae, top_prior, pool_frames_per_second=10).cpu()
    opp = {**pp, "x_cond": want_x[0], "y_cond": want_y[0, 0]}
    for i in range(2):
        ref = jo.get_acts(wav[i], vq, opp, ocfg, meanpool=True, pool_frames_per_second=10)
        per_frame = (got[i] - ref).norm(dim=1) / ref.norm(dim=1)
        assert got[i].shape == ref.shape and (per_frame < 2e-2).float().mean().item() > 0.9


@pytest.mark.parametrize("d", [1, 3, 9, 27])
def test_resblock_tensor_core_kernel_matches_simt_and_fp64(d):
    """The split-TF32 res-block (default) against the fp32 SIMT kernel (LLARK_JB_CONV_TC=0) and an fp64 conv1d
    reference: both must sit at fp32 rounding level (the 3x split keeps ~22 mantissa bits), on a time length that is not a
    multiple of the 256-step tile and with the dilation's halo crossing tile borders."""
    import torch.nn.functional as F

    from llark_b200 import ops

    g = torch.Generator().manual_seed(d)
    N, T = 2, 3000
    x = torch.randn(N, 32, T, generator=g)
    w1 = torch.randn(32, 32, 3, generator=g) / math.sqrt(96)
    b1 = torch.randn(32, generator=g) * 0.1
    w2 = torch.randn(32, 32, 1, generator=g) / math.sqrt(32)
    b2 = torch.randn(32, generator=g) * 0.1
    h = F.conv1d(F.relu(x.double()), w1.double(), b1.double(), padding=d, dilation=d)
    ref = x.double() + F.conv1d(F.relu(h), w2.double(), b2.double())
    args = [t.cuda().contiguous() for t in (x, w1, b1, w2, b2)]
    os.environ["LLARK_JB_CONV_TC"] = "0"
    try:
        simt = ops.jb_resblock(*args, d).cpu()
    finally:
        os.environ.pop("LLARK_JB_CONV_TC", None)
    tc = ops.jb_resblock(*args, d).cpu()
    check_close(f"resblock_tc_vs_fp64:d{d}", _rel(tc, ref), 2e-6)
    check_close(f"resblock_simt_vs_fp64:d{d}", _rel(simt, ref), 2e-6)
    check_close(f"resblock_tc_vs_simt:d{d}", _rel(tc, simt), 2e-6)


@pytest.mark.parametrize("T", [2, 126, 128, 130, 1000])
@pytest.mark.parametrize("kind,c_in", [("down", 1), ("down", 32), ("down", 64), ("k3", 32), ("res1", 32), ("res27", 32), ("res64", 32), ("res81", 32)])
def test_convolutions_at_the_edges_of_their_tiles_match_fp64(kind, c_in, T):
    """The tcgen05 convolutions (tiles of 128 time steps, several per CTA and clip) against fp64 conv1d: fewer steps than a tile, one
    more than a tile, halos that cross clip ends. Split operands keep 22 bits and chains are 12 products long: 1e-6 of the result."""
    import torch.nn.functional as F

    from llark_b200 import ops

    g = torch.Generator().manual_seed(T + c_in)
    N = 3
    x = torch.randn(N, c_in, T, generator=g)
    xd = x.double()
    if kind == "down":
        w, b = torch.randn(32, c_in, 4, generator=g) / math.sqrt(4 * c_in), torch.randn(32, generator=g) * 0.1
        got, ref = ops.jb_conv_down(x.cuda(), w.cuda(), b.cuda()), F.conv1d(xd, w.double(), b.double(), stride=2, padding=1)
    elif kind == "k3":
        w, b = torch.randn(64, 32, 3, generator=g) / math.sqrt(96), torch.randn(64, generator=g) * 0.1
        got, ref = ops.jb_conv_k3(x.cuda(), w.cuda(), b.cuda()), F.conv1d(xd, w.double(), b.double(), padding=1)
    else:
        d = int(kind[3:])
        w1, b1 = torch.randn(32, 32, 3, generator=g) / math.sqrt(96), torch.randn(32, generator=g) * 0.1
        w2, b2 = torch.randn(32, 32, 1, generator=g) / math.sqrt(32), torch.randn(32, generator=g) * 0.1
        got = ops.jb_resblock(*(t.cuda() for t in (x, w1, b1, w2, b2)), d)
        h = F.conv1d(F.relu(xd), w1.double(), b1.double(), padding=d, dilation=d)
        ref = xd + F.conv1d(F.relu(h), w2.double(), b2.double())
    assert _rel(got.cpu(), ref) < 1e-6


@pytest.mark.parametrize("T", [2, 431, 432, 433, 1000])
@pytest.mark.parametrize("dils", [(1, 3, 9, 27), (27, 9, 3, 1), (32, 32, 32), (2, 5), (1, 3, 9, 27, 81), (40, 1, 1)])
def test_res_blocks_in_one_visit_match_fp64(dils, T):
    """Runs of res blocks against fp64 conv1d block after block: shorter than a window's results, one step more, windows that begin and
    end at the clip's ends, runs whose last block goes alone. Split operands keep 24 bits: 1e-6 of the result, as block by block."""
    import torch.nn.functional as F

    from llark_b200 import ops

    g = torch.Generator().manual_seed(T + len(dils))
    x = torch.randn(3, 32, T, generator=g)
    blocks, ref = [], x.double()
    for d in dils:
        w1, b1 = torch.randn(32, 32, 3, generator=g) / math.sqrt(96), torch.randn(32, generator=g) * 0.1
        w2, b2 = torch.randn(32, 32, 1, generator=g) / math.sqrt(32), torch.randn(32, generator=g) * 0.1
        blocks.append((w1.cuda(), b1.cuda(), w2.cuda(), b2.cuda()))
        h = F.conv1d(F.relu(ref), w1.double(), b1.double(), padding=d, dilation=d)
        ref = ref + F.conv1d(F.relu(h), w2.double(), b2.double())
    got = ops.jb_resblocks(x.cuda(), blocks, dils)
    one = x.cuda()
    for b, d in zip(blocks, dils):
        one = ops.jb_resblock(one, *b, d)
    assert _rel(got.cpu(), ref) < 1e-6
    assert _rel(got.cpu(), ref) < 1.2 * _rel(one.cpu(), ref) + 1e-8


def _by_fma(fn, *args):
    """fn with the FMA kernels of the encoder's convolutions."""
    os.environ["LLARK_JB_CONV_TC"] = "0"
    try:
        return fn(*args)
    finally:
        os.environ.pop("LLARK_JB_CONV_TC", None)


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf"), 3.4e38, -3.4027e38])
@pytest.mark.parametrize("kind,c_in", [("down", 32), ("down", 64), ("k3", 32)])
def test_values_that_do_not_split_come_out_where_conv1d_puts_them(kind, c_in, bad):
    """NaN, infinities and numbers whose leading part rounds to infinity: exactly the steps that see them differ, as sums of products
    have it; a NaN of the GPU's own arithmetic (0x7fffffff) too. All other steps keep their split products (1e-6, as above)."""
    import torch.nn.functional as F

    from llark_b200 import ops

    g = torch.Generator().manual_seed(c_in)
    T, c_out, taps = 300, 64 if kind == "k3" else 32, 3 if kind == "k3" else 4
    x = torch.randn(2, c_in, T, generator=g)
    w = torch.randn(c_out, c_in, taps, generator=g) / (taps * c_in)
    w[0, 5] = 0.0  # 0 times infinity
    b = torch.randn(c_out, generator=g) * 0.1
    x[0, 5, 0], x[0, 7, 131], x[1, c_in - 1, T - 1] = bad, bad, bad
    xc = x.cuda()
    if bad != bad:
        xc[0, 7, 131] = (torch.full((1,), float("inf"), device="cuda") - float("inf"))[0]
    op = ops.jb_conv_k3 if kind == "k3" else ops.jb_conv_down
    got = op(xc, w.cuda(), b.cuda()).cpu()
    ref = F.conv1d(x.double(), w.double(), b.double(), stride=1 if kind == "k3" else 2, padding=1).float()
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf())
    assert torch.equal(got[got.isinf()], ref[ref.isinf()])
    ok = ref.isfinite()
    big = ok & (ref.abs() > 1e30)
    assert big.any() == (abs(bad) < float("inf"))
    # fp32 sums of at most 256 products
    assert ((got[ok].double() - ref[ok].double()).abs() <= 256 * 2.0 ** -24 * F.conv1d(
        x.nan_to_num(0, 0, 0).abs().double(), w.abs().double(), b.abs().double(), stride=1 if kind == "k3" else 2, padding=1)[ok]).all()
    if abs(bad) > 3.402e38:  # rounds to infinity: these steps are sums of FMAs
        assert torch.equal(_by_fma(op, xc, w.cuda(), b.cuda()).cpu()[big], got[big])


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf"), 3.4e38, -3.4027e38, 2e25])
@pytest.mark.parametrize("dils", [(1, 3, 9, 27), (27, 1), (3,), (40, 1), (81,)])
@pytest.mark.parametrize("where", ["values", "weights", "bias"])
def test_res_blocks_with_values_that_do_not_split(dils, where, bad):
    """NaN, infinities and numbers whose sums may pass the largest one, among the values, the weights and the biases: the same steps are
    infinite and NaN as with the FMA kernels, block after block (relu(NaN) is 0 in both), and all others differ by roundings: two ways of 128
    products in a block, 1e-5 of what a step holds."""
    from llark_b200 import ops

    g = torch.Generator().manual_seed(len(dils))
    T = 1200
    x = torch.randn(2, 32, T, generator=g)
    blocks = [[torch.randn(32, 32, 3, generator=g) / math.sqrt(96), torch.randn(32, generator=g) * 0.1,
               torch.randn(32, 32, 1, generator=g) / math.sqrt(32), torch.randn(32, generator=g) * 0.1] for _ in dils]
    if where == "values":
        x[0, 5, 0], x[0, 7, 431], x[1, 31, T - 1] = bad, bad, bad
    elif where == "weights":
        blocks[0][0][3, 4, 1] = bad
    else:
        blocks[0][1][9] = bad
    blocks, x = [tuple(t.cuda() for t in b) for b in blocks], x.cuda()
    got, want = ops.jb_resblocks(x, blocks, dils), _by_fma(ops.jb_resblocks, x, blocks, dils)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    ok = want.isfinite()
    size = torch.where(ok, want.abs(), 0).amax(1, keepdim=True)  # of a step: its channels are sums of the same numbers
    assert ((got - want).abs() <= 1e-5 * (1 + size))[ok].all()
    if where == "values" and bad == float("inf"):
        assert not want.isfinite()[0, :, 431 - dils[0]].all()  # the neighbours see it


def test_a_nan_sample_stays_nan_through_the_encoder():
    """From the second level on the activations' NaN is the one the GPU's arithmetic gives; relu(NaN) is 0 in the res blocks (fmaxf), so
    the latents that see it through the residual sums are NaN, with either kind of kernel."""
    jo, ocfg, cfg = _cfgs()
    from llark_b200.jukebox.model import JukeboxVQVAE

    m = JukeboxVQVAE(cfg, jo.init_vqvae_params(ocfg, seed=0))
    audio = torch.rand(1, 1, ocfg.sample_length, generator=torch.Generator().manual_seed(5)) * 2 - 1
    audio[0, 0, ocfg.sample_length // 2] = float("nan")
    got = m.encode_top_latents(audio.cuda())
    want = _by_fma(m.encode_top_latents, audio.cuda())
    assert want.isnan().any() and not want.isnan().all()
    assert torch.equal(got.isnan(), want.isnan())


def _fma(a, b, c):
    """a b + c in fp32, rounded once: the exact sum of the product and c rounded to odd in 64 bits, which leaves what rounding to 24 needs."""
    p, c = a.double() * b.double(), c.double()  # the product of two fp32 numbers is exact
    p, c = torch.broadcast_tensors(p, c)
    s = p + c
    bb = s - p
    err = (p - (s - bb)) + (c - bb)  # what s lacks, exactly
    bits = s.view(torch.int64)
    odd = torch.where((err != 0) & (bits & 1 == 0) & s.isfinite(), torch.where((err > 0) == (s > 0), bits + 1, bits - 1), bits)
    return odd.view(torch.float64).float()


def _walk(x, cb):
    """The first least of (|x|^2 - 2 x.k) + |k|^2 for x [N, 64, T], every sum FMA after FMA in the order of the channels; 0 where none is
    below infinity."""
    flat = x.permute(0, 2, 1).reshape(-1, 64)
    zero = flat.new_zeros
    xx, kk, dot = zero(len(flat)), zero(len(cb)), zero(len(flat), len(cb))
    for e in range(64):
        xx, kk = _fma(flat[:, e], flat[:, e], xx), _fma(cb[:, e], cb[:, e], kk)
        dot = _fma(flat[:, e, None], cb[None, :, e], dot)
    dist = _fma(dot.new_tensor(-2.0), dot, xx[:, None]) + kk[None]
    dist = torch.where(dist < float("inf"), dist, torch.full_like(dist, float("inf")))
    return (dist == dist.min(1, keepdim=True).values).int().argmax(1).view(x.shape[0], x.shape[2]), dist


@pytest.mark.parametrize("T,n_codes", [(1, 1), (129, 256), (130, 257), (300, 2048), (128, 1000),  # walked as they are
                                       (4800, 257), (4737, 2048), (9600, 300), (9473, 2047)])  # CTAs of 128 vectors, of 256
@pytest.mark.parametrize("kind", ["spread", "crowded", "close pairs", "lengths apart", "equal", "not finite", "large"])
def test_nearest_code_is_that_of_the_walk_over_all_codes(T, n_codes, kind):
    """The candidates that tensor cores leave against fp32 walks over all codes, which must name the same ones: codes far apart, codes
    closer together than bf16 tells them apart (lists overflow), pairs of codes a few units of the last place of dist apart, the same with
    lengths that grow a hundredfold from tile to tile, equal codes, numbers that are not finite, squares near the largest number."""
    from llark_b200 import ops

    g = torch.Generator().manual_seed(T + n_codes)
    x, cb = torch.randn(2, 64, T, generator=g), torch.randn(n_codes, 64, generator=g)
    if kind == "crowded":
        cb = cb[:1] + 1e-3 * cb
    if kind in ("close pairs", "lengths apart"):
        if kind == "lengths apart":
            cb *= 10.0 ** (torch.arange(n_codes) // 128 % 3 - 1.0)[:, None]
        cb[n_codes // 2:] = cb[:n_codes - n_codes // 2] * (1 + 3e-7 * torch.randn(n_codes - n_codes // 2, 64, generator=g))
        x = (cb[torch.randint(0, n_codes, (2 * T,), generator=g)] * 0.9 + 0.02 * torch.randn(2 * T, 64, generator=g)).view(2, T, 64).permute(0, 2, 1).contiguous()
    if kind == "equal":
        cb = cb[torch.arange(n_codes) % 3 if n_codes >= 3 else torch.zeros(n_codes, dtype=torch.long)]
    if kind == "not finite":
        cb[n_codes // 2, 3] = float("inf")
        cb[n_codes // 3, 5] = float("nan")
        cb[n_codes // 4] = 1e25  # |k|^2 overflows
        x[0, 1, 0], x[1, 2, T - 1], x[1, 0, T // 2] = float("nan"), float("inf"), 1e25
    if kind == "large":  # |k|^2 just below the largest number, or above it
        cb *= 1.8446e19 * (1 + 1e-5 * torch.randn(n_codes, 1, generator=g)) / cb.norm(dim=1, keepdim=True)
        x[1] *= 1e18
    codes = ops.jb_vq_encode(x.cuda(), cb.cuda())
    want, dist = _walk(x.cuda(), cb.cuda())
    assert torch.equal(codes, want)
    if kind in ("close pairs", "lengths apart") and n_codes > 1:  # the test's point: the two nearest are within the bound of each other
        two = dist.topk(2, dim=1, largest=False).values
        assert ((two[:, 1] - two[:, 0]) < 2.0 ** -13 * cb.norm(dim=1).max() ** 2).float().mean() > 0.9


@pytest.mark.parametrize("T,n_codes", [(1, 5), (64, 2048), (65, 2047), (200, 37)])
def test_nearest_code_in_every_slice_of_the_codebook(T, n_codes):
    """Codebooks that end inside a tile, vectors that end inside a row tile: the fp32 distances of one walk over all codes, the first
    minimum wins."""
    from llark_b200 import ops

    g = torch.Generator().manual_seed(T)
    x, cb = torch.randn(2, 64, T, generator=g), torch.randn(n_codes, 64, generator=g)
    cb[n_codes // 2] = cb[0]  # a tie across slices
    x[0, :, 0] = cb[0]
    codes = ops.jb_vq_encode(x.cuda(), cb.cuda()).cpu()
    flat = x.permute(0, 2, 1).reshape(-1, 64).double()
    dist = (flat.pow(2).sum(1, keepdim=True) - 2 * flat @ cb.double().t() + cb.double().pow(2).sum(1)[None])
    best = dist.min(1).values
    got = dist.gather(1, codes.view(-1, 1)).squeeze(1)
    assert ((got - best) <= 1e-4 * best.clamp_min(1.0)).all()  # fp32 sums of 64 terms
    assert codes[0, 0].item() == 0  # the first of two equal ones
