"""ORACLE (test infrastructure only -- never imported by the product path).  PARITY UNPINNED for the network:

CPU/PyTorch restatement of the Jukebox "5b" front end as LLark uses it: VQ-VAE top-level (level 2) encoder ->
nearest-code bottleneck -> prior embedding + 36 factored-attention transformer blocks (only_encode) -> 10 Hz
mean-pool.  The arithmetic lives in openai/jukebox @ 08efbbc1d4ed1a3cef96e08a931944c8b4d63bb3
(docker/jukebox-embed.dockerfile:50-51), which the reference does NOT vendor and not installed; neither the
source nor the weights are reachable offline.  This file restates the published architecture
([UPSTREAM-RECALLED]) and anchors on the reference's own call sites:

    jukebox/main.py:29-45   load_audio_from_file   (mono mean, peak normalise)          -> normalize_audio
    jukebox/main.py:48-51   maybe_pad_audio_to_max_len                                     -> pad_or_truncate
    jukebox/main.py:54-68   get_z -> vqvae.encode, zs[-1]                                  -> vqvae_encode_top
    jukebox/main.py:71-98   get_cond (constant for the fixed metas)                        -> x_cond / y_cond tensors
    jukebox/main.py:101-110 get_final_activations -> prior.forward(only_encode, fp16=False) -> prior_forward
    jukebox/main.py:113-130 windowed_average (AvgPool1d(frame, frame), floor)               -> windowed_average
    jukebox/main.py:133-173 get_acts_from_file                                              -> get_acts

Only `windowed_average` / the frame arithmetic are pinned against the reference itself (tests/golden/pool_ref.pt,
generated by importing jukebox/main.py in place).  The network restatement has no golden vectors from upstream.
"""
import math
from dataclasses import dataclass
from math import floor

import torch
import torch.nn.functional as F

JUKEBOX_SAMPLE_RATE = 44100
T_FULL = 8192
JUKEBOX_EXPECTED_SAMPLES_LEN = 1048576
ACTS_SAMPLE_RATE = T_FULL / (JUKEBOX_EXPECTED_SAMPLES_LEN / JUKEBOX_SAMPLE_RATE)  # jukebox/main.py:10-22


def frame_len(pool_frames_per_second):
    return floor(ACTS_SAMPLE_RATE / pool_frames_per_second)  # jukebox/main.py:157


@dataclass
class JukeboxCfg:
    # VQ-VAE level-2 encoder (hparams.py: vqvae)
    sample_length: int = JUKEBOX_EXPECTED_SAMPLES_LEN
    downs_t: tuple = (3, 2, 2)
    width: int = 32
    depth: int = 4
    emb_width: int = 64
    l_bins: int = 2048
    dilation_growth_rate: int = 3
    # prior_5b as loaded by the reference (prior_depth forced to 36, jukebox/main.py:197)
    n_ctx: int = 8192
    prior_width: int = 4800
    prior_depth: int = 36
    heads: int = 8
    m_attn: float = 0.25
    m_mlp: float = 1.0
    blocks: int = 128
    ln_eps: float = 1e-5

    @property
    def hop(self):
        return 2 ** sum(self.downs_t)

    @property
    def attn_width(self):
        return int(self.m_attn * self.prior_width)

    @property
    def mlp_width(self):
        return int(self.m_mlp * self.prior_width)

    @property
    def block_ctx(self):
        return self.n_ctx // self.blocks


def tiny_cfg():
    """Small shapes with the same structure (three encoder blocks, three attention patterns)."""
    return JukeboxCfg(sample_length=128 * 256, l_bins=64, n_ctx=256, prior_width=64, prior_depth=3, heads=2,
                      m_attn=0.5, blocks=16)


# ------------------------------------------------------------------------------------------------ parameters
def init_vqvae_params(cfg, seed=0):
    g = torch.Generator().manual_seed(seed)
    p = {}
    c_in = 1
    for b, down_t in enumerate(cfg.downs_t):
        for i in range(down_t):
            cin = c_in if i == 0 else cfg.width
            p[f"enc.{b}.down.{i}.w"] = torch.randn(cfg.width, cin, 4, generator=g) / math.sqrt(cin * 4)
            p[f"enc.{b}.down.{i}.b"] = torch.randn(cfg.width, generator=g) * 0.02
            for d in range(cfg.depth):
                p[f"enc.{b}.res.{i}.{d}.w1"] = torch.randn(cfg.width, cfg.width, 3, generator=g) / math.sqrt(cfg.width * 3)
                p[f"enc.{b}.res.{i}.{d}.b1"] = torch.randn(cfg.width, generator=g) * 0.02
                p[f"enc.{b}.res.{i}.{d}.w2"] = torch.randn(cfg.width, cfg.width, 1, generator=g) / math.sqrt(cfg.width)
                p[f"enc.{b}.res.{i}.{d}.b2"] = torch.randn(cfg.width, generator=g) * 0.02
        p[f"enc.{b}.proj.w"] = torch.randn(cfg.emb_width, cfg.width, 3, generator=g) / math.sqrt(cfg.width * 3)
        p[f"enc.{b}.proj.b"] = torch.randn(cfg.emb_width, generator=g) * 0.02
        c_in = cfg.emb_width
    p["codebook"] = torch.randn(cfg.l_bins, cfg.emb_width, generator=g)
    return p


def init_prior_params(cfg, seed=1):
    g = torch.Generator().manual_seed(seed)
    W, A, Mw = cfg.prior_width, cfg.attn_width, cfg.mlp_width
    p = {"x_emb": torch.randn(cfg.l_bins, W, generator=g) * 0.02,
         "pos_emb": torch.randn(cfg.n_ctx, W, generator=g) * 0.01,
         # constants produced by get_cond for the fixed metas of jukebox/main.py:81-89
         "x_cond": torch.randn(cfg.n_ctx, W, generator=g) * 0.01,
         "y_cond": torch.randn(W, generator=g) * 0.02}
    for d in range(cfg.prior_depth):
        q = f"blk.{d}."
        p[q + "ln0.g"] = 1 + 0.1 * torch.randn(W, generator=g)
        p[q + "ln0.b"] = 0.02 * torch.randn(W, generator=g)
        p[q + "c_attn.w"] = torch.randn(W, 3 * A, generator=g) * (0.7 / math.sqrt(W))  # Conv1D: [n_in, n_out]
        p[q + "c_attn.b"] = 0.02 * torch.randn(3 * A, generator=g)
        p[q + "c_proj.w"] = torch.randn(A, W, generator=g) * (0.3 / math.sqrt(A))
        p[q + "c_proj.b"] = 0.02 * torch.randn(W, generator=g)
        p[q + "ln1.g"] = 1 + 0.1 * torch.randn(W, generator=g)
        p[q + "ln1.b"] = 0.02 * torch.randn(W, generator=g)
        p[q + "fc.w"] = torch.randn(W, Mw, generator=g) * (0.7 / math.sqrt(W))
        p[q + "fc.b"] = 0.02 * torch.randn(Mw, generator=g)
        p[q + "fc_proj.w"] = torch.randn(Mw, W, generator=g) * (0.3 / math.sqrt(Mw))
        p[q + "fc_proj.b"] = 0.02 * torch.randn(W, generator=g)
    return p


# ------------------------------------------------------------------------------------------------ pre/post-processing
def normalize_audio(audio):
    """jukebox/main.py:36-45: channel mean then divide by max-abs (skipped when 0). audio [C,n] or [n]."""
    if audio.ndim == 1:
        audio = audio[None]
    audio = audio.mean(dim=0)
    norm = audio.abs().max()
    if norm > 0:
        audio = audio / norm
    return audio.flatten()


def pad_or_truncate(audio, n=JUKEBOX_EXPECTED_SAMPLES_LEN):
    """jukebox/main.py:48-51 (right zero-pad) and :59 (truncate)."""
    if audio.numel() < n:
        audio = F.pad(audio, (0, n - audio.numel()))
    return audio[:n]


def windowed_average(acts, frame, ceil_mode=False):
    """jukebox/main.py:113-130."""
    assert acts.ndim == 2
    a = acts[None].transpose(1, 2)
    a = F.avg_pool1d(a, frame, stride=frame, ceil_mode=ceil_mode)
    return a.transpose(1, 2).squeeze(0)


# ------------------------------------------------------------------------------------------------ VQ-VAE level 2
def encoder_top(x, p, cfg):
    """x [N,1,T] -> [N,64,T/128]: EncoderConvBlocks (Conv1d k4 s2 p1 + Resnet1D(dilations 3^d)) then Conv1d k3."""
    h = x
    for b, down_t in enumerate(cfg.downs_t):
        for i in range(down_t):
            h = F.conv1d(h, p[f"enc.{b}.down.{i}.w"], p[f"enc.{b}.down.{i}.b"], stride=2, padding=1)
            for d in range(cfg.depth):
                dil = cfg.dilation_growth_rate ** d
                r = F.conv1d(F.relu(h), p[f"enc.{b}.res.{i}.{d}.w1"], p[f"enc.{b}.res.{i}.{d}.b1"], padding=dil,
                             dilation=dil)
                r = F.conv1d(F.relu(r), p[f"enc.{b}.res.{i}.{d}.w2"], p[f"enc.{b}.res.{i}.{d}.b2"])
                h = h + r
        h = F.conv1d(h, p[f"enc.{b}.proj.w"], p[f"enc.{b}.proj.b"], padding=1)
    return h


def vq_nearest(x, codebook):
    """bottleneck.encode: x [N,64,T] -> codes int64 [N,T]; dist = sum x^2 - 2 x k^T + sum k^2, argmin."""
    N, E, T = x.shape
    xf = x.permute(0, 2, 1).reshape(-1, E)
    dist = xf.pow(2).sum(-1, keepdim=True) - 2 * xf @ codebook.t() + codebook.pow(2).sum(-1)[None]
    return dist.argmin(-1).view(N, T), dist


def vqvae_encode_top(audio, p, cfg):
    """jukebox/main.py:61-63: vqvae.encode(x[N,T,1]) and keep zs[-1]."""
    x = audio.view(audio.shape[0], 1, -1).float()
    return vq_nearest(encoder_top(x, p, cfg), p["codebook"])[0]


# ------------------------------------------------------------------------------------------------ prior (only_encode)
def _layernorm(x, g, b, eps):
    return F.layer_norm(x, (x.shape[-1],), g, b, eps)


def _dense_attn(q, k, v, causal, scale):
    w = torch.matmul(q * scale, (k * scale).transpose(-1, -2))
    if causal:
        n = w.shape[-1]
        mask = torch.ones(n, n).tril()
        w = w * mask + -1e9 * (1 - mask)
    return torch.matmul(F.softmax(w, dim=-1), v)


def factored_attention(qkv, cfg, pattern):
    """qkv [N,T,3A] -> [N,T,A]. pattern 0 block, 1 transposed block, 2 previous block (attn_order=2 cycle)."""
    N, T, _ = qkv.shape
    A, nh = cfg.attn_width, cfg.heads
    dh = A // nh
    bc = T // cfg.blocks if cfg.blocks <= T else T
    nb = T // bc
    scale = 1.0 / math.sqrt(math.sqrt(dh))
    q, k, v = qkv.chunk(3, dim=2)

    def heads(t):
        return t.view(N, T, nh, dh).permute(0, 2, 1, 3)  # [N,nh,T,dh]

    q, k, v = heads(q), heads(k), heads(v)
    if pattern == 0:
        f = lambda t: t.reshape(N, nh, nb, bc, dh)
        a = _dense_attn(f(q), f(k), f(v), True, scale).reshape(N, nh, T, dh)
    elif pattern == 1:
        f = lambda t: t.reshape(N, nh, nb, bc, dh).transpose(2, 3)  # [N,nh,bc,nb,dh]
        a = _dense_attn(f(q), f(k), f(v), True, scale).transpose(2, 3).reshape(N, nh, T, dh)
    else:
        qb = q.reshape(N, nh, nb, bc, dh)
        prev = lambda t: F.pad(t.reshape(N, nh, nb, bc, dh)[:, :, :-1], (0, 0, 0, 0, 1, 0))
        a = _dense_attn(qb, prev(k), prev(v), False, scale).reshape(N, nh, T, dh)
    return a.permute(0, 2, 1, 3).reshape(N, T, A)


def prior_forward(codes, p, cfg):
    """ConditionalAutoregressive2D.forward(only_encode=True, fp16=False): codes int64 [N,T] -> fp32 [N,T,W]."""
    N, T = codes.shape
    x = p["x_emb"][codes]
    x = torch.roll(x, 1, dims=1)
    x[:, 0] = p["y_cond"]
    x = x + p["pos_emb"][None, :T] + p["x_cond"][None, :T]
    for d in range(cfg.prior_depth):
        q = f"blk.{d}."
        h = _layernorm(x, p[q + "ln0.g"], p[q + "ln0.b"], cfg.ln_eps)
        qkv = torch.addmm(p[q + "c_attn.b"], h.view(-1, h.shape[-1]), p[q + "c_attn.w"]).view(N, T, -1)
        a = factored_attention(qkv, cfg, d % 3)
        a = torch.addmm(p[q + "c_proj.b"], a.reshape(-1, a.shape[-1]), p[q + "c_proj.w"]).view(N, T, -1)
        h = _layernorm(x + a, p[q + "ln1.g"], p[q + "ln1.b"], cfg.ln_eps)
        m = torch.addmm(p[q + "fc.b"], h.view(-1, h.shape[-1]), p[q + "fc.w"])
        m = m * torch.sigmoid(1.702 * m)  # quick-GELU
        m = torch.addmm(p[q + "fc_proj.b"], m, p[q + "fc_proj.w"]).view(N, T, -1)
        x = x + a + m
    return x


def get_acts(audio, vq_params, prior_params, cfg, meanpool=True, pool_frames_per_second=10):
    """jukebox/main.py:133-173 for an in-memory waveform (decode/resample J1 happens outside)."""
    audio = normalize_audio(audio)
    input_len = audio.numel()
    latent_len = floor(cfg.n_ctx * input_len / cfg.sample_length)
    audio = pad_or_truncate(audio, cfg.sample_length)
    z = vqvae_encode_top(audio[None], vq_params, cfg)
    if z.shape[-1] < cfg.n_ctx:
        raise ValueError("Audio file is not long enough")
    acts = prior_forward(z[:, : cfg.n_ctx], prior_params, cfg).squeeze(0).float()
    acts = acts[:latent_len]
    if meanpool:
        if not pool_frames_per_second:
            acts = acts.mean(dim=0)
        else:
            fl = floor((cfg.n_ctx / (cfg.sample_length / JUKEBOX_SAMPLE_RATE)) / pool_frames_per_second)
            acts = windowed_average(acts, fl)
    return acts


# ------------------------------------------------------------------------------------------------ label conditioning (J4)
# [UPSTREAM-RECALLED] jukebox/prior/conditioners.py (LabelConditioner, RangeEmbedding, SimpleEmbedding),
# jukebox/data/labels.py (Labeller), jukebox/prior/prior.py (SimplePrior.get_y / get_cond) @ 08efbbc, as reached from
# jukebox/main.py:71-98. prior_5b: labels_v3, y_bins = (604 genres, 7898 artists), t_bins = 64, max_bow_genre_size = 1,
# min_duration 60 s, max_duration 600 s, n_tokens = 0 (no lyrics).
@dataclass
class LabelCfg:
    genre_bins: int = 604
    artist_bins: int = 7898
    t_bins: int = 64
    max_bow_genre_size: int = 1
    min_duration: float = 60.0
    max_duration: float = 600.0
    sr: int = JUKEBOX_SAMPLE_RATE
    n_tokens: int = 0


def init_label_params(cfg, lcfg, seed=2, init_scale=1.0):
    """SimpleEmbedding / RangeEmbedding tables (nn.Embedding, std 0.01 * init_scale)."""
    g = torch.Generator().manual_seed(seed)
    W = cfg.prior_width
    std = 0.01 * init_scale
    return {"y_emb.genre": torch.randn(lcfg.genre_bins, W, generator=g) * std,
            "y_emb.artist": torch.randn(lcfg.artist_bins, W, generator=g) * std,
            "y_emb.total_length": torch.randn(lcfg.t_bins, W, generator=g) * std,
            "y_emb.absolute_pos": torch.randn(lcfg.t_bins, W, generator=g) * std,
            "y_emb.relative_pos": torch.randn(lcfg.t_bins, W, generator=g) * std}


def make_labels(metas, sample_length, lcfg, artist_ids=None, genre_ids=None):
    """Labeller.get_batch_labels (labels.py): y = [total_length, offset, sample_length, artist_id, genre ids padded with
    -1 to max_bow_genre_size, lyric tokens (none for 5b)] per meta; v3 names are lower-cased and unknown names map to 0."""
    artist_ids = artist_ids or {"unknown": 0}
    genre_ids = genre_ids or {"unknown": 0}
    ys = []
    for m in metas:
        a = artist_ids.get(m["artist"].lower(), 0)
        gs = [genre_ids.get(w, 0) for w in [m["genre"].lower()]][: lcfg.max_bow_genre_size]
        gs = gs + [-1] * (lcfg.max_bow_genre_size - len(gs))
        ys.append([int(m["total_length"]), int(m["offset"]), int(sample_length), a, *gs])
    return torch.tensor(ys, dtype=torch.int64)


def get_y(y, start, sample_length, raw_to_tokens):
    """SimplePrior.get_y: level sample length into column 2, offset advanced by start * raw_to_tokens."""
    y = y.clone()
    y[:, 2] = int(sample_length)
    y[:, 1:2] = y[:, 1:2] + int(start * raw_to_tokens)
    return y


def range_bins(pos_start, pos_end, n_time, bins, lo, hi, clamp=False):
    """RangeEmbedding.forward up to the table lookup: fp32 positions interpolated over n_time steps, normalised to
    [lo, hi) and floored into `bins` bins. pos_* float tensors [N,1]."""
    pos_start = pos_start.float()
    if pos_end is not None:
        if clamp:
            pos_end = pos_end.clamp(lo, hi)
        pos_end = pos_end.float()
    if n_time != 1:
        interpolation = torch.arange(0, n_time, dtype=torch.float).view(1, n_time) / n_time
        position = pos_start + (pos_end - pos_start) * interpolation
    else:
        position = pos_start
    normalised = (position - lo) / (hi - lo)
    return (bins * normalised).floor().long()


def label_conditioner(p, y, cfg, lcfg):
    """LabelConditioner.forward(y) -> (start_emb [N,1,W], pos_emb [N,n_ctx,W]) = (y_cond, x_cond) of the top-level prior
    (SimplePrior.get_cond: x_cond = y_pos when the level has no upsampling conditioner)."""
    total_length, offset, length, artist, genre = y[:, 0:1], y[:, 1:2], y[:, 2:3], y[:, 3:4], y[:, 4:]
    artist_emb = p["y_emb.artist"][artist]
    mask = (genre >= 0).float().unsqueeze(2)
    genre_emb = (p["y_emb.genre"][genre.clamp(0)] * mask).sum(dim=1, keepdim=True)
    start_emb = genre_emb + artist_emb
    start, end = offset, offset + length
    total_length, start, end = total_length.float(), start.float(), end.float()
    sr = lcfg.sr
    b_total = range_bins(total_length, None, 1, lcfg.t_bins, lcfg.min_duration * sr, lcfg.max_duration * sr)
    b_abs = range_bins(start, end, cfg.n_ctx, lcfg.t_bins, 0.0, lcfg.max_duration * sr)
    b_rel = range_bins(start / total_length, end / total_length, cfg.n_ctx, lcfg.t_bins, 0.0, 1.0, clamp=True)
    pos_emb = p["y_emb.total_length"][b_total] + p["y_emb.absolute_pos"][b_abs] + p["y_emb.relative_pos"][b_rel]
    return start_emb, pos_emb


def get_cond(p, cfg, lcfg, n_samples=8, artist_ids=None, genre_ids=None):
    """jukebox/main.py:71-98: the fixed metas (artist / genre "unknown", 62 s total, offset 0), n_samples copies, row 0
    kept: -> (x_cond [1, n_ctx, W], y_cond [1, 1, W])."""
    total = (int(62 * JUKEBOX_SAMPLE_RATE) // cfg.hop) * cfg.hop
    metas = [dict(artist="unknown", genre="unknown", total_length=total, offset=0, lyrics="lyrics go here!!!")] * n_samples
    y = get_y(make_labels(metas, cfg.n_ctx * cfg.hop, lcfg, artist_ids, genre_ids), 0, cfg.n_ctx * cfg.hop, cfg.hop)
    y_cond, x_cond = label_conditioner(p, y, cfg, lcfg)
    return x_cond[0, : cfg.n_ctx][None], y_cond[0][None]


# ------------------------------------------------------------------------------------------------ checkpoint names (J7)
def upstream_vqvae_keys(cfg, level=2):
    """[UPSTREAM-RECALLED] state-dict names of vqvae.pth.tar for the level-`level` encoder and codebook ->
    names used here. Encoder(level) = level_blocks[b].model = Sequential(Sequential(Conv1d, Resnet1D)..., Conv1d);
    Resnet1D.model = Sequential(ResConv1DBlock...); ResConv1DBlock.model = Sequential(ReLU, Conv1d k3, ReLU, Conv1d k1)."""
    m = {}
    for b, down_t in enumerate(cfg.downs_t[: level + 1]):
        base = f"encoders.{level}.level_blocks.{b}.model."
        for i in range(down_t):
            for s, t in (("weight", "w"), ("bias", "b")):
                m[f"{base}{i}.0.{s}"] = f"enc.{b}.down.{i}.{t}"
                for d in range(cfg.depth):
                    m[f"{base}{i}.1.model.{d}.model.1.{s}"] = f"enc.{b}.res.{i}.{d}.{t}1"
                    m[f"{base}{i}.1.model.{d}.model.3.{s}"] = f"enc.{b}.res.{i}.{d}.{t}2"
        for s, t in (("weight", "w"), ("bias", "b")):
            m[f"{base}{down_t}.{s}"] = f"enc.{b}.proj.{t}"
    m[f"bottleneck.level_blocks.{level}.k"] = "codebook"
    return m


def upstream_prior_keys(cfg):
    """[UPSTREAM-RECALLED] state-dict names of prior_level_2.pth.tar (SimplePrior: .prior = ConditionalAutoregressive2D,
    .y_emb = LabelConditioner) -> names used here, for the first cfg.prior_depth blocks only: the checkpoint has 72
    blocks, the reference builds 36 and loads non-strictly (jukebox/main.py:197, make_models.py.patch:7-8)."""
    m = {"prior.x_emb.weight": "x_emb", "prior.pos_emb.pos_emb": "pos_emb",
         "y_emb.bow_genre_emb.emb.weight": "y_emb.genre", "y_emb.artist_emb.emb.weight": "y_emb.artist",
         "y_emb.total_length_emb.emb.weight": "y_emb.total_length",
         "y_emb.absolute_pos_emb.emb.weight": "y_emb.absolute_pos",
         "y_emb.relative_pos_emb.emb.weight": "y_emb.relative_pos"}
    for d in range(cfg.prior_depth):
        u, q = f"prior.transformer._attn_mods.{d}.", f"blk.{d}."
        m.update({u + "ln_0.weight": q + "ln0.g", u + "ln_0.bias": q + "ln0.b",
                  u + "attn.c_attn.w": q + "c_attn.w", u + "attn.c_attn.b": q + "c_attn.b",
                  u + "attn.c_proj.w": q + "c_proj.w", u + "attn.c_proj.b": q + "c_proj.b",
                  u + "ln_1.weight": q + "ln1.g", u + "ln_1.bias": q + "ln1.b",
                  u + "mlp.c_fc.w": q + "fc.w", u + "mlp.c_fc.b": q + "fc.b",
                  u + "mlp.c_proj.w": q + "fc_proj.w", u + "mlp.c_proj.b": q + "fc_proj.b"})
    return m
