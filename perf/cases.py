"""The work that is timed when a kernel of this framework changes: listed cases and a generator of more of the same ranges.

Every case goes through an entry point that a user's program calls: the model classes (training step, decoding), the ops of a
training step, the Jukebox front end, and the layers and engine of the generation path. `prepare` makes the inputs and what
such a program keeps (weights, caches), `run` is one pass, `exact` is the same pass restated in 64 bits with plain torch.
"""
import math

import torch
import torch.nn.functional as F

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


# ---------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # The training step of the audio-conditioned model: Llama-2-7B's layer and head sizes, 512 tokens with 240 frames of
        # audio in them, per-GPU batch of 16. One decoder layer stands for the thirty-two equal ones.
        dict(name="train_step", kind="train", width=4096, ff=11008, layers=1, vocab=32004, batch=16, seq=512, frames=240),
        # Causal attention of a training step alone, forward and backward, at the longest context the data loader allows.
        dict(name="attention_train", kind="attention", heads=32, batch=4, seq=2048, masked=True),
        # The Jukebox front end's first half: 24 s waveforms to VQ-VAE codes, fp32.
        dict(name="vqvae_encode", kind="encoder", clips=4, samples=1048576),
        # Its second half: the prior's blocks over 8192 codes per clip. Three blocks: one of each attention pattern.
        dict(name="prior_blocks", kind="prior", clips=2, tokens=8192, blocks=3, precision="bf16"),
        # Answering one question: a decode step of the 7B sizes at batch 1, two layers and the head.
        dict(name="decode_one", kind="decode", width=4096, ff=11008, layers=2, vocab=32004, batch=1, context=1024),
        # Captioning a set of tracks: the same with 32 requests side by side.
        dict(name="decode_batch", kind="decode", width=4096, ff=11008, layers=2, vocab=32004, batch=32, context=1500),
        # Prompts through a gated-linear-recurrence layer, lengths as they come.
        dict(name="hgrn2_prompts", kind="recurrence", type="hgrn2", width=2048, heads=16, requests=4, tokens=2048),
        # Prompts through a gated-delta-rule layer, odd lengths.
        dict(name="delta_prompts", kind="recurrence", type="delta", width=2048, heads=16, requests=3, tokens=1777),
        # Prompts through a sliding-window attention layer with grouped key / value heads.
        dict(name="window_prompts", kind="window", width=4096, heads=32, kv_heads=8, window=1024, requests=4, tokens=2048, context=0),
        # One token each for 32 requests whose rings are full.
        dict(name="window_decode", kind="window", width=4096, heads=32, kv_heads=8, window=1024, requests=32, tokens=1, context=1300),
        # The routed experts of a decode step: few tokens, most experts hit.
        dict(name="experts_decode", kind="moe", width=2048, ff=1024, experts=32, top=4, tokens=32),
        # A whole call of the serving engine: a batch of prompts, then one token per request four times.
        dict(name="serve_small", kind="serve", width=2048, ff=8192, heads=16, window=1024, layers=4, vocab=32000, requests=8,
             prompt=150, steps=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "attention", "encoder", "prior", "decode", "decode", "recurrence", "recurrence", "window", "window",
                       "moe", "moe", "serve"])
    if kind == "train":
        width = rng.choice([512, 1024, 2048, 4096])
        seq = rng.randint(96, 512)
        return dict(kind=kind, width=width, ff={512: 1408, 1024: 2816, 2048: 5504, 4096: 11008}[width], layers=rng.randint(1, 2) if width < 4096 else 1,
                    vocab=rng.choice([32004, 32003, 8192]), batch=_log_int(rng, 1, 16), seq=seq, frames=rng.randint(5, seq // 2))
    if kind == "attention":
        seq = _log_int(rng, 64, 2048)
        return dict(kind=kind, heads=rng.choice([8, 16, 32]), batch=_log_int(rng, 1, max(1, min(32, 8192 // seq))), seq=seq,
                    masked=rng.random() < 0.5)
    if kind == "encoder":
        return dict(kind=kind, clips=rng.randint(1, 4), samples=128 * rng.randint(1024, 8192))
    if kind == "prior":
        precision = rng.choice(["bf16", "bf16", "tf32"])
        return dict(kind=kind, clips=rng.randint(1, 2) if precision == "bf16" else 1, tokens=1024 * rng.randint(2, 8), blocks=3,
                    precision=precision)
    if kind == "decode":
        width = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, width=width, ff={1024: 2816, 2048: 5504, 4096: 11008}[width], layers=2, vocab=rng.choice([32004, 32003, 8192]),
                    batch=_log_int(rng, 1, 48), context=_log_int(rng, 40, 2000))
    if kind == "recurrence":
        heads = rng.choice([8, 16, 32])
        return dict(kind=kind, type=rng.choice(["hgrn2", "delta"]), width=heads * 128, heads=heads, requests=rng.randint(1, 4),
                    tokens=_log_int(rng, 50, 2048))
    if kind == "window":
        heads = rng.choice([8, 16, 32])
        kv = rng.choice([heads // 4, heads // 2, heads])
        common = dict(kind=kind, width=heads * 128, heads=heads, kv_heads=kv, window=rng.choice([512, 1000, 1024, 2048]))
        if rng.random() < 0.5:
            return dict(common, requests=rng.randint(1, 4), tokens=_log_int(rng, 50, 2048), context=0)
        return dict(common, requests=_log_int(rng, 1, 48), tokens=1, context=_log_int(rng, 40, 2000))
    if kind == "moe":
        width = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, width=width, ff=rng.choice([512, 1024]), experts=rng.choice([32, 64]), top=rng.choice([4, 6]),
                    tokens=_log_int(rng, 1, 4096))
    width = rng.choice([1024, 2048])
    return dict(kind=kind, width=width, ff=4 * width, heads=width // 128, window=rng.choice([128, 1024]), layers=4, vocab=32000,
                requests=_log_int(rng, 1, 32), prompt=_log_int(rng, 20, 300), steps=rng.randint(1, 4))


def prepare(case, seed):
    return _KINDS[case["kind"]].prepare(case, seed)


def run(state):
    return state["kind"].run(state)


def work(case):
    return _KINDS[case["kind"]].work(case)


def tolerance(case):
    return _KINDS[case["kind"]].tolerance(case)


def exact(case, seed):
    with torch.no_grad():
        return _KINDS[case["kind"]].exact(case, seed)


# ---------------------------------------------------------------------------------------------------------------- shared parts
class _Random:
    """Seeded tensors on the GPU. Weights are bf16 numbers, as a checkpoint stores them."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        return (mean + std * torch.randn(*shape, generator=self.g, device="cuda")).to(dtype)

    def matrix(self, n_out, n_in, gain=1.0):
        return self.normal(n_out, n_in, std=gain / math.sqrt(n_in))

    def uniform(self, *shape, low=0.0, high=1.0):
        return (low + (high - low) * torch.rand(*shape, generator=self.g, device="cuda")).to(BF16)

    def ints(self, low, high, *shape):
        return torch.randint(low, high, shape, generator=self.g, device="cuda")


def _lens(case):
    """Ragged request lengths: the first is case["tokens"], the others lie between half of it and all of it."""
    n = case["tokens"]
    return [max(1, round(n * (1.0 - 0.5 * ((i * 0.618034) % 1.0)))) for i in range(case["requests"])]


def _rms64(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rope64(x, pos, base, interleaved):
    """x [..., T, heads, D] rotated by pos [T]."""
    D = x.shape[-1]
    f = float(base) ** (-2.0 * torch.arange(D // 2, dtype=F64, device=x.device) / D)
    a = pos.to(F64)[:, None] * f[None]
    c, s = a.cos()[:, None, :], a.sin()[:, None, :]
    if interleaved:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    u, v = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend64(q, k, v, visible, scale):
    """q [T, H, D], k, v [S, H, D], visible bool [T, S] -> [T, H, D]; a few heads at a time."""
    out = torch.empty_like(q)
    for h in range(0, q.shape[1], 4):
        s = torch.einsum("thd,shd->hts", q[:, h:h + 4], k[:, h:h + 4]) * scale
        p = torch.softmax(s.masked_fill(~visible[None], -math.inf), -1)
        out[:, h:h + 4] = torch.einsum("hts,shd->thd", p, v[:, h:h + 4])
    return out


class _Kind:
    pass


# ---------------------------------------------------------------------------------------------------------------- Llama models
_START, _END, _PATCH, _PAD = 1, 2, 3, 4  # marker tokens of the synthetic vocabulary; text starts behind them
_MM = 4800                               # width of a Jukebox frame
_EPS = 1e-5


def _llama_weights(case, r):
    H, I, V = case["width"], case["ff"], case["vocab"]
    w = {"model.embed_tokens.weight": r.normal(V, H, std=0.5), "lm_head.weight": r.normal(V, H, std=1.0 / math.sqrt(H)),
         "model.norm.weight": r.normal(H, mean=1.0, std=0.1), "model.mm_projector.weight": r.matrix(H, _MM),
         "model.mm_projector.bias": r.normal(H, std=0.02)}
    for l in range(case["layers"]):
        p = f"model.layers.{l}."
        for n in "qkvo":
            w[p + f"self_attn.{n}_proj.weight"] = r.matrix(H, H, 0.7)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = r.matrix(I, H, 0.7), r.matrix(I, H, 0.7)
        w[p + "mlp.down_proj.weight"] = r.matrix(H, I, 0.7)
        w[p + "input_layernorm.weight"] = r.normal(H, mean=1.0, std=0.1)
        w[p + "post_attention_layernorm.weight"] = r.normal(H, mean=1.0, std=0.1)
    return w


def _llama_model(case, r):
    from llark_b200.models.llamav2 import WrappedLlamav2Config, WrappedLlamav2ForCausalLM

    hf = WrappedLlamav2Config(hidden_size=case["width"], intermediate_size=case["ff"], num_hidden_layers=case["layers"],
                              num_attention_heads=case["width"] // 128, num_key_value_heads=case["width"] // 128,
                              vocab_size=case["vocab"], max_position_embeddings=2048, rms_norm_eps=_EPS)
    hf.mm_hidden_size = _MM
    old = torch.get_default_dtype()
    torch.set_default_dtype(BF16)
    try:
        with torch.device("cuda"):
            model = WrappedLlamav2ForCausalLM(hf)
            model.get_model().initialize_adapter_modules()
    finally:
        torch.set_default_dtype(old)
    model.to(BF16)
    weights = _llama_weights(case, r)
    with torch.no_grad():
        for n, p in model.named_parameters():
            p.copy_(weights[n])
    aec = model.get_model().audio_encoder_config
    aec.use_audio_start_end = True
    aec.audio_start_token, aec.audio_end_token, aec.audio_patch_token = _START, _END, _PATCH
    # what the training script trains: everything but the head, and of the token table only the marker rows
    for p in model.get_output_embeddings().parameters():
        p.requires_grad = False
    model.get_model().orig_embeds_params = [None]
    model.validate = "lazy"
    return model


def _llama_layer64(w, l, x, pos, visible, heads):
    """One decoder layer on x [T, H]; returns (x, keys, values)."""
    p = f"model.layers.{l}."
    T, H = x.shape
    h = _rms64(x, w[p + "input_layernorm.weight"], _EPS)
    q, k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"].t()).view(T, heads, -1) for n in "qkv")
    q, k = _rope64(q, pos, 10000.0, False), _rope64(k, pos, 10000.0, False)
    s = torch.einsum("thd,shd->hts", q, k) / math.sqrt(q.shape[-1])
    o = torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(~visible, -math.inf), -1), v)
    x = x + o.reshape(T, H) @ w[p + "self_attn.o_proj.weight"].t()
    h = _rms64(x, w[p + "post_attention_layernorm.weight"], _EPS)
    h = F.silu(h @ w[p + "mlp.gate_proj.weight"].t()) * (h @ w[p + "mlp.up_proj.weight"].t())
    return x + h @ w[p + "mlp.down_proj.weight"].t(), k, v


def _llama_matrix_weights(case):
    H, I = case["width"], case["ff"]
    return case["layers"] * (4 * H * H + 3 * H * I)


class _Train(_Kind):
    """Forward and backward of the training step: loss, logits and every gradient."""

    @staticmethod
    def _batch(case, r):
        B, S, n = case["batch"], case["seq"], case["frames"]
        ids = r.ints(_PAD + 1, case["vocab"], B, S)
        labels = ids.clone()
        for b in range(B):
            at = 1 + (7 * b) % max(1, S - n - 3)
            ids[b, at], ids[b, at + n + 1] = _START, _END
            ids[b, at + 1:at + n + 1] = _PATCH
            labels[b, :at + n + 2] = -100
            if b % 3 == 1:  # padded on the right, as the collator does
                pad = min(S // 8, S - at - n - 3)
                if pad > 0:
                    ids[b, S - pad:], labels[b, S - pad:] = _PAD, -100
        labels[0, S - 1] = ids[0, S - 1] = _PAD + 1
        return dict(input_ids=ids, attention_mask=ids.ne(_PAD), labels=labels, audio_encodings=r.normal(B, n, _MM, dtype=F32))

    @staticmethod
    def prepare(case, seed):
        r = _Random(seed)
        model = _llama_model(case, r)
        return dict(kind=_Train, model=model, batch=_Train._batch(case, r))

    @staticmethod
    def run(s):
        model = s["model"]
        model.zero_grad(set_to_none=True)
        out = model(**s["batch"])
        out.loss.backward()
        return dict(loss=out.loss, logits=out.logits, grads={n: p.grad for n, p in model.named_parameters() if p.requires_grad})

    @staticmethod
    def work(case):
        M, H, V, S = case["batch"] * case["seq"], case["width"], case["vocab"], case["seq"]
        w = _llama_matrix_weights(case)
        flops = 6.0 * M * w + 4.0 * M * H * V + case["layers"] * 3.5 * 4.0 * M * H * (S + 1) / 2
        flops += 4.0 * case["batch"] * case["frames"] * _MM * H
        return dict(bytes=2.0 * (2 * w + 2 * V * H + 2 * _MM * H) + 2.0 * M * V + 4.0 * case["batch"] * case["frames"] * _MM, flops=flops)

    @staticmethod
    def tolerance(case):
        return {"rel": 3e-2}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w = {n: t.to(F64) for n, t in _llama_weights(case, r).items()}
        bt = _Train._batch(case, r)
        train = [n for n in w if n != "lm_head.weight"]
        grads = {n: torch.zeros_like(w[n]) for n in train}
        ids, heads = bt["input_ids"], case["width"] // 128
        B, S = ids.shape
        pos = torch.arange(S, device="cuda")
        causal = pos[None] <= pos[:, None]
        count = (bt["labels"][:, 1:] != -100).sum()
        logits, loss = [], 0.0
        for b in range(B):  # one sample at a time: the loss is a sum over them
            with torch.enable_grad():
                p = {n: t.detach().requires_grad_(n in grads) for n, t in w.items()}
                e = p["model.embed_tokens.weight"][ids[b]]
                marker = (ids[b] == _START) | (ids[b] == _END)
                e = torch.where(marker[:, None], e, e.detach())
                at = int((ids[b] == _START).nonzero()[0])
                n = case["frames"]
                feat = bt["audio_encodings"][b].to(BF16).to(F64) @ p["model.mm_projector.weight"].t() + p["model.mm_projector.bias"]
                x = torch.cat([e[:at + 1], feat, e[at + n + 1:]])
                vis = causal & bt["attention_mask"][b][None]
                for l in range(case["layers"]):
                    x, _, _ = _llama_layer64(p, l, x, pos, vis, heads)
                z = _rms64(x, p["model.norm.weight"], _EPS) @ p["lm_head.weight"].t()
                part = F.cross_entropy(z[:-1], bt["labels"][b, 1:], ignore_index=-100, reduction="sum") / count
                got = torch.autograd.grad(part, [p[n] for n in train])
            for n, g in zip(train, got):
                grads[n] += g
            logits.append(z.detach().to(F32))
            loss = loss + part.detach()
        return dict(loss=loss, logits=torch.stack(logits), grads=grads)


class _Decode(_Kind):
    """One token per request against the KV cache: logits, and the keys and values that the step adds."""

    @staticmethod
    def _ids(case, r):
        return r.ints(_PAD + 1, case["vocab"], case["batch"], case["context"] + 1)

    @staticmethod
    def prepare(case, seed):
        r = _Random(seed)
        model = _llama_model(case, r).eval()
        ids = _Decode._ids(case, r)
        n = case["context"]
        with torch.no_grad():
            cache = None
            for b in range(0, case["batch"], 8):  # prompts eight at a time: their logits are large
                out = model(input_ids=ids[b:b + 8, :n], use_cache=True)
                part = out.past_key_values
                if case["batch"] <= 8:
                    cache = part
                    break
                if cache is None:
                    cache = model.engine.new_cache(case["batch"], part.s_max, ids.device)
                for l in range(case["layers"]):
                    cache.k[l][b:b + 8].copy_(part.k[l])
                    cache.v[l][b:b + 8].copy_(part.v[l])
                del out, part
            cache.length = n
        return dict(kind=_Decode, model=model, cache=cache, last=ids[:, n:].contiguous(), context=n)

    @staticmethod
    def run(s):
        cache, n = s["cache"], s["context"]
        cache.length = n  # the same step again: its keys and values go to the same place
        with torch.no_grad():
            out = s["model"](input_ids=s["last"], past_key_values=cache, use_cache=True)
        return dict(logits=out.logits, keys=[k[:, n] for k in cache.k], values=[v[:, n] for v in cache.v])

    @staticmethod
    def work(case):
        B, n, H = case["batch"], case["context"], case["width"]
        w = _llama_matrix_weights(case) + case["vocab"] * H
        return dict(bytes=2.0 * w + case["layers"] * 4.0 * B * (n + 1) * H + 2.0 * B * case["vocab"],
                    flops=2.0 * B * w + case["layers"] * 4.0 * B * (n + 1) * H)

    @staticmethod
    def tolerance(case):
        return {"rel": 2e-2}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w = {n: t.to(F64) for n, t in _llama_weights(case, r).items()}
        ids = _Decode._ids(case, r)
        heads, T = case["width"] // 128, case["context"] + 1
        pos = torch.arange(T, device="cuda")
        causal = pos[None] <= pos[:, None]
        logits, keys, values = [], [[] for _ in range(case["layers"])], [[] for _ in range(case["layers"])]
        for b in range(case["batch"]):
            x = w["model.embed_tokens.weight"][ids[b]]
            for l in range(case["layers"]):
                x, k, v = _llama_layer64(w, l, x, pos, causal, heads)
                keys[l].append(k[-1].reshape(-1))
                values[l].append(v[-1].reshape(-1))
            logits.append(_rms64(x[-1:], w["model.norm.weight"], _EPS) @ w["lm_head.weight"].t())
        return dict(logits=torch.stack(logits), keys=[torch.stack(k) for k in keys], values=[torch.stack(v) for v in values])


class _Attention(_Kind):
    """Causal attention of a training step on the packed projection, forward and backward; masked: right-padded samples."""

    @staticmethod
    def _inputs(case, seed):
        r = _Random(seed)
        M, H = case["batch"] * case["seq"], case["heads"] * 128
        qkv, dout = r.normal(M, 3 * H), r.normal(M, H, std=0.1)
        mask = None
        if case["masked"]:
            pad = torch.tensor([(b * case["seq"]) // (4 * case["batch"]) for b in range(case["batch"])], device="cuda")
            mask = (torch.arange(case["seq"], device="cuda")[None] < (case["seq"] - pad)[:, None]).to(torch.uint8).contiguous()
        return qkv, dout, mask

    @staticmethod
    def prepare(case, seed):
        qkv, dout, mask = _Attention._inputs(case, seed)
        return dict(kind=_Attention, case=case, qkv=qkv, dout=dout, mask=mask)

    @staticmethod
    def run(s):
        from llark_b200 import ops

        c = s["case"]
        out, lse = ops.attn_fwd(s["qkv"], s["mask"], c["batch"], c["seq"], c["heads"], 128)
        dqkv = ops.attn_bwd(s["qkv"], s["mask"], out, s["dout"], lse, c["batch"], c["seq"], c["heads"], 128)
        return out, dqkv

    @staticmethod
    def work(case):
        M, H, S = case["batch"] * case["seq"], case["heads"] * 128, case["seq"]
        return dict(bytes=2.0 * M * H * (3 + 1 + 1 + 3), flops=3.5 * 4.0 * M * H * (S + 1) / 2)

    @staticmethod
    def tolerance(case):
        return {"rel": 1e-2}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        qkv, dout, mask = _Attention._inputs(case, seed)
        B, S, NH = case["batch"], case["seq"], case["heads"]
        pos = torch.arange(S, device="cuda")
        causal = pos[None] <= pos[:, None]
        out, grad = [], []
        for b in range(B):
            x = qkv.view(B, S, 3, NH, 128)[b].to(F64)
            d = dout.view(B, S, NH, 128)[b].to(F64)
            vis = causal if mask is None else causal & mask[b].bool()[None]
            with torch.enable_grad():
                leaf = x.detach().requires_grad_(True)
                s = torch.einsum("thd,shd->hts", leaf[:, 0], leaf[:, 1]) / math.sqrt(128.0)
                o = torch.einsum("hts,shd->thd", torch.softmax(s.masked_fill(~vis, -math.inf), -1), leaf[:, 2])
                g, = torch.autograd.grad(o, leaf, d)
            out.append(o.detach().reshape(S, -1))
            grad.append(g.reshape(S, -1))
        return torch.cat(out), torch.cat(grad)


# ---------------------------------------------------------------------------------------------------------------- Jukebox
class _Encoder(_Kind):
    """Waveforms to latents (fp32 convolutions) and codes (nearest entry of the codebook)."""
    downs, dilations = (3, 2, 2), (1, 3, 9, 27)

    @staticmethod
    def _weights(r):
        st, c_in = {}, 1
        n = lambda *s, std: r.normal(*s, std=std, dtype=F32)  # noqa: E731
        for b, down in enumerate(_Encoder.downs):
            for i in range(down):
                cin = c_in if i == 0 else 32
                st[f"enc.{b}.down.{i}.w"], st[f"enc.{b}.down.{i}.b"] = n(32, cin, 4, std=(4 * cin) ** -0.5), n(32, std=0.02)
                for d in range(4):
                    q = f"enc.{b}.res.{i}.{d}."
                    st[q + "w1"], st[q + "b1"] = n(32, 32, 3, std=96 ** -0.5), n(32, std=0.02)
                    st[q + "w2"], st[q + "b2"] = n(32, 32, 1, std=32 ** -0.5), n(32, std=0.02)
            st[f"enc.{b}.proj.w"], st[f"enc.{b}.proj.b"] = n(64, 32, 3, std=96 ** -0.5), n(64, std=0.02)
            c_in = 64
        st["codebook"] = n(2048, 64, std=1.0)
        return st

    @staticmethod
    def _wave(case, r):
        t = torch.arange(case["samples"], device="cuda", dtype=F32) / 44100.0
        f = r.normal(case["clips"], 1, std=80.0, mean=330.0, dtype=F32)
        return (0.5 * torch.sin(2 * math.pi * f * t[None]) + r.normal(case["clips"], case["samples"], std=0.2, dtype=F32))[:, None].contiguous()

    @staticmethod
    def prepare(case, seed):
        from llark_b200.jukebox.model import JukeboxConfig, JukeboxVQVAE

        r = _Random(seed)
        vq = JukeboxVQVAE(JukeboxConfig(sample_length=case["samples"]), _Encoder._weights(r), "cuda")
        return dict(kind=_Encoder, vq=vq, wave=_Encoder._wave(case, r))

    @staticmethod
    def run(s):
        from llark_b200 import ops

        latents = s["vq"].encode_top_latents(s["wave"])
        return latents, ops.jb_vq_encode(latents, s["vq"].w["codebook"])

    @staticmethod
    def work(case):
        n, T = case["clips"], case["samples"]
        flops, moved, c_in = 0.0, 4.0 * n * T, 1
        for down in _Encoder.downs:
            for i in range(down):
                T //= 2
                flops += 2.0 * n * T * 32 * 4 * (c_in if i == 0 else 32) + 4 * 2.0 * n * T * 32 * 32 * 4
            flops += 2.0 * n * T * 64 * 32 * 3
            c_in = 64
        return dict(bytes=moved + n * T * (64 * 4.0 + 8), flops=flops + 2.0 * n * T * 64 * 2048)

    @staticmethod
    def tolerance(case):
        return {"rel": 2e-5, "differ": 1e-3}  # four times the error seen against exact(); codes: near-ties

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w = {k: v.to(F64) for k, v in _Encoder._weights(r).items()}

        def conv(x, k, b, stride=1, dilation=1, pad=0):  # few channels: a sum over taps of matrix products
            x = F.pad(x, (pad, pad))
            n = (x.shape[-1] - dilation * (k.shape[2] - 1) - 1) // stride + 1
            y = b[:, None]
            for j in range(k.shape[2]):
                y = y + k[:, :, j] @ x[:, j * dilation:j * dilation + (n - 1) * stride + 1:stride]
            return y

        latents, codes = [], []
        for h in _Encoder._wave(case, r).to(F64):
            for b, down in enumerate(_Encoder.downs):
                for i in range(down):
                    h = conv(h, w[f"enc.{b}.down.{i}.w"], w[f"enc.{b}.down.{i}.b"], stride=2, pad=1)
                    for d, dil in enumerate(_Encoder.dilations):
                        q = f"enc.{b}.res.{i}.{d}."
                        u = conv(h.clamp(min=0), w[q + "w1"], w[q + "b1"], dilation=dil, pad=dil)
                        h = h + conv(u.clamp(min=0), w[q + "w2"], w[q + "b2"])
                h = conv(h, w[f"enc.{b}.proj.w"], w[f"enc.{b}.proj.b"], pad=1)
            latents.append(h)
            k = w["codebook"]
            codes.append((k.square().sum(1)[None] - 2 * h.t() @ k.t()).argmin(1))
        return torch.stack(latents), torch.stack(codes)


class _Prior(_Kind):
    """Codes to activations of the prior's first blocks (layer norm, factored attention, quick-GELU feed-forward)."""
    W, A, heads = 4800, 1200, 8

    @staticmethod
    def _weights(case, r):
        W, A = _Prior.W, _Prior.A
        n = lambda *s, std, mean=0.0: r.normal(*s, std=std, mean=mean, dtype=F32)  # noqa: E731
        st = {"x_emb": n(2048, W, std=0.02), "pos_emb": n(8192, W, std=0.01), "x_cond": n(8192, W, std=0.01), "y_cond": n(W, std=0.02)}
        for d in range(case["blocks"]):
            q = f"blk.{d}."
            for ln in ("ln0", "ln1"):
                st[q + ln + ".g"], st[q + ln + ".b"] = n(W, mean=1.0, std=0.1), n(W, std=0.02)
            for name, i, o, gain in (("c_attn", W, 3 * A, 0.7), ("c_proj", A, W, 0.3), ("fc", W, W, 0.7), ("fc_proj", W, W, 0.3)):
                st[q + name + ".w"] = n(i, o, std=gain / math.sqrt(i)).to(BF16).to(F32)
                st[q + name + ".b"] = n(o, std=0.02)
        return st

    @staticmethod
    def prepare(case, seed):
        from llark_b200.jukebox.model import JukeboxConfig, PriorTransformer

        r = _Random(seed)
        prior = PriorTransformer(JukeboxConfig(prior_depth=case["blocks"]), _Prior._weights(case, r), "cuda", case["precision"])
        prior.only_encode = True
        return dict(kind=_Prior, prior=prior, codes=r.ints(0, 2048, case["clips"], case["tokens"]))

    @staticmethod
    def run(s):
        return s["prior"].forward(s["codes"])

    @staticmethod
    def work(case):
        W, A, T = _Prior.W, _Prior.A, case["tokens"]
        M, w = case["clips"] * T, W * 3 * A + A * W + 2 * W * W
        keys = (T // 128 + 1) / 2 + 129 / 2 + T // 128  # of the three patterns
        return dict(bytes=case["blocks"] * w * (2.0 if case["precision"] == "bf16" else 4.0) + 4.0 * M * W,
                    flops=case["blocks"] * (2.0 * M * w + 4.0 * M * A * keys / 3))

    @staticmethod
    def tolerance(case):
        return {"rel": 1.2e-2 if case["precision"] == "bf16" else 4e-3}

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w = {k: v.to(F64) for k, v in _Prior._weights(case, r).items()}
        codes = r.ints(0, 2048, case["clips"], case["tokens"])
        T, W, A, nh = case["tokens"], _Prior.W, _Prior.A, _Prior.heads
        nb, bc, dh = 128, T // 128, A // nh

        def norm(x, q):
            return F.layer_norm(x, (W,), w[q + ".g"], w[q + ".b"], 1e-5)

        def dense(q, k, v, causal):
            s = q @ k.transpose(-1, -2) / math.sqrt(dh)
            if causal:
                n = s.shape[-1]
                s = s.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=s.device).tril(), -math.inf)
            return torch.softmax(s, -1) @ v

        out = []
        for c in codes:
            x = torch.cat([w["y_cond"][None], w["x_emb"][c][:-1]]) + w["pos_emb"][:T] + w["x_cond"][:T]
            for d in range(case["blocks"]):
                p = f"blk.{d}."
                qkv = norm(x, p + "ln0") @ w[p + "c_attn.w"] + w[p + "c_attn.b"]
                q, k, v = (t.view(nb, bc, nh, dh) for t in qkv.chunk(3, 1))
                if d % 3 == 0:    # causal inside a block
                    a = dense(*(t.permute(0, 2, 1, 3) for t in (q, k, v)), True).permute(0, 2, 1, 3)
                elif d % 3 == 1:  # causal over the blocks, same place in each
                    a = dense(*(t.permute(1, 2, 0, 3) for t in (q, k, v)), True).permute(2, 0, 1, 3)
                else:             # everything in the block before; the first block sees zeros
                    k, v = (F.pad(t[:-1], (0, 0, 0, 0, 0, 0, 1, 0)) for t in (k, v))
                    a = dense(*(t.permute(0, 2, 1, 3) for t in (q, k, v)), False).permute(0, 2, 1, 3)
                x = x + a.reshape(T, A) @ w[p + "c_proj.w"] + w[p + "c_proj.b"]
                h = norm(x, p + "ln1") @ w[p + "fc.w"] + w[p + "fc.b"]
                x = x + (h * torch.sigmoid(1.702 * h)) @ w[p + "fc_proj.w"] + w[p + "fc_proj.b"]
            out.append(x.to(F32))
        return torch.stack(out)


# ---------------------------------------------------------------------------------------------------------------- generation path
def _conv64(x, w):
    """Causal depthwise convolution over time: x [T, C], w [C, taps]."""
    y = torch.zeros_like(x)
    for j in range(w.shape[1]):
        back = w.shape[1] - 1 - j
        if back < x.shape[0]:
            y[back:] += w[:, j] * x[:x.shape[0] - back]
    return y


def _hgrn2_weights(r, width, heads):
    D = 128
    n = heads * D
    return {"q": r.matrix(n, width), "f": r.matrix(n, width), "v": r.matrix(n, width), "f.b": r.normal(n, mean=1.0, std=1.0),
            "lower": r.uniform(n, low=0.0, high=0.95), "norm": r.normal(D, mean=1.0, std=0.1), "o": r.matrix(width, n)}


def _hgrn2_64(w, xs, heads, eps):
    """xs: list of [T, width], one per request -> (outputs [sum T, width], states [requests, heads, D, E])."""
    D = 128
    lens = [x.shape[0] for x in xs]
    x = torch.nn.utils.rnn.pad_sequence(xs, batch_first=True)  # [B, T, width]
    B, T, _ = x.shape
    q = F.silu(x @ w["q"].t()).view(B, T, heads, D)
    f = (w["lower"] + (1 - w["lower"]) * torch.sigmoid(x @ w["f"].t() + w["f.b"])).view(B, T, heads, D)
    v = (x @ w["v"].t()).view(B, T, heads, D)
    live = torch.arange(T, device="cuda")[None] < torch.tensor(lens, device="cuda")[:, None]
    f = torch.where(live[:, :, None, None], f, 1.0)  # past its end a request's state stands still
    S, o = torch.zeros(B, heads, D, D, dtype=F64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        S.mul_(f[:, t, :, :, None]).addcmul_((1 - f[:, t])[:, :, :, None], v[:, t][:, :, None, :])
        o[:, t] = torch.matmul(q[:, t][:, :, None, :], S)[:, :, 0]
    y = _rms64(o, w["norm"], eps).reshape(B, T, -1) @ w["o"].t()
    return torch.cat([y[b, :n] for b, n in enumerate(lens)]), S


class _Recurrence(_Kind):
    """Prompts through one recurrent layer of the generation path: its outputs and the states it leaves."""
    eps = 1e-5

    @staticmethod
    def _weights(case, r):
        width, heads, D = case["width"], case["heads"], 128
        if case["type"] == "hgrn2":
            return _hgrn2_weights(r, width, heads), dict(heads=heads, dim=D, vdim=D)
        n = heads * D
        w = {k: r.matrix(n, width) for k in "qkvg"}
        w.update({k + ".conv": r.normal(n, 4, std=0.5) for k in "qkv"})
        w.update({"b": r.matrix(heads, width), "a": r.matrix(heads, width), "A_log": r.normal(heads, mean=-1.0, std=0.5),
                  "dt_bias": r.normal(heads, mean=-1.0, std=1.0), "norm": r.normal(D, mean=1.0, std=0.1), "o": r.matrix(width, n)})
        return w, dict(heads=heads, kv_heads=heads, dim=D, vdim=D)

    @staticmethod
    def prepare(case, seed):
        from llark_b200.mixers import MIXERS
        from llark_b200.state_cache import StateCache

        r = _Random(seed)
        w, spec = _Recurrence._weights(case, r)
        cls = MIXERS[case["type"]]
        cache = StateCache("cuda", n_slots=case["requests"])
        mixer = cls(cls.Weights(w, "", spec, case["width"], torch.device("cuda"), BF16), cache, _Recurrence.eps, BF16, 4096)
        lens = _lens(case)
        return dict(kind=_Recurrence, cache=cache, mixer=mixer, lens=lens, x=r.normal(sum(lens), case["width"]))

    @staticmethod
    def run(s):
        cache = s["cache"]
        slots = [cache.alloc() for _ in s["lens"]]
        y = s["mixer"].forward(s["x"], cache.layout(slots, s["lens"]), cache)
        for slot in reversed(slots):
            cache.release(slot)
        return y, cache.view(s["mixer"].h_state)

    @staticmethod
    def work(case):
        n, H, W, D = sum(_lens(case)), case["heads"], case["width"], 128
        w = 4 * W * H * D if case["type"] == "hgrn2" else 5 * W * H * D + 2 * W * H
        return dict(bytes=2.0 * w + 2.0 * n * W + 4.0 * n * W + 4.0 * case["requests"] * H * D * D,
                    flops=2.0 * n * w + (5.0 if case["type"] == "hgrn2" else 9.0) * n * H * D * D)

    @staticmethod
    def tolerance(case):
        return {"rel": 8e-3}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w, _ = _Recurrence._weights(case, r)
        w = {k: v.to(F64) for k, v in w.items()}
        lens, H, D = _lens(case), case["heads"], 128
        xs = list(r.normal(sum(lens), case["width"]).to(F64).split(lens))
        if case["type"] == "hgrn2":
            return _hgrn2_64(w, xs, H, _Recurrence.eps)
        pad = torch.nn.utils.rnn.pad_sequence
        q, k, v = (pad([F.silu(_conv64(x @ w[n].t(), w[n + ".conv"])) for x in xs], batch_first=True) for n in "qkv")
        x = pad(xs, batch_first=True)
        B, T, _ = x.shape
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k, v = unit(q.view(B, T, H, D)) / math.sqrt(D), unit(k.view(B, T, H, D)), v.view(B, T, H, D)
        beta = torch.sigmoid(x @ w["b"].t())
        g = torch.exp(-torch.exp(w["A_log"]) * F.softplus(x @ w["a"].t() + w["dt_bias"]))
        live = (torch.arange(T, device="cuda")[None] < torch.tensor(lens, device="cuda")[:, None])[:, :, None]
        beta, g = torch.where(live, beta, 0.0), torch.where(live, g, 1.0)
        S, o = torch.zeros(B, H, D, D, dtype=F64, device="cuda"), torch.empty_like(v)
        for t in range(T):
            S.mul_(g[:, t, :, None, None])
            u = beta[:, t, :, None] * (v[:, t] - torch.matmul(k[:, t][:, :, None], S)[:, :, 0])
            S.addcmul_(k[:, t][..., None], u[:, :, None])
            o[:, t] = torch.matmul(q[:, t][:, :, None], S)[:, :, 0]
        y = _rms64(o, w["norm"], _Recurrence.eps) * F.silu((x @ w["g"].t()).view(B, T, H, D))
        y = y.reshape(B, T, -1) @ w["o"].t()
        return torch.cat([y[b, :n] for b, n in enumerate(lens)]), S


class _Window(_Kind):
    """Rotary sliding-window attention with grouped key / value heads: whole prompts (context 0), or the next token of
    requests that hold `context` tokens."""

    @staticmethod
    def _weights(case, r):
        W, H, G = case["width"], case["heads"], case["kv_heads"]
        return {"q": r.matrix(H * 128, W), "k": r.matrix(G * 128, W), "v": r.matrix(G * 128, W), "o": r.matrix(W, H * 128)}

    @staticmethod
    def _inputs(case, r):
        lens = _lens(case) if case["context"] == 0 else [case["tokens"]] * case["requests"]
        past = r.normal(case["requests"], case["context"], case["width"])
        return lens, past, r.normal(sum(lens), case["width"])

    @staticmethod
    def prepare(case, seed):
        from llark_b200.mixers import MIXERS
        from llark_b200.state_cache import StateCache

        r = _Random(seed)
        w = _Window._weights(case, r)
        spec = dict(heads=case["heads"], kv_heads=case["kv_heads"], dim=128, vdim=128, scale=128 ** -0.5,
                    mask=dict(size=case["window"]), rot=dict(base=10000.0, dims=128))
        cls = MIXERS["rotary_attention_window"]
        cache = StateCache("cuda", n_slots=case["requests"])
        mixer = cls(cls.Weights(w, "", spec, case["width"], torch.device("cuda"), BF16), cache, 1e-5, BF16, 4096)
        lens, past, x = _Window._inputs(case, r)
        slots = []
        if case["context"]:  # bring the requests to where they are
            slots = [cache.alloc() for _ in lens]
            for slot, p in zip(slots, past):
                mixer.forward(p, cache.layout([slot], [case["context"]]), cache)
                cache.advance([slot], [case["context"]])
        return dict(kind=_Window, cache=cache, mixer=mixer, lens=lens, slots=slots, x=x)

    @staticmethod
    def run(s):
        cache, slots = s["cache"], s["slots"]
        if slots:
            return s["mixer"].forward(s["x"], cache.layout(slots, s["lens"]), cache)
        slots = [cache.alloc() for _ in s["lens"]]
        y = s["mixer"].forward(s["x"], cache.layout(slots, s["lens"]), cache)
        for slot in reversed(slots):
            cache.release(slot)
        return y

    @staticmethod
    def work(case):
        W, H, G, win, n0 = case["width"], case["heads"], case["kv_heads"], case["window"], case["context"]
        lens = _lens(case) if n0 == 0 else [case["tokens"]] * case["requests"]
        n, w = sum(lens), 2 * W * (H + G) * 128
        keys = sum(min(win, n0 + i + 1) for ln in lens for i in range(ln))
        old = sum(min(n0, win) for _ in lens)
        return dict(bytes=2.0 * w + 6.0 * n * W + 4.0 * (old + n) * G * 128, flops=2.0 * n * w + 4.0 * keys * H * 128)

    @staticmethod
    def tolerance(case):
        return {"rel": 1.4e-2}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w = {k: v.to(F64) for k, v in _Window._weights(case, r).items()}
        lens, past, x = _Window._inputs(case, r)
        H, G, n0 = case["heads"], case["kv_heads"], case["context"]
        out = []
        for p, new in zip(past, x.split(lens)):
            h = torch.cat([p, new]).to(F64)
            T = h.shape[0]
            pos = torch.arange(T, device="cuda")
            q, k, v = ((h @ w[n].t()).view(T, -1, 128) for n in "qkv")
            q, k = _rope64(q, pos, 10000.0, True)[n0:], _rope64(k, pos, 10000.0, True)
            k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
            back = pos[n0:, None] - pos[None]
            o = _attend64(q, k, v, (back >= 0) & (back < case["window"]), 128 ** -0.5)
            out.append(o.reshape(T - n0, -1) @ w["o"].t())
        return torch.cat(out)


class _Experts(_Kind):
    """A routed mixture of experts with the residual sum: x + (y + sum of the chosen experts)."""
    groups, keep, scale = 8, 4, 2.5

    @staticmethod
    def _weights(case, r):
        W, n, f = case["width"], case["experts"], case["ff"]
        return {"router": r.matrix(n, W, 1.5), "gate": r.normal(n, f, W, std=W ** -0.5), "up": r.normal(n, f, W, std=W ** -0.5),
                "down": r.normal(n, W, f, std=f ** -0.5)}

    @staticmethod
    def _inputs(case, r):
        n, W = case["tokens"], case["width"]
        return r.normal(n, W, dtype=F32), r.normal(n, W, dtype=F32), r.normal(n, W)

    @staticmethod
    def prepare(case, seed):
        from llark_b200.mixers import FEED_FORWARDS

        r = _Random(seed)
        w = _Experts._weights(case, r)
        named = {"router": w["router"]}
        for e in range(case["experts"]):
            named.update({f"e{e}.{n}": w[n][e] for n in ("gate", "up", "down")})
        spec = dict(router=dict(experts=case["experts"], top=case["top"], scale=_Experts.scale,
                                groups=dict(count=_Experts.groups, keep=_Experts.keep)), expert=dict(ff=case["ff"]))
        cls = FEED_FORWARDS["moe"]
        ff = cls(cls.Weights(named, "", spec, case["width"], torch.device("cuda"), BF16), BF16)
        x, y, x_act = _Experts._inputs(case, r)
        return dict(kind=_Experts, ff=ff, x=x, y=y, x_act=x_act)

    @staticmethod
    def run(s):
        return s["ff"].residual(s["x"], s["y"], s["x_act"])

    @staticmethod
    def work(case):
        n, W, f = case["tokens"], case["width"], case["ff"]
        hit = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** n)
        return dict(bytes=hit * 3 * W * f * 2.0 + n * W * 14.0, flops=n * case["top"] * 6.0 * W * f)

    @staticmethod
    def tolerance(case):
        return {"rel": 4e-3}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        r = _Random(seed)
        w = {k: v.to(F64) for k, v in _Experts._weights(case, r).items()}
        x, y, h = (t.to(F64) for t in _Experts._inputs(case, r))
        n, per = case["experts"], case["experts"] // _Experts.groups
        score = torch.sigmoid(h @ w["router"].t())
        by_group = score.view(-1, _Experts.groups, per)
        best = by_group.topk(min(2, per), -1).values.sum(-1).topk(_Experts.keep, -1).indices
        kept = torch.zeros(score.shape[0], _Experts.groups, dtype=torch.bool, device="cuda").scatter_(1, best, True)
        choice = by_group.masked_fill(~kept[:, :, None], -math.inf).view(-1, n).topk(case["top"], -1).indices
        wt = score.gather(1, choice)
        wt = wt / wt.sum(-1, keepdim=True) * _Experts.scale
        out = x + y
        for e in range(n):
            at, k = (choice == e).nonzero(as_tuple=True)
            if at.numel():
                u = h[at]
                z = (F.silu(u @ w["gate"][e].t()) * (u @ w["up"][e].t())) @ w["down"][e].t()
                out.index_add_(0, at, z * wt[at, k][:, None])
        return out


class _Serve(_Kind):
    """Whole calls of the serving engine: a packed batch of prompts, then single tokens; logits of every step."""
    eps = 1e-5

    @staticmethod
    def _config(case):
        layers = []
        for i in range(case["layers"]):
            if i % 4 == 3:
                layers.append(dict(type="attention", mixer=dict(heads=case["heads"], kv_heads=case["heads"], dim=128, vdim=128,
                                                                mask=dict(size=case["window"]), scale=128 ** -0.5),
                                   mlp=dict(kind="dense", ff=case["ff"])))
            else:
                layers.append(dict(type="hgrn2", mixer=dict(heads=case["heads"], dim=128, vdim=128), mlp=None))
        return dict(architecture="Kelutar", vocab=case["vocab"], width=case["width"], max_positions=1024,
                    embedding=dict(scale=math.sqrt(case["width"])), norm=dict(eps=_Serve.eps), canon=dict(taps=4), layers=layers)

    @staticmethod
    def _weights(case, r):
        C, n = case["width"], case["heads"] * 128
        w = {"embed": r.matrix(case["vocab"], C), "pos": r.matrix(1024, C, 0.5 * math.sqrt(C)),
             "final.norm": r.normal(C, mean=1.0, std=0.1), "head": r.matrix(case["vocab"], C)}
        for i in range(case["layers"]):
            p = f"l{i}."
            w[p + "norm1"], w[p + "canon1"] = r.normal(C, mean=1.0, std=0.1), r.normal(C, 4, std=0.3)
            if i % 4 == 3:
                w.update({p + "mix." + k: r.matrix(n, C) for k in "qkg"})
                w.update({p + "mix.q.b": r.normal(n, std=0.1), p + "mix.k.b": r.normal(n, std=0.1), p + "mix.o": r.matrix(C, n),
                          p + "mix.q.norm": r.normal(128, mean=1.0, std=0.1), p + "mix.k.norm": r.normal(128, mean=1.0, std=0.1),
                          p + "mix.temp": r.normal(case["heads"], mean=1.0, std=0.1), p + "norm2": r.normal(C, mean=1.0, std=0.1),
                          p + "mlp.up": r.matrix(case["ff"], C), p + "mlp.down": r.matrix(C, case["ff"])})
            else:
                w.update({p + "mix." + k: v for k, v in _hgrn2_weights(r, C, case["heads"]).items()})
        return w

    @staticmethod
    def _tokens(case, seed):
        g = torch.Generator().manual_seed(int(seed))
        lens = _lens(dict(tokens=case["prompt"], requests=case["requests"]))
        return [torch.randint(0, case["vocab"], (n + case["steps"],), generator=g).tolist() for n in lens], lens

    @staticmethod
    def prepare(case, seed):
        from llark_b200.engine_kelutar import KelutarEngine
        from llark_b200.models.kelutar import KelutarConfig

        engine = KelutarEngine(KelutarConfig.from_dict(_Serve._config(case)), _Serve._weights(case, _Random(seed)), "cuda", BF16)
        tokens, lens = _Serve._tokens(case, seed)
        return dict(kind=_Serve, engine=engine, cache=engine.new_cache(case["requests"]), tokens=tokens, lens=lens, steps=case["steps"])

    @staticmethod
    def run(s):
        engine, cache = s["engine"], s["cache"]
        slots = [cache.alloc() for _ in s["lens"]]
        out = [engine.step(cache, slots, [t[:n] for t, n in zip(s["tokens"], s["lens"])])]
        for k in range(s["steps"]):
            out.append(engine.step(cache, slots, [t[n + k:n + k + 1] for t, n in zip(s["tokens"], s["lens"])]))
        for slot in reversed(slots):
            cache.release(slot)
        return out

    @staticmethod
    def work(case):
        C, n, F_ = case["width"], case["heads"] * 128, case["ff"]
        w = case["layers"] * 4 * C * n + (case["layers"] // 4) * 2 * C * F_
        head, R, k = case["vocab"] * C, case["requests"], case["steps"]
        toks = sum(_lens(dict(tokens=case["prompt"], requests=R)))
        state = 8.0 * case["layers"] * R * n * 128
        return dict(bytes=(k + 1) * (2.0 * (w + head) + 4.0 * R * case["vocab"]) + (k + 0.5) * state,
                    flops=2.0 * (toks + k * R) * w + 2.0 * (k + 1) * R * head)

    @staticmethod
    def tolerance(case):
        return {"rel": 1.4e-2}  # four times the error seen against exact()

    @staticmethod
    def exact(case, seed):
        w = {k: v.to(F64) for k, v in _Serve._weights(case, _Random(seed)).items()}
        tokens, lens = _Serve._tokens(case, seed)
        xs = []
        for t in tokens:
            ids = torch.tensor(t, device="cuda")
            xs.append(w["embed"][ids] * math.sqrt(case["width"]) + w["pos"][:len(t)])
        H = case["heads"]
        for i in range(case["layers"]):
            p = f"l{i}."
            m = {k[len(p) + 4:]: v for k, v in w.items() if k.startswith(p + "mix.")}
            hs = [x + _conv64(x, w[p + "canon1"]) for x in xs]
            if i % 4 == 3:
                ys = []
                for h in hs:
                    T = h.shape[0]
                    q, k = (h @ m["q"].t() + m["q.b"]).view(T, H, 128), (h @ m["k"].t() + m["k.b"]).view(T, H, 128)
                    pos = torch.arange(T, device="cuda")
                    back = pos[:, None] - pos[None]
                    qn = _rms64(q, m["q.norm"], _Serve.eps) * m["temp"][:, None]
                    o = _attend64(qn, _rms64(k, m["k.norm"], _Serve.eps), k, (back >= 0) & (back < case["window"]), 128 ** -0.5)
                    ys.append((o.reshape(T, -1) * torch.sigmoid(h @ m["g"].t())) @ m["o"].t())
            else:
                y, _ = _hgrn2_64(m, hs, H, _Serve.eps)
                ys = y.split([h.shape[0] for h in hs])
            xs = [x + _rms64(y, w[p + "norm1"], _Serve.eps) for x, y in zip(xs, ys)]
            if i % 4 == 3:
                xs = [x + _rms64(torch.relu(x @ w[p + "mlp.up"].t()) ** 2 @ w[p + "mlp.down"].t(), w[p + "norm2"], _Serve.eps) for x in xs]
        return [_rms64(torch.stack([x[n - 1 + k] for x, n in zip(xs, lens)]), w["final.norm"], _Serve.eps) @ w["head"].t()
                for k in range(case["steps"] + 1)]


_KINDS = {"train": _Train, "decode": _Decode, "attention": _Attention, "encoder": _Encoder, "prior": _Prior,
          "recurrence": _Recurrence, "window": _Window, "moe": _Experts, "serve": _Serve}
