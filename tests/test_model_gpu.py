"""Model-level parity on the GPU: llark_b200.models.llamav2.WrappedLlamav2ForCausalLM (CUDA path through the
C-ABI) against (a) the golden vectors produced by the REFERENCE's own class and (b) the oracle restatement run on
CPU on the same seeded inputs. Tolerances (stated per assert): the reference trains in bf16, so two bf16 pipelines
are compared by relative Frobenius norm and the CUDA path's error against the fp32 reference must not exceed the bf16
reference's own error by more than 50 %. Bounds are ~2x the errors measured on a B200
(logits 4.5e-3 - 1.4e-2, gradients 8e-3 - 1.8e-2, in-place accumulation 2.5e-3)."""
import os

import pytest
import torch

from llark_b200.testing import check_close  # noqa: E402

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")
BF16 = torch.bfloat16


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return ((a - b).norm() / (b.norm() + 1e-30)).item()


from llark_b200.testing import build_model, to_cuda as _to_cuda  # noqa: E402


@pytest.fixture(scope="module")
def gold():
    return torch.load(os.path.join(GOLD, "llama_tiny_ref.pt"), weights_only=False)


@pytest.mark.parametrize("detach", [True, False])
def test_forward_backward_matches_reference_golden(gold, detach):
    from oracle import llama_oracle as lo

    cfg = lo.LlamaCfg(**gold["cfg"])
    params = lo.init_params(cfg, seed=gold["seed"])
    batch = lo.make_batch(cfg, B=2, S=48, F_frames=5, seed=0)
    model = build_model(cfg, params, detach_text=detach)
    out = model(**_to_cuda(batch))
    out.loss.backward()
    tag = "detach" if detach else "nodetach"
    ref16, ref32 = gold[f"bf16_{tag}"], gold[f"fp32_{tag}"]
    # loss: 2e-3 relative to the bf16 reference run
    assert abs(out.loss.item() - ref16["loss"].item()) < 2e-3 * ref16["loss"].item()
    valid = batch["attention_mask"]
    lg = out.logits.float().cpu()[valid]
    check_close("test_forward_backward_matches_reference_golden:_rel_lg_ref16_logits_float_valid_", _rel(lg, ref16["logits"].float()[valid]), 1e-2)
    err_mine = _rel(lg, ref32["logits"][valid])
    err_ref = _rel(ref16["logits"].float()[valid], ref32["logits"][valid])
    assert err_mine < 1.5 * err_ref + 1e-3, (err_mine, err_ref)
    named = dict(model.named_parameters())
    for n, entry in ref16["grads"].items():
        g = named[n].grad
        if entry is None:
            assert g is None, n
            continue
        assert g is not None, n
        assert abs(g.float().norm().item() - entry["norm"]) <= 5e-2 * max(entry["norm"], 1e-6), n
        if "full" in entry:
            check_close(f"test_forward_backward_matches_reference_golden:_rel_g_float_entry_full_float_:{n}", _rel(g.float(), entry["full"].float()), 2e-2)
        if "nonzero_rows" in entry:
            rows = g.float().abs().sum(-1).nonzero().flatten().tolist()
            assert rows == entry["nonzero_rows"], n
    # gradients are views of ONE flat bucket (single all-reduce / fused AdamW)
    flat = model.engine.flat
    for n, p in model.named_parameters():
        if p.grad is not None:
            assert flat.grads.data_ptr() <= p.grad.data_ptr() < flat.grads.data_ptr() + 2 * flat.grads.numel()


def test_matches_oracle_on_fresh_seed_with_list_encodings_and_accumulation():
    from oracle import llama_oracle as lo

    cfg = lo.LlamaCfg(hidden_size=512, intermediate_size=768, num_layers=3, num_heads=4, vocab_size=520,
                      mm_hidden_size=96, audio_start_token=518, audio_end_token=519, audio_patch_token=517,
                      pad_token=516)
    params = lo.init_params(cfg, seed=3)
    batch = lo.make_batch(cfg, B=3, S=80, F_frames=7, seed=5, pad_last=9)
    # ragged frame counts -> list-valued audio_encodings (collator keeps a list, data_modules.py:213-218)
    ids = batch["input_ids"]
    pos0 = 4
    ids[0, pos0 + 1 + 7] = cfg.pad_token - 1  # overwrite old end token
    ids[0, pos0 + 1: pos0 + 1 + 4] = cfg.audio_patch_token
    ids[0, pos0 + 1 + 4] = cfg.audio_end_token
    g = torch.Generator().manual_seed(11)
    encs = [torch.randn(4, cfg.mm_hidden_size, generator=g) * 0.5] + [batch["audio_encodings"][i] for i in (1, 2)]
    batch["audio_encodings"] = encs
    pb = {k: v.to(BF16) for k, v in params.items()}
    loss_o, logits_o, grads_o = lo.forward_backward(pb, cfg, batch, detach_text=True)
    model = build_model(cfg, params, detach_text=True)
    cb = _to_cuda(batch)
    cb["audio_encodings"] = [e.cuda() for e in encs]
    out = model(**cb)
    out.loss.backward()
    assert abs(out.loss.item() - loss_o.item()) < 3e-3 * loss_o.item()
    valid = batch["attention_mask"]
    check_close("test_matches_oracle_on_fresh_seed_with_list_encodings_and_accumulation:_rel_out_logits_float_cpu_valid_logits_o", _rel(out.logits.float().cpu()[valid], logits_o.float()[valid]), 1e-2)
    named = dict(model.named_parameters())
    for n, go in grads_o.items():
        if go is None:
            assert named[n].grad is None
            continue
        check_close(f"test_matches_oracle_on_fresh_seed_with_list_encodings_and_accumulation:_rel_named_n_grad_float_go_float_:{n}", _rel(named[n].grad.float(), go.float()), 2e-2)
    # second micro-batch accumulates in place (wgrad epilogue R = C): grads double
    g1 = {n: p.grad.float().clone() for n, p in named.items() if p.grad is not None}
    out2 = model(**cb)
    out2.loss.backward()
    for n, g in g1.items():
        check_close(f"test_matches_oracle_on_fresh_seed_with_list_encodings_and_accumulation:_rel_named_n_grad_float_2_g_:{n}", _rel(named[n].grad.float(), 2 * g), 1e-2)  # (embed_tokens: bf16 atomics, measured 2.6e-3; every other tensor is exact)
    # zero_grad(set_to_none) -> overwrite mode again
    model.zero_grad(set_to_none=True)
    out3 = model(**cb)
    out3.loss.backward()
    for n, g in g1.items():
        check_close(f"test_matches_oracle_on_fresh_seed_with_list_encodings_and_accumulation:_rel_named_n_grad_float_g_:{n}", _rel(named[n].grad.float(), g), 1e-2)  # embed_tokens rows are bf16 atomics: run-to-run order differs (measured up to 1.0e-3)


def test_value_errors_and_no_grad_forward(gold):
    from oracle import llama_oracle as lo

    cfg = lo.LlamaCfg(**gold["cfg"])
    params = lo.init_params(cfg, seed=0)
    batch = lo.make_batch(cfg, B=2, S=48, F_frames=5, seed=0)
    model = build_model(cfg, params)
    with torch.no_grad():
        out = model(**_to_cuda(batch))
    assert out.loss is not None and not out.loss.requires_grad
    out_nolabel = model(input_ids=batch["input_ids"].cuda(), attention_mask=batch["attention_mask"].cuda(),
                        audio_encodings=batch["audio_encodings"].cuda())
    assert out_nolabel.loss is None and out_nolabel.logits.shape == (2, 48, cfg.vocab_size)
    bad = _to_cuda(batch)
    bad["input_ids"] = bad["input_ids"].clone()
    bad["input_ids"][0, 4 + 5 + 1] = 7  # end token removed: reference raises ValueError (llamav2.py:146-152)
    with pytest.raises(ValueError):
        model(**bad)
    t = model(**_to_cuda(batch), return_dict=False)
    assert isinstance(t, tuple) and len(t) == 2


def test_llama7b_layer_shapes_run():
    """One decoder layer at the real Llama-2-7B widths (H 4096, I 11008, 32 heads, V 32004, F 240, S 512)."""
    from oracle import llama_oracle as lo

    cfg = lo.LlamaCfg(hidden_size=4096, intermediate_size=11008, num_layers=1, num_heads=32, vocab_size=32004,
                      mm_hidden_size=4800, audio_start_token=32002, audio_end_token=32003, audio_patch_token=32001,
                      pad_token=32000)
    torch.manual_seed(0)
    from llark_b200.models.llamav2 import WrappedLlamav2Config, WrappedLlamav2ForCausalLM

    hf = WrappedLlamav2Config(hidden_size=4096, intermediate_size=11008, num_hidden_layers=1, num_attention_heads=32,
                              num_key_value_heads=32, vocab_size=32004, rms_norm_eps=1e-5)
    with torch.device("cuda"):
        model = WrappedLlamav2ForCausalLM(hf)
        model.get_model().initialize_adapter_modules()
    model.to(BF16)
    aec = model.get_model().audio_encoder_config
    aec.audio_start_token, aec.audio_end_token, aec.audio_patch_token = 32002, 32003, 32001
    for p in model.get_output_embeddings().parameters():
        p.requires_grad = False
    model.get_model().orig_embeds_params = [None]
    batch = lo.make_batch(cfg, B=2, S=512, F_frames=240, seed=1, pad_last=40)
    params = {n: p.detach().float().cpu() for n, p in model.named_parameters()}
    out = model(**_to_cuda(batch))
    out.loss.backward()
    loss_o, logits_o, grads_o = lo.forward_backward({k: v.to(BF16) for k, v in params.items()}, cfg, batch,
                                                    detach_text=True)
    assert abs(out.loss.item() - loss_o.item()) < 3e-3 * loss_o.item()
    valid = batch["attention_mask"]
    check_close("test_llama7b_layer_shapes_run:_rel_out_logits_float_cpu_valid_logits_o", _rel(out.logits.float().cpu()[valid], logits_o.float()[valid]), 2e-2)
    named = dict(model.named_parameters())
    for n in ("model.mm_projector.weight", "model.layers.0.mlp.down_proj.weight", "model.layers.0.self_attn.q_proj.weight",
              "model.norm.weight"):
        check_close(f"test_llama7b_layer_shapes_run:_rel_named_n_grad_float_grads_o_n_float_:{n}", _rel(named[n].grad.float(), grads_o[n].float()), 3.5e-2)


def test_optimizer_step_then_backward_overwrites_stale_grads(gold):
    """After the fused optimizer step the gradient bucket is 'consumed': the next backward must overwrite it
    (no stale accumulation), and the loss must go down on the same batch."""
    from oracle import llama_oracle as lo
    from llark_b200.optim import LlarkAdamW

    cfg = lo.LlamaCfg(**gold["cfg"])
    model = build_model(cfg, lo.init_params(cfg, seed=0))
    opt = LlarkAdamW(model, lr=1e-3)
    batch = _to_cuda(lo.make_batch(cfg, B=2, S=48, F_frames=5, seed=0))
    l0 = model(**batch).loss
    l0.backward()
    opt.step()
    out = model(**batch)
    out.loss.backward()
    g_a = {n: p.grad.float().clone() for n, p in model.named_parameters() if p.grad is not None}
    model.zero_grad(set_to_none=True)
    model(**batch).loss.backward()
    for n, p in model.named_parameters():
        if p.grad is not None:
            assert torch.equal(p.grad.float(), g_a[n]), n
    assert out.loss.item() < l0.item()
    # explicit zero_grad() between accumulation windows also works
    opt.zero_grad()
    model(**batch).loss.backward()
    model(**batch).loss.backward()
    for n, p in model.named_parameters():
        if p.grad is not None:
            check_close(f"test_optimizer_step_then_backward_overwrites_stale_grads:_rel_p_grad_float_2_g_a_n_:{n}", _rel(p.grad.float(), 2 * g_a[n]), 1e-2)  # (embed_tokens: bf16 atomics, measured 1.9e-3)


def test_generate_greedy_decoding_without_cache():
    """WrappedLlamav2ForCausalLM.generate (m2t/infer.py:146-152 call shape): cache-less greedy decoding on the CUDA
    engine. Every generated token must be the argmax of a teacher-forced forward up to bf16 noise, the sequence must
    equal the reference's GenerationMixin.generate (tests/golden/generation_ref.pt, fp32) up to the first step whose
    fp32 top-2 margin is below 0.05, and eos / stopping criteria / max_length must cut it where the reference's do."""
    from oracle import llama_oracle as lo
    from oracle.make_golden_generation import StopOnToken, gen_inputs

    gold_gen = torch.load(os.path.join(GOLD, "generation_ref.pt"), weights_only=False)["generate"]
    cfg, params, ids, enc = gen_inputs()
    model = build_model(cfg, params)
    ids_c, enc_c = ids.cuda(), enc.cuda()
    P = ids.shape[1]
    seq = model.generate(input_ids=ids_c, audio_encodings=enc_c, max_new_tokens=8, labels=None, example_id="x")
    assert seq.shape == (1, P + 8) and torch.equal(seq[:, :P], ids_c)
    with torch.no_grad():
        logits = model(input_ids=seq[:, :-1], audio_encodings=enc_c).logits.float()[0]
    for t in range(P, P + 8):
        row = logits[t - 1]
        assert row[seq[0, t]] >= row.max() - 3e-2 * row.abs().max(), t
    ref = gold_gen["sequences"]["plain"][0]
    ref_logits = lo.forward(params, cfg, ref[None, :-1], None, None, enc)[1][0]
    for t in range(P, P + 8):
        top = ref_logits[t - 1].topk(2).values
        if (top[0] - top[1]).item() < 0.05:
            break
        assert seq[0, t].item() == ref[t].item(), t
    new = seq[0, P:].tolist()
    # eos: emitted, then generation stops
    first = new.index(new[2])
    out = model.generate(input_ids=ids_c, audio_encodings=enc_c, max_new_tokens=8, eos_token_id=new[2])
    assert out[0].tolist() == seq[0, : P + first + 1].tolist()
    # stopping criterion (the KeywordsStoppingCriteria calling convention)
    first = new.index(new[3])
    out = model.generate(input_ids=ids_c, audio_encodings=enc_c, max_new_tokens=8, stopping_criteria=[StopOnToken(new[3])])
    assert out[0].tolist() == seq[0, : P + first + 1].tolist()
    # max_length counts the prompt
    out = model.generate(input_ids=ids_c, audio_encodings=enc_c, max_length=P + 3)
    assert out[0].tolist() == seq[0, : P + 3].tolist()
    with pytest.raises(NotImplementedError):
        model.generate(input_ids=ids_c, audio_encodings=enc_c, do_sample=True)




def test_generate_with_kv_cache_matches_cacheless():
    """Prefill + single-token decode steps against the KV cache (LLARK_KV_CACHE=1) must pick the same tokens as the
    cache-less loop and reproduce its last-position logits (bf16 noise only)."""
    from oracle.make_golden_generation import gen_inputs

    cfg, params, ids, enc = gen_inputs()
    model = build_model(cfg, params)
    ids_c, enc_c = ids.cuda(), enc.cuda()
    os.environ["LLARK_KV_CACHE"] = "0"
    ref = model.generate(input_ids=ids_c, audio_encodings=enc_c, max_new_tokens=8)
    with torch.no_grad():
        full = model(input_ids=ref[:, :-1], audio_encodings=enc_c).logits.float()
    os.environ["LLARK_KV_CACHE"] = "1"
    try:
        got = model.generate(input_ids=ids_c, audio_encodings=enc_c, max_new_tokens=8)
        out = model(input_ids=ids_c, audio_encodings=enc_c, use_cache=True)
        cache = out.past_key_values
        assert len(cache) == ids.shape[1] and torch.allclose(out.logits.float(), full[:, : ids.shape[1]], atol=3e-2)
        step = model(input_ids=ref[:, ids.shape[1]: ids.shape[1] + 1], past_key_values=cache, use_cache=True)
        assert step.logits.shape == (1, 1, cfg.vocab_size) and len(cache) == ids.shape[1] + 1
        assert torch.allclose(step.logits.float()[0, 0], full[0, ids.shape[1]], atol=5e-2)
    finally:
        os.environ.pop("LLARK_KV_CACHE", None)
    assert torch.equal(got, ref)


def test_activation_recompute_is_bit_identical_on_gpu(gold):
    """LLARK_RECOMPUTE=1 (what --gradient_checkpointing True selects under memory pressure): the backward regenerates each
    layer's activations from its input with the same kernels, so loss and every gradient match the plain step bit for
    bit. Written after the round's GPU budget was spent (the CPU stand-in version of this test runs in the CPU suite)."""
    from oracle import llama_oracle as lo

    cfg = lo.LlamaCfg(**gold["cfg"])
    batch = _to_cuda(lo.make_batch(cfg, B=2, S=48, F_frames=5, seed=0))
    res = []
    for mode in ("0", "1"):
        model = build_model(cfg, lo.init_params(cfg, seed=0))
        model.engine.recompute = mode
        out = model(**batch)
        out.loss.backward()
        res.append((out.loss.item(), model.engine.flat.grads.clone(), model.engine.recomputed_last_step))
    assert [r[2] for r in res] == [False, True]
    assert res[0][0] == res[1][0] and torch.equal(res[0][1], res[1][1])


def test_wrapped_trainer_follows_the_reference_trajectory_on_gpu(tmp_path):
    """GPU twin of tests/test_trainstep_cpu.py: WrappedTrainer + the fused AdamW kernel on the CUDA engine against the
    reference's 4-step trajectory (tests/golden/trainstep_ref.pt). Written after the round's GPU budget was spent."""
    from oracle import llama_oracle as lo
    from test_trainstep_cpu import GOLD as TRAJ, check_against_reference, run_trajectory

    gold_t = torch.load(TRAJ, weights_only=False)
    cfg = lo.LlamaCfg(**gold_t["cfg"])
    model = build_model(cfg, lo.init_params(cfg, seed=gold_t["seed"]), detach_text=True)
    trainer = run_trajectory(model, gold_t, tmp_path)
    check_against_reference(trainer, model, gold_t, loss_tol=1e-2, delta_tol=0.05, cos_min=0.98)


def test_frozen_backbone_projector_only_training_on_gpu(gold):
    """GPU twin of tests/test_engine_host_cpu.py::test_frozen_backbone_projector_only_training (--freeze_backbone True):
    null weight-gradient pointers for every decoder tensor, dgrad through all layers, a bucket with two trainable tensors."""
    from oracle import llama_oracle as lo
    from llark_b200.optim import LlarkAdamW

    cfg = lo.LlamaCfg(**gold["cfg"])
    params = lo.init_params(cfg, seed=0)
    batch = lo.make_batch(cfg, B=2, S=48, F_frames=5, seed=1)
    model = build_model(cfg, params, detach_text=True)
    model.requires_grad_(False)
    for p in model.get_model().mm_projector.parameters():
        p.requires_grad = True
    for p in model.get_input_embeddings().parameters():
        p.requires_grad = True
    opt = LlarkAdamW(model, lr=1e-2)
    out = model(**_to_cuda(batch))
    out.loss.backward()
    _, _, grads_o = lo.forward_backward({k: v.to(torch.bfloat16) for k, v in params.items()}, cfg, batch)
    named = dict(model.named_parameters())
    for n in ("model.mm_projector.weight", "model.mm_projector.bias", "model.embed_tokens.weight"):
        check_close(f"test_frozen_backbone_projector_only_training_on_gpu:_rel_named_n_grad_float_grads_o_n_float_:{n}", _rel(named[n].grad.float(), grads_o[n].float()), 2e-2)
    assert all(p.grad is None for n, p in named.items() if "layers" in n or n in ("model.norm.weight", "lm_head.weight"))
    l0 = out.loss.item()
    for _ in range(3):
        opt.step()
        model(**_to_cuda(batch)).loss.backward()
    with torch.no_grad():
        assert model(**_to_cuda(batch)).loss.item() < l0


@pytest.mark.parametrize("gemm_mode,tol", [("3xtf32", 1e-3), ("tf32", 2e-3)])
def test_fp32_verification_mode_meets_the_1e3_logit_criterion(gold, gemm_mode, tol, capsys):
    """north_star: "fp32 logits within 1e-3 relative" of the reference's own PyTorch path. LLARK_VERIFY=fp32 runs the forward
    with fp32 tensors end to end (3xTF32 products on the tcgen05 core + csrc/verify_fp32.cu) and is compared with the fp32
    run of the REFERENCE's WrappedLlamav2ForCausalLM stored in tests/golden/llama_tiny_ref.pt. Criterion: relative
    Frobenius error over the valid rows AND max |error| / max |logit| both <= 1e-3 (plain single-pass TF32 is also
    measured, against a looser bound, to show what the 3x split buys). The measured errors are printed."""
    from oracle import llama_oracle as lo

    cfg = lo.LlamaCfg(**gold["cfg"])
    params = lo.init_params(cfg, seed=gold["seed"])
    batch = lo.make_batch(cfg, B=2, S=48, F_frames=5, seed=0)
    model = build_model(cfg, params, dtype=torch.float32)
    ref = gold["fp32_detach"]
    os.environ["LLARK_VERIFY"] = "fp32"
    os.environ["LLARK_VERIFY_GEMM"] = gemm_mode
    try:
        with torch.no_grad():
            out = model(**_to_cuda(batch))
    finally:
        os.environ.pop("LLARK_VERIFY", None)
        os.environ.pop("LLARK_VERIFY_GEMM", None)
    valid = batch["attention_mask"]
    lg, want = out.logits.float().cpu()[valid], ref["logits"][valid]
    fro = _rel(lg, want)
    mx = ((lg - want).abs().max() / want.abs().max()).item()
    dl = abs(out.loss.item() - ref["loss"].item()) / ref["loss"].item()
    with capsys.disabled():
        print(f"\n[fp32 verify {gemm_mode}] logits rel-Frobenius {fro:.3e}, max-abs/max {mx:.3e}, loss rel {dl:.3e}")
    assert out.logits.dtype == torch.float32
    assert fro <= tol and mx <= tol and dl <= tol, (fro, mx, dl)
