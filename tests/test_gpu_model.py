"""GPU parity tests of the mirrored `mmfreelm` API (modules, layer, model, generate) against the CPU oracle
and the reference fixtures.  Run with `-m gpu` on a B200."""
import numpy as np
import pytest
import torch

from oracle import mmfree_oracle as O

pytestmark = pytest.mark.gpu


def _close_up_to_code_flips(got, ref, typical, worst):
    """See tests/test_oracle_golden.py: quantisation is discontinuous, so two correct implementations agree
    to `typical` on almost every element and to `worst` on all (relative to max|ref|)."""
    scale = np.abs(ref).max()
    d = np.abs(got - ref)
    assert np.quantile(d, 0.5) <= typical * scale, ("typical", np.quantile(d, 0.5) / scale)
    assert d.max() <= worst * scale, ("worst", d.max() / scale)


@pytest.fixture(scope="module")
def mm():
    import matmulfreellm_b200 as pkg
    pkg.install_as_mmfreelm()
    assert torch.cuda.is_available()
    return pkg


def tiny_cfg():
    return O.OracleConfig(vocab_size=32000, hidden_size=256, num_hidden_layers=2, intermediate_size=704)


def build_gpu_model(sd, cfg, dtype):
    """Load the oracle's fp32 state dict into the CUDA model, pack from fp32, then cast."""
    from mmfreelm.models import HGRNBitConfig, HGRNBitForCausalLM
    hf = HGRNBitConfig(vocab_size=cfg.vocab_size, hidden_size=cfg.hidden_size, num_hidden_layers=cfg.num_hidden_layers,
                       intermediate_size=cfg.intermediate_size, rms_norm_eps=cfg.rms_norm_eps)
    model = HGRNBitForCausalLM(hf).eval()
    missing, unexpected = model.load_state_dict(sd, strict=True)
    assert not missing and not unexpected
    model = model.cuda()
    model.pack_weights()
    return model.to(dtype)


def test_mmfreelm_import_paths(mm):
    import mmfreelm
    from mmfreelm import HGRNBitForCausalLM, HGRNBitModel  # noqa: F401
    from mmfreelm.layers import HGRNBitAttention  # noqa: F401
    from mmfreelm.models import HGRNBitConfig  # noqa: F401
    from mmfreelm.models.utils import RecurrentCache  # noqa: F401
    from mmfreelm.modules import FusedRMSNormSwishGate, RMSNorm  # noqa: F401
    from mmfreelm.modules.activations import swiglu  # noqa: F401
    from mmfreelm.ops import fused_recurrent_hgrn  # noqa: F401
    from mmfreelm.ops.fusedbitnet import BitLinear, FusedBitLinear, activation_quant, weight_quant  # noqa: F401
    from mmfreelm.ops.hgrn import chunk_hgrn  # noqa: F401
    assert mmfreelm.__version__ == "0.1"


def test_fused_bitlinear_module(mm):
    """FusedBitLinear(x) for bf16 [..., K] input: equal to the integer oracle rounded to bf16; and within the
    stated bf16 tolerance (rel 1e-2) of the reference's float BitLinear math."""
    from mmfreelm.ops.fusedbitnet import BitLinear, FusedBitLinear, activation_quant, weight_quant
    x, w, _ = O.bitlinear_case(2 * 5, 2048, 384, seed=4)
    g = torch.Generator().manual_seed(8)
    nw = 1.0 + 0.1 * torch.randn(2048, generator=g)
    for cls, eps in ((FusedBitLinear, 1e-6), (BitLinear, 1e-8)):
        lin = cls(2048, 384)
        with torch.no_grad():
            lin.weight.copy_(w)
            lin.norm.weight.copy_(nw)
        lin = lin.cuda()
        y = lin(x.view(2, 5, 2048).cuda())
        assert y.shape == (2, 5, 384) and y.dtype == torch.bfloat16
        codes, mean = O.ternary_codes(w)
        ref_int = O.bitlinear_int(x, nw, codes, mean, eps, out_dtype=torch.bfloat16)[0]
        assert torch.equal(y.cpu().view(10, 384), ref_int)
        ref_float = O.bitlinear_ref(x.float(), nw, w, eps=eps)
        assert (y.cpu().float().view(10, 384) - ref_float).abs().max() <= 1e-2 * ref_float.abs().max()
    xf = torch.randn(6, 256, generator=g)
    assert torch.allclose(activation_quant(xf.cuda()).cpu(), O.activation_quant(xf), rtol=1e-6, atol=1e-7)
    wf = torch.randn(128, 256, generator=g) * 0.02
    assert torch.allclose(weight_quant(wf.cuda()).cpu(), O.weight_quant(wf), rtol=1e-6, atol=1e-9)


@pytest.mark.parametrize("M", [2, 5])
def test_linear_quant_fn_takes_any_strides(mm, M):
    """layer_norm_linear_quant_fn on a slice with an odd row pitch and start, on a transposed and on an expanded input: the result
    of a contiguous copy."""
    from mmfreelm.ops.fusedbitnet import layer_norm_linear_quant_fn
    K, N = 256, 384
    g = torch.Generator().manual_seed(M)
    w, nw = (torch.randn(N, K, generator=g) * 0.02).cuda(), torch.rand(K, generator=g).cuda()
    wide = torch.randn(M, K + 3, generator=g).bfloat16().cuda()
    for x in (wide[:, 1:K + 1], torch.randn(K, M, generator=g).bfloat16().cuda().t(), wide[:1, :K].expand(M, K), wide[:, :K].view(1, M, K)):
        want = layer_norm_linear_quant_fn(x.clone(memory_format=torch.contiguous_format), nw, None, w, None, is_rms_norm=True)
        assert torch.equal(layer_norm_linear_quant_fn(x, nw, None, w, None, is_rms_norm=True), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bitlinear_row_pitches(mm, dtype):
    """A BitLinear takes a single row whatever its pitch says (a slice of a wider tensor, an expanded row); rows at a pitch that is
    not a multiple of 16 bytes, or below their length, are refused, and so is a row that does not start on 16 bytes."""
    from matmulfreellm_b200._lib import MMFreeError
    from mmfreelm.ops.fusedbitnet import FusedBitLinear
    K, N = 256, 130
    layer = FusedBitLinear(K, N).cuda()
    layer.pack_weights()
    layer = layer.to(dtype)
    wide = torch.randn(4, K + 9, generator=torch.Generator().manual_seed(1)).cuda().to(dtype)
    want = layer(wide[:, :K].contiguous())
    assert torch.equal(layer(wide[:1, :K]), want[:1]) and torch.equal(layer(wide[0, :K].expand(1, K)), want[:1])
    assert torch.equal(layer(wide[:1, None, :K]), want[:1, None])
    padded = torch.nn.functional.pad(wide, (0, 7))
    for M in (1, 2, 3, 4):
        assert torch.equal(layer(padded[:M, :K]), want[:M])
        for bad in (wide[:M, 1:K + 1], *([wide[:M, :K], wide[0, :K].expand(M, K)] if M > 1 else [])):
            with pytest.raises(MMFreeError):
                layer(bad)


def test_hgrn_ops_reference_selfcheck_shapes(mm):
    """The reference's own self-check (recurrent_fuse.py:188-217): B,H,T,D = 8,4,512,128, bf16, seed 42,
    g = sigmoid(randn), x = (1-g)*randn, random h0 — fused op against the naive loop."""
    from mmfreelm.ops.hgrn import chunk_hgrn, fused_recurrent_hgrn
    torch.manual_seed(42)
    B, H, T, D = 8, 4, 512, 128
    g = torch.randn(B, H, T, D).sigmoid()
    x = ((1 - g) * torch.randn(B, H, T, D)).bfloat16()
    g = g.bfloat16()
    h0 = torch.randn(B, H, D).bfloat16()
    o_ref, ht_ref = O.naive_recurrent_hgrn(x, g, h0, True)
    o, ht = fused_recurrent_hgrn(x.cuda(), g.cuda(), h0.cuda(), output_final_state=True)
    assert o.dtype == torch.bfloat16 and ht.dtype == torch.bfloat16 and ht.shape == (B, H, D)
    assert (o.cpu().float() - o_ref.float()).abs().max() <= 1e-2 * o_ref.float().abs().max()
    assert (ht.cpu().float() - ht_ref).abs().max() <= 1e-2 * ht_ref.abs().max()
    o2, none = fused_recurrent_hgrn(x.cuda(), g.cuda())
    assert none is None
    # chunk_hgrn takes the LOG gate and returns an fp32 state
    oc, htc = chunk_hgrn(x.cuda(), g.float().log().cuda(), h0.cuda(), output_final_state=True)
    assert htc.dtype == torch.float32
    assert (oc.cpu().float() - o_ref.float()).abs().max() <= 1e-2 * o_ref.float().abs().max()
    assert (htc.cpu() - ht_ref).abs().max() <= 1e-4 * ht_ref.abs().max()


def test_norm_modules(mm):
    from mmfreelm.modules import FusedRMSNormSwishGate, RMSNorm
    g = torch.Generator().manual_seed(3)
    x = torch.randn(2, 7, 256, generator=g).bfloat16()
    o = torch.randn(2, 7, 256, generator=g).bfloat16()
    res = torch.randn(2, 7, 256, generator=g).bfloat16()
    norm = RMSNorm(256, eps=1e-6).cuda()
    gate = FusedRMSNormSwishGate(256, eps=1e-6).cuda()
    w = torch.ones(256)
    y, r = norm(x.cuda(), res.cuda(), True)
    y_ref, r_ref = O.rms_norm_ref(x, w, residual=res, eps=1e-6, prenorm=True)
    assert (y.cpu().float() - y_ref.float()).abs().max() <= 2 ** -7 * y_ref.float().abs().max()
    assert torch.equal(r.cpu(), r_ref)
    yg = gate(x.cuda(), o.cuda())
    ref = O.swish_gate_norm_ref(x, o, w, 1e-6)
    assert (yg.cpu().float() - ref.float()).abs().max() <= 2 ** -7 * ref.float().abs().max()
    assert "RMSNorm(256, eps=1e-06)" == repr(norm)


def test_tiny_model_fp32_vs_oracle_and_reference(mm, golden):
    """The tiny configuration the reference itself can run on a CPU (2 layers, hidden 256, intermediate 704, vocab
    32000, batch 2 x 128, fp32): logits and final HGRN states against the integer oracle and against the reference's
    own output."""
    g = golden["tiny_model"]
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=0)
    sd["model.lower_bounds"] = torch.from_numpy(g["lower_bounds"])
    ids = torch.from_numpy(g["ids"])
    model = build_gpu_model(sd, cfg, torch.float32)
    out = model(ids.cuda(), use_cache=True)
    logits = out.logits.cpu()
    states = [s[0].cpu() for s in out.past_key_values]
    assert logits.shape == (2, 128, 32000) and states[0].shape == (2, 1, 256) and states[0].dtype == torch.float32

    oracle = O.OracleHGRNBit(cfg, sd, dtype=torch.float32, linear="int", bitlinear_eps=1e-6)
    ref_logits, ref_states = oracle.forward(ids)
    _close_up_to_code_flips(logits.numpy(), ref_logits.numpy(), 2e-6, 2e-2)
    for s, r in zip(states, ref_states):
        _close_up_to_code_flips(s.numpy(), r.numpy(), 1e-5, 2e-2)      # fp32 state: typical << 1e-4
    assert (logits.argmax(-1) == ref_logits.argmax(-1)).float().mean() >= 0.97

    # the reference itself: its CPU-runnable variant (BitLinear.forward) uses eps 1e-8 inside BitLinear where
    # the fused GPU call uses 1e-6, so the fixture is compared with the modules switched to 1e-8
    from mmfreelm.ops.fusedbitnet import BitLinear
    for m in model.modules():
        if isinstance(m, BitLinear):
            m.NORM_EPS = 1e-8
    model._fused_runner = None          # the fused chain caches each layer's eps when it is built
    out8 = model(ids.cuda(), use_cache=True)
    _close_up_to_code_flips(out8.logits[:, g["logits_pos"]].cpu().numpy(), g["logits_at"], 2e-5, 5e-2)
    for i, s in enumerate(out8.past_key_values):
        _close_up_to_code_flips(s[0].cpu().numpy(), g["states"][i], 2e-5, 5e-2)
    for m in model.modules():
        if isinstance(m, BitLinear):
            del m.NORM_EPS
    model._fused_runner = None

    # prefill + one cached step == one longer forward (incremental decoding is consistent)
    full = model(ids[:, :65].cuda(), use_cache=False).logits[:, -1]
    o1 = model(ids[:, :64].cuda(), use_cache=True)
    o2 = model(ids[:, 64:65].cuda(), past_key_values=o1.past_key_values, use_cache=True).logits[:, -1]
    _close_up_to_code_flips(o2.cpu().numpy(), full.cpu().numpy(), 2e-6, 2e-2)


@pytest.mark.parametrize("dtype,typical,worst", [(torch.float32, 1e-5, 3e-2), (torch.bfloat16, 1e-2, 1e-1), (torch.float16, 2e-3, 1e-1)])
def test_greedy_decode_64_steps_matches_oracle(mm, dtype, typical, worst):
    """Greedy decoding for 64 steps, batch 2, prompt 32, through the CUDA-graph decoder and through `generate`.
    A sequence may leave the oracle's path only at a step where the oracle's own top-2 margin is within twice the
    logit error MEASURED for that row in the teacher-forced pass of the same run (oracle.greedy_parity); the
    teacher-forced logits stay within the stated tolerance; in fp32 the tokens are identical, in half precision (a
    random-init model has near-flat logits, so ties do occur) a large share of the teacher-forced rows is bit-identical."""
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=5)
    ids = torch.randint(0, 32000, (2, 32), generator=torch.Generator().manual_seed(6))
    model = build_gpu_model(sd, cfg, dtype)
    oracle = O.OracleHGRNBit(cfg, sd, dtype=dtype, linear="int", bitlinear_eps=1e-6)
    dec = GreedyDecoder(model, 2)
    r = O.greedy_parity(oracle, ids, 64, dec, lambda p: model(p.cuda(), use_cache=False, last_token_only=True).logits[:, -1])
    assert dec.graph is not None
    print(f"[greedy {dtype}] identical tokens {r['identical_fraction']:.3f} ({r['identical_sequences']}/2 sequences); logit error per "
          f"row: median {r['err_median']:.2e}, max {r['err_max']:.2e}; bit-identical rows {r['exact_rows']:.3f}; min oracle top-2 "
          f"margin {r['min_margin']:.2e}")
    assert r["explained"], r["violations"]
    if dtype == torch.float32:
        assert r["identical_fraction"] >= 0.99
    else:
        # with two free-running sequences the identical-token fraction only says how early the first tie fell (measured
        # 0.15 - 0.74); the robust figure is the share of teacher-forced rows whose logits are bit-identical (0.65 - 0.87)
        assert r["exact_rows"] >= 0.4
    # `generate` (the reference's entry point) gives the decoder's tokens
    got = model.generate(ids.cuda(), max_new_tokens=64)
    assert got.shape == (2, 96) and torch.equal(got[:, :32].cpu(), ids)
    own = [dec.prefill(ids.cuda()).clone()]
    for _ in range(63):
        own.append(dec.step().clone())
    assert torch.equal(got[:, 32:], torch.stack(own, 1))
    # teacher-forced, all positions at once: feed the oracle's tokens and compare every position's logits
    ref_tokens, _ = oracle.greedy(ids, 64)
    seq = torch.cat([ids, ref_tokens], 1)
    ref_logits, _ = oracle.forward(seq)
    logits = model(seq.cuda(), use_cache=False).logits.float().cpu()
    _close_up_to_code_flips(logits.numpy(), ref_logits.float().numpy(), typical, worst)


def test_fused_chain_equals_module_path(mm):
    """HGRNBitForCausalLM.forward runs a chain of fused kernels; with `fuse = False` it runs module by module
    (RMSNorm, FusedBitLinear, swiglu, ... each as its own call).  Same arithmetic, same rounding points."""
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=9)
    sd["model.lower_bounds"] = 0.5 * torch.randn(2, 256, generator=torch.Generator().manual_seed(3))
    ids = torch.randint(0, 32000, (3, 40), generator=torch.Generator().manual_seed(10)).cuda()
    for dtype, typical, worst in ((torch.float32, 1e-6, 2e-2), (torch.bfloat16, 4e-3, 1e-1)):
        model = build_gpu_model(sd, cfg, dtype)
        fused = model(ids, use_cache=True)
        model.fuse = False
        plain = model(ids, use_cache=True)
        del model.fuse
        _close_up_to_code_flips(fused.logits.float().cpu().numpy(), plain.logits.float().cpu().numpy(), typical, worst)
        for a, b in zip(fused.past_key_values, plain.past_key_values):
            _close_up_to_code_flips(a[0].cpu().numpy(), b[0].cpu().numpy(), typical, worst)
        # last_token_only and a cached step agree with the full forward
        last = model(ids, use_cache=False, last_token_only=True).logits
        assert torch.equal(last[:, 0], fused.logits[:, -1])
        o1 = model(ids[:, :39], use_cache=True)
        o2 = model(ids[:, 39:], past_key_values=o1.past_key_values, use_cache=True)
        _close_up_to_code_flips(o2.logits[:, -1].float().cpu().numpy(), fused.logits[:, -1].float().cpu().numpy(), typical, worst)


def test_long_prompt_uses_persistent_kernel_with_identical_results(mm):
    """A prompt of 6 x 512 tokens is large enough for the persistent tensor-core kernel (192- / 256-token tiles, work
    list per CTA).  The contraction is exact integer arithmetic, so logits and states must be identical to a run
    with that kernel switched off (override 7 = 2 of the experiments build: one CTA per tile)."""
    from matmulfreellm_b200 import _lib
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=12)
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    ids = torch.randint(0, 32000, (6, 512), generator=torch.Generator().manual_seed(13)).cuda()
    a = model(ids, use_cache=True)
    with _lib.experiments_library() as lib:      # the build that exports the configuration overrides
        lib.mmf_tuning(7, 2)
        b = model(ids, use_cache=True)
    assert torch.equal(a.logits, b.logits)
    for x, y in zip(a.past_key_values, b.past_key_values):
        assert torch.equal(x[0], y[0])
    # 3072 rows also put the row-wise kernels on their four-rows-per-CTA build.  Sequences are independent, so one of them
    # run alone (512 rows: one row per CTA, another contraction tiling) must give the same bits.
    for i in (0, 5):
        c = model(ids[i:i + 1], use_cache=True)
        assert torch.equal(c.logits[0], a.logits[i])
        for x, y in zip(c.past_key_values, a.past_key_values):
            assert torch.equal(x[0][0], y[0][i])
    from matmulfreellm_b200 import kernels
    kernels.check_status()


def test_left_padded_prompt_fused_equals_module_path(mm):
    """A left-padded batch (attention_mask with leading zeros) runs through the fused chain with the mask applied
    inside the scan; the module-by-module path applies it as the reference does (i.mul_(mask))."""
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=21)
    ids = torch.randint(0, 32000, (3, 48), generator=torch.Generator().manual_seed(22)).cuda()
    mask = torch.ones(3, 48, dtype=torch.long, device="cuda")
    mask[0, :5] = 0
    mask[2, :17] = 0
    for dtype, typical, worst in ((torch.float32, 1e-6, 2e-2), (torch.bfloat16, 4e-3, 1e-1)):
        model = build_gpu_model(sd, cfg, dtype)
        fused = model(ids, attention_mask=mask, use_cache=True)
        model.fuse = False
        plain = model(ids, attention_mask=mask, use_cache=True)
        del model.fuse
        _close_up_to_code_flips(fused.logits.float().cpu().numpy(), plain.logits.float().cpu().numpy(), typical, worst)
        for a, b in zip(fused.past_key_values, plain.past_key_values):
            _close_up_to_code_flips(a[0].cpu().numpy(), b[0].cpu().numpy(), typical, worst)
        # and the mask matters: without it the padded rows give different states
        nomask = model(ids, use_cache=True)
        assert not torch.equal(nomask.past_key_values[0][0][2], fused.past_key_values[0][0][2])


def test_masked_decode_token_runs_in_the_fused_step(mm):
    """A single cached token whose attention_mask entry is 0 (hgrn_bit.py:119-120 with T = 1) is handled inside the
    fused decode step: same logits and states as the module-by-module path, and a masked sequence's state only decays."""
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=23)
    ids = torch.randint(0, 32000, (3, 10), generator=torch.Generator().manual_seed(24)).cuda()
    step_mask = torch.tensor([[1], [0], [1]], device="cuda")
    for dtype, typical, worst in ((torch.float32, 1e-6, 2e-2), (torch.bfloat16, 4e-3, 1e-1)):
        model = build_gpu_model(sd, cfg, dtype)
        assert model._can_fuse(ids[:, -1:], None, step_mask, None)
        outs = []
        for fuse in (True, False):
            model.fuse = fuse
            o1 = model(ids[:, :9], use_cache=True)
            before = [s[0].clone() for s in o1.past_key_values]
            o2 = model(ids[:, 9:], attention_mask=step_mask, past_key_values=o1.past_key_values, use_cache=True)
            outs.append((o2.logits.float().cpu().numpy(), [s[0].float().cpu().numpy() for s in o2.past_key_values], before))
        del model.fuse
        _close_up_to_code_flips(outs[0][0], outs[1][0], typical, worst)
        for a, b in zip(outs[0][1], outs[1][1]):
            _close_up_to_code_flips(a, b, typical, worst)
        # masked sequence (row 1): h' = f * h with 0 < f < 1, so every state component shrinks and keeps its sign
        h0 = outs[0][2][0][1].float().cpu().numpy()
        h1 = outs[0][1][0][1]
        assert np.all(np.abs(h1) <= np.abs(h0) + 1e-12) and np.all(h1 * h0 >= 0)
        assert not np.all(np.abs(outs[0][1][0][0]) <= np.abs(outs[0][2][0][0].float().cpu().numpy()))   # an unmasked row receives input
    mm.kernels.check_status()


def test_generate_api(mm):
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=1)
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    ids = torch.randint(0, 32000, (3, 5), generator=torch.Generator().manual_seed(0)).cuda()
    a = model.generate(ids, max_new_tokens=4)
    b = model.generate(ids, max_length=9)
    assert a.shape == (3, 9) and torch.equal(a, b)
    with pytest.raises(ValueError):
        model.model(input_ids=ids, inputs_embeds=torch.zeros(3, 5, 256, device="cuda"))
    with pytest.raises(ValueError):
        model.model()
    with pytest.raises(NotImplementedError):
        model.generate(ids, num_beams=4)
    # options that would change the result are refused, not ignored; their neutral values pass
    for bad in (dict(repetition_penalty=1.3), dict(min_length=7), dict(top_k=50), dict(stopping_criteria=[object()]),
                dict(no_such_option=1), dict(eos_token_id=5, pad_token_id=0)):
        with pytest.raises(NotImplementedError):
            model.generate(ids, max_new_tokens=2, **bad)
    assert torch.equal(model.generate(ids, max_new_tokens=4, repetition_penalty=1.0, top_k=0, num_beams=1, use_cache=True,
                                      pad_token_id=0), a)
    # sampling: reproducible from the generator's seed (top_p -> 0 picks among the tied maxima: kernel-level test)
    g1 = torch.Generator(device="cuda").manual_seed(7)
    g2 = torch.Generator(device="cuda").manual_seed(7)
    s1 = model.generate(ids, max_new_tokens=6, do_sample=True, top_p=0.4, temperature=0.6, generator=g1)
    s2 = model.generate(ids, max_new_tokens=6, do_sample=True, top_p=0.4, temperature=0.6, generator=g2)
    assert s1.shape == (3, 11) and torch.equal(s1, s2) and torch.equal(s1[:, :5], ids)
    s0 = model.generate(ids, max_new_tokens=4, do_sample=True, top_p=0.0, generator=g1)
    assert s0.shape == a.shape and torch.equal(s0[:, :5], ids)


def test_packed_checkpoint_round_trip(mm, tmp_path):
    """save_packed -> load_packed: the loaded model never holds a latent weight, serves the same packed bytes and
    produces identical logits and tokens; the bytes in the file are the oracle's packing of the oracle's ternary codes."""
    from matmulfreellm_b200 import checkpoint
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=31)
    sd["model.lower_bounds"] = 0.3 * torch.randn(2, 256, generator=torch.Generator().manual_seed(4))
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    path = str(tmp_path / "tiny.mmfpack.npz")
    info = checkpoint.save_packed(model, path)
    n_ternary = sum(v.numel() for k, v in sd.items() if k.endswith("_proj.weight") or k == "lm_head.weight")
    assert info["bitlinear"] == 2 * 6 + 1
    assert info["bytes"] < n_ternary // 4 + 2 * 32000 * 256 + 300_000      # 2 bits per weight + the bf16 embedding table
    # file contents against the oracle (host only)
    _, manifest, z = checkpoint.read_packed(path)
    name = "model.layers.1.mlp.gate_proj"
    codes, mean = O.ternary_codes(sd[name + ".weight"])
    assert np.array_equal(z[name + ".packed"].view(np.uint32), O.pack_ternary(codes).reshape(-1))
    assert z[name + ".scale"][0] == np.float32(mean) and manifest["bitlinear"][name] == [1408, 256]
    # load and compare
    loaded = checkpoint.load_packed(path, "cuda")
    assert all(m.weight.numel() == 0 for m in loaded.modules() if type(m).__name__ in ("BitLinear", "FusedBitLinear"))
    ids = torch.randint(0, 32000, (2, 24), generator=torch.Generator().manual_seed(5)).cuda()
    a, b = model(ids, use_cache=True), loaded(ids, use_cache=True)
    assert torch.equal(a.logits, b.logits)
    for x, y in zip(a.past_key_values, b.past_key_values):
        assert torch.equal(x[0], y[0])
    assert torch.equal(model.generate(ids, max_new_tokens=8), loaded.generate(ids, max_new_tokens=8))


@pytest.mark.parametrize("ckpt_dtype", [torch.float32, torch.float16])
def test_reference_format_checkpoint_to_packed_model(mm, tmp_path, ckpt_dtype):
    """The loading path of the reference's generate.py:7-9 with a checkpoint written locally in the published format
    (config.json + safetensors with the reference's state-dict keys; the published files cannot be downloaded here):
    AutoModelForCausalLM.from_pretrained -> cuda -> pack_weights -> half precision, then save_packed / load_packed.
    The loaded weights are the saved ones (nothing is re-initialised or rescaled on load), logits equal those of a
    model built directly from the same state dict, the oracle agrees, and the packed file reproduces them exactly."""
    from transformers import AutoModelForCausalLM
    from mmfreelm.models import HGRNBitConfig, HGRNBitForCausalLM
    from matmulfreellm_b200 import checkpoint
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=41)
    sd["model.lower_bounds"] = 0.3 * torch.randn(2, 256, generator=torch.Generator().manual_seed(2))
    src = HGRNBitForCausalLM(HGRNBitConfig(vocab_size=cfg.vocab_size, hidden_size=cfg.hidden_size,
                                           num_hidden_layers=cfg.num_hidden_layers, intermediate_size=cfg.intermediate_size,
                                           rms_norm_eps=cfg.rms_norm_eps)).eval()
    src.load_state_dict(sd, strict=True)
    hf_dir = str(tmp_path / "hf")
    src.to(ckpt_dtype).save_pretrained(hf_dir)
    stored = {k: v.to(ckpt_dtype) for k, v in sd.items()}            # what the file holds

    loaded = AutoModelForCausalLM.from_pretrained(hf_dir, dtype=ckpt_dtype).eval()
    assert type(loaded).__name__ == "HGRNBitForCausalLM" and loaded.config.model_type == "hgrn_bit"
    got = loaded.state_dict()
    assert sorted(got) == sorted(stored)
    for k in stored:
        assert torch.equal(got[k], stored[k]), k                       # includes o_proj / down_proj: no second rescale
    loaded = loaded.cuda()
    loaded.pack_weights()                                              # ternarise from the checkpoint's own precision
    loaded = loaded.bfloat16()
    direct = build_gpu_model({k: v.float() for k, v in stored.items()}, cfg, torch.bfloat16)
    ids = torch.randint(0, 32000, (2, 24), generator=torch.Generator().manual_seed(5)).cuda()
    a, b = loaded(ids, use_cache=True), direct(ids, use_cache=True)
    assert torch.equal(a.logits, b.logits)
    oracle = O.OracleHGRNBit(cfg, {k: v.float() for k, v in stored.items()}, dtype=torch.bfloat16, linear="int", bitlinear_eps=1e-6)
    ref_logits, _ = oracle.forward(ids.cpu())
    _close_up_to_code_flips(a.logits.float().cpu().numpy(), ref_logits.float().numpy(), 1e-2, 1e-1)
    path = str(tmp_path / "m.mmfpack.npz")
    checkpoint.save_packed(loaded, path)
    again = checkpoint.load_packed(path, "cuda")
    c = again(ids, use_cache=True)
    assert torch.equal(a.logits, c.logits)
    for x, y in zip(a.past_key_values, c.past_key_values):
        assert torch.equal(x[0], y[0])
    # a checkpoint without lm_head.weight (tied embeddings were never part of the published models): loading reports it
    import os
    from safetensors.torch import load_file, save_file
    f = os.path.join(hf_dir, "model.safetensors")
    tensors = load_file(f)
    del tensors["lm_head.weight"]
    save_file(tensors, f, metadata={"format": "pt"})
    _, info = AutoModelForCausalLM.from_pretrained(hf_dir, dtype=ckpt_dtype, output_loading_info=True)
    assert "lm_head.weight" in info["missing_keys"]


def test_inplace_weight_change_is_repacked_without_an_explicit_call(mm):
    """The reference re-ternarises on every forward.  Here codes are cached, so a weight that is replaced or modified in
    place after a forward (load_state_dict, weight.mul_) must be repacked on the next forward without anyone calling
    pack_weights(): logits then match the oracle for the NEW weights."""
    cfg = tiny_cfg()
    sd1, sd2 = O.random_weights(cfg, seed=51), O.random_weights(cfg, seed=52)
    model = build_gpu_model(sd1, cfg, torch.float32)
    ids = torch.randint(0, 32000, (2, 20), generator=torch.Generator().manual_seed(7))
    first = model(ids.cuda(), use_cache=False).logits
    model.load_state_dict({k: v.cuda() for k, v in sd2.items()}, strict=True)          # no pack_weights() afterwards
    second = model(ids.cuda(), use_cache=False).logits
    assert not torch.equal(first, second)
    ref, _ = O.OracleHGRNBit(cfg, sd2, dtype=torch.float32, linear="int", bitlinear_eps=1e-6).forward(ids)
    _close_up_to_code_flips(second.cpu().numpy(), ref.numpy(), 2e-6, 2e-2)
    with torch.no_grad():
        model.lm_head.weight.mul_(-1.0)                                                  # in-place edit of one weight
    third = model(ids.cuda(), use_cache=False).logits
    assert torch.equal(third, -second)                                                   # codes flip sign, scale unchanged
    # a cast keeps codes that pack_weights() made from fp32: same tokens before and after .bfloat16() up to bf16 rounding
    model.pack_weights()
    codes_before = mm.kernels.unpack_codes(model.lm_head.packed()).clone()
    model = model.bfloat16()
    assert torch.equal(mm.kernels.unpack_codes(model.lm_head.packed()), codes_before)


def test_decoder_replays_repeated_prompt_lengths_from_a_graph(mm):
    """GreedyDecoder runs the first prompt of a length eagerly and captures the pass on the second one; every later
    prompt of that length is a graph replay.  Eager, captured and replayed passes give identical tokens, a prompt starts
    from the zero state whatever ran before, and other lengths are unaffected."""
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=3)
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    g = torch.Generator().manual_seed(9)
    prompts = [torch.randint(0, 32000, (3, 12), generator=g).cuda() for _ in range(4)]
    other = torch.randint(0, 32000, (3, 7), generator=g).cuda()
    ref = GreedyDecoder(model, 3, use_graph=False)
    want = [ref.generate(p, 6) for p in prompts]
    want_other = ref.generate(other, 6)
    dec = GreedyDecoder(model, 3)
    got = [dec.generate(prompts[0], 6), dec.generate(prompts[1], 6)]      # eager, then capture + replay
    assert 12 in dec._prompt_graphs
    got.append(dec.generate(other, 6))                                     # another length in between (eager)
    got += [dec.generate(prompts[2], 6), dec.generate(prompts[3], 6)]      # replays
    assert 7 not in dec._prompt_graphs
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert torch.equal(got[2], want_other)
    assert torch.equal(got[3], want[2]) and torch.equal(got[4], want[3])
    mm.kernels.check_status()


def test_prompt_graph_with_the_persistent_contraction(mm):
    """A prompt of 8 x 256 tokens on 2048-wide layers is large enough for the persistent contraction kernel (clusters of
    two CTAs, programmatic dependent launch); captured in the decoder's prompt graph and replayed it gives the tokens of the
    eager pass."""
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = O.OracleConfig(vocab_size=32000, hidden_size=2048, num_hidden_layers=1, intermediate_size=5632)
    sd = O.random_weights(cfg, seed=17)
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    g = torch.Generator().manual_seed(18)
    prompts = [torch.randint(0, 32000, (8, 256), generator=g).cuda() for _ in range(3)]
    ref = GreedyDecoder(model, 8, use_graph=False)
    want = [ref.generate(p, 4) for p in prompts]
    dec = GreedyDecoder(model, 8)
    got = [dec.generate(p, 4) for p in prompts]          # eager, capture + replay, replay
    assert 256 in dec._prompt_graphs
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    mm.kernels.check_status()


def test_decoder_step_driven_from_pinned_host_buffers(mm):
    """`GreedyDecoder.step_host`: ids in from pinned host memory, new tokens out to pinned host memory, the two copies
    captured in the same CUDA graph as the step — the token stream equals the device-resident loop, and unpinned or
    misshaped buffers are refused."""
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=8)
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    ids = torch.randint(0, 32000, (3, 7), generator=torch.Generator().manual_seed(3)).cuda()
    ref = GreedyDecoder(model, 3)
    want = [ref.prefill(ids).clone()]
    for _ in range(12):
        want.append(ref.step().clone())
    dec = GreedyDecoder(model, 3)
    ids_host = torch.empty(3, 1, dtype=torch.int64).pin_memory()
    out_host = torch.empty(3, dtype=torch.int64).pin_memory()
    first = dec.prefill(ids).cpu()
    assert torch.equal(first, want[0].cpu())
    ids_host.copy_(first[:, None])
    for t in range(12):
        dec.step_host(ids_host, out_host)
        torch.cuda.current_stream().synchronize()
        assert torch.equal(out_host, want[t + 1].cpu()), t
        ids_host.copy_(out_host[:, None])
    with pytest.raises(ValueError):
        dec.step_host(torch.empty(3, 1, dtype=torch.int64), out_host)
    with pytest.raises(ValueError):
        dec.step_host(ids_host, torch.empty(4, dtype=torch.int64).pin_memory())


def test_last_logits_follow_the_graph_that_ran(mm):
    """`GreedyDecoder.last_logits` after every kind of step is the logits of that step, whichever graphs were captured before:
    the token of the step is their arg-max, and they equal those of a decoder without graphs bit for bit."""
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=27), cfg, torch.bfloat16)
    g = torch.Generator().manual_seed(5)
    B = 3
    prompts = [torch.randint(0, cfg.vocab_size, (B, 7), generator=g).cuda() for _ in range(4)]
    dec, eager = GreedyDecoder(model, B), GreedyDecoder(model, B, use_graph=False)
    ids_host = torch.zeros(B, 1, dtype=torch.int64).pin_memory()
    out_host = torch.zeros(B, dtype=torch.int64).pin_memory()

    def advance(kind):
        for d in (dec, eager):
            if kind == "host":
                ids_host.copy_(d.ids)
                torch.cuda.synchronize()
                d.step_host(ids_host, out_host)
                torch.cuda.synchronize()
            elif kind == "step":
                d.step()
            else:
                d.prefill(prompts[kind])
        assert torch.equal(dec.last_logits, eager.last_logits), kind
        assert torch.equal(dec.last_logits.gather(1, dec.ids)[:, 0], dec.last_logits.amax(1)), kind

    for kind in (0, "host", 1, "host", "step", "host", "step", 2, "step", "step", 3, "host"):
        advance(kind)
    out = model(input_ids=prompts[0], use_cache=True, last_token_only=True)
    dec.seed(out.past_key_values, out.logits[:, -1])
    assert torch.equal(dec.last_logits, out.logits[:, -1])


@pytest.mark.parametrize("fuse", [True, False])
def test_captured_graphs_keep_the_weights_they_read(mm, fuse):
    """Packed weights that were replaced stay alive while a decoder holds a graph that reads them (only their lifetime is looked
    at), and no longer."""
    import gc
    import weakref
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=4), cfg, torch.bfloat16)
    model.fuse = fuse
    ids = torch.randint(0, cfg.vocab_size, (2, 6), device="cuda")
    out_host = torch.zeros(2, dtype=torch.int64).pin_memory()

    def step(dec):
        dec.step()

    def host(dec):
        dec.step_host(torch.zeros(2, 1, dtype=torch.int64).pin_memory(), out_host)

    def prompt(dec):
        dec.prefill(ids)
        dec.prefill(ids)

    with torch.no_grad():
        for capture in (step, host, prompt):
            dec = GreedyDecoder(model, 2)
            capture(dec)
            torch.cuda.synchronize()
            read = [weakref.ref(model._fused_runner)] if fuse else \
                [weakref.ref(m._packed) for m in model.modules() if getattr(m, "_packed", None) is not None]
            for p in model.parameters():
                p.mul_(0.5)
            model(input_ids=ids)                      # repacks
            gc.collect()
            assert all(r() is not None for r in read), capture
            del dec
            gc.collect()
            assert all(r() is None for r in read), capture


def test_native_calls_check_the_device(mm):
    """On a GPU that the library was not built for, the calls that go through the native host path raise the device check's
    error, as the others do (the check is made to fail here: it runs once per device)."""
    from matmulfreellm_b200 import _lib, kernels
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=4), cfg, torch.bfloat16)
    ids = torch.zeros(1, 3, dtype=torch.int64, device="cuda")
    model(input_ids=ids)
    layer = model.model.layers[0].mlp.down_proj
    x = torch.randn(2, 8, cfg.intermediate_size, device="cuda").bfloat16()

    def refuse(index):
        assert index == torch.cuda.current_device()
        raise _lib.MMFreeError("mmf_check_device", -5, "built for sm_100a only")

    native = _lib.native()
    calls = (lambda: layer(x), lambda: layer(x[0, :1]), lambda: kernels.hgrn_scan(x, x, None, True, False), lambda: model(input_ids=ids))
    native.set_hooks(_lib.MMFreeError, kernels.stream_workspace, refuse)
    try:
        for fn in calls:
            with pytest.raises(_lib.MMFreeError, match="mmf_check_device failed with MMF_ERR_ARCH"):
                fn()
    finally:
        native.set_hooks(_lib.MMFreeError, kernels.stream_workspace, _lib.require_device)
    for fn in calls:
        fn()


def test_forwards_from_several_threads(mm):
    """A forward releases the GIL while it launches: four threads on streams of their own, sharing one model, get what one thread gets."""
    import threading
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=9), cfg, torch.bfloat16)
    layer = model.model.layers[0].mlp.down_proj
    g = torch.Generator().manual_seed(2)
    work = [torch.randint(0, cfg.vocab_size, shape, generator=g).cuda() for shape in ((1, 1), (2, 1), (5, 1), (12, 1), (33, 1), (3, 40), (1, 300), (8, 150))]
    rows = [torch.randn(m, cfg.intermediate_size, generator=g).bfloat16().cuda() for m in (1, 2, 7, 200)]

    def one_pass():
        with torch.no_grad():
            return [model(input_ids=ids).logits for ids in work] + [layer(x) for x in rows]

    want = one_pass()
    torch.cuda.synchronize()
    wrong = []

    def thread(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    got = one_pass()
                    torch.cuda.current_stream().synchronize()
                    wrong.extend((k, i) for i, (a, b) in enumerate(zip(got, want)) if not torch.equal(a, b))
        except Exception as e:                       # noqa: BLE001 - reported by the assertion below
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=thread, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_launch_count_is_the_number_of_kernels(mm):
    """`_lib.launch_count`, which the benchmark reports, advances by the kernels that a call really launches: the kernel nodes
    of a graph captured from it (time-split scans make two passes; a forward of one, four or 32 rows takes different chains)."""
    from cuda.bindings import runtime as rt
    from matmulfreellm_b200 import _lib, kernels
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=4), cfg, torch.bfloat16)
    layer = model.model.layers[0].mlp.down_proj
    g = torch.Generator(device="cuda").manual_seed(1)

    def scan(B, T, D, into=None):
        x = torch.randn(B, T, D, generator=g, device="cuda").bfloat16()
        gate = torch.rand(B, T, D, generator=g, device="cuda").bfloat16()
        return lambda: kernels.hgrn_scan(x, gate, None, True, False, torch.float32, into)

    def gated(B, T, D):
        x, s = torch.randn(B, T, 2 * D, generator=g, device="cuda").bfloat16(), torch.zeros(B, D, device="cuda")
        return lambda: kernels.hgrn_gated(x[:, :, :D], x[:, :, D:], None, s)

    def forward(B, T):
        ids = torch.randint(0, cfg.vocab_size, (B, T), device="cuda")
        cache = model.model.init_cache(B)
        return lambda: model(input_ids=ids, past_key_values=cache, use_cache=True)

    def linear(M):
        x = torch.randn(M, cfg.intermediate_size, generator=g, device="cuda").bfloat16()
        return lambda: layer(x)

    calls = {"scan, split": scan(1, 2048, 128), "scan": scan(8, 64, 128), "scan of one step": scan(3, 1, 128),
             "scan into a given state": scan(1, 2048, 128, torch.empty(1, 128, device="cuda")), "gated, split": gated(1, 1024, 64),
             "prompt, split": forward(1, 1024), "prompt": forward(2, 40), "step of 1": forward(1, 1), "step of 4": forward(4, 1),
             "step of 12": forward(12, 1), "step of 32": forward(32, 1), "linear 1": linear(1), "linear 5": linear(5)}
    side = torch.cuda.Stream()
    with torch.no_grad():
        for name, call in calls.items():
            with torch.cuda.stream(side):
                call()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph(keep_graph=True)
            with torch.cuda.graph(graph, stream=side):
                before = _lib.launch_count
                call()
                counted = _lib.launch_count - before
            raw = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
            err, _, n = rt.cudaGraphGetNodes(raw, 0)
            err, nodes, n = rt.cudaGraphGetNodes(raw, n)
            kinds = [rt.cudaGraphNodeGetType(node)[1] for node in nodes[:n]]
            assert counted == sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds), name


def test_generate_graph_path_equals_step_loop(mm):
    """`generate` replays greedy decode steps from a CUDA graph; tokens, the handling of eos (finished sequences
    keep emitting it, the result ends where the last sequence finishes) and left-padded prompts must equal the
    step-by-step loop, also when batch sizes alternate and after the weights change."""
    cfg = tiny_cfg()
    sd = O.random_weights(cfg, seed=4)
    model = build_gpu_model(sd, cfg, torch.bfloat16)
    g = torch.Generator().manual_seed(2)
    ids3 = torch.randint(0, 32000, (3, 9), generator=g).cuda()
    ids5 = torch.randint(0, 32000, (5, 4), generator=g).cuda()
    for ids in (ids3, ids5, ids3):
        want = model.generate(ids, max_new_tokens=40, use_graph=False)
        got = model.generate(ids, max_new_tokens=40)
        assert torch.equal(got, want)
        new = want[:, ids.shape[1]:]
        # eos choices: a token every sequence emits at some step (cuts the result), one that only one sequence
        # emits (that sequence is padded with it), one that never appears
        common = [t for t in new[0].tolist() if all(t in row for row in new.tolist())]
        for eos in ([common[0]] if common else []) + [int(new[1, 3]), 31999]:
            a = model.generate(ids, max_new_tokens=40, eos_token_id=eos, use_graph=False)
            b = model.generate(ids, max_new_tokens=40, eos_token_id=eos)
            assert torch.equal(a, b), eos
    assert len([k for k in model._greedy_decoders if k != "key"]) == 2
    mask = torch.ones(3, 9, dtype=torch.int64, device="cuda")
    mask[0, :4] = 0
    mask[2, :1] = 0
    assert torch.equal(model.generate(ids3, max_new_tokens=12, attention_mask=mask),
                       model.generate(ids3, max_new_tokens=12, attention_mask=mask, use_graph=False))
    # sampling through the graph decoder draws the same random numbers in the same order as the step loop
    for eos in (None, int(want[0, -3])):
        g1 = torch.Generator(device="cuda").manual_seed(11)
        g2 = torch.Generator(device="cuda").manual_seed(11)
        a = model.generate(ids3, max_new_tokens=24, do_sample=True, top_p=0.8, temperature=0.9, generator=g1, eos_token_id=eos)
        b = model.generate(ids3, max_new_tokens=24, do_sample=True, top_p=0.8, temperature=0.9, generator=g2, eos_token_id=eos,
                           use_graph=False)
        assert torch.equal(a, b), eos
    # new weights: the cached decoders (graphs with the old weight pointers baked in) must not be reused
    with torch.no_grad():
        model.model.layers[0].mlp.down_proj.weight.mul_(-1.0)
    model.pack_weights()
    assert torch.equal(model.generate(ids3, max_new_tokens=12), model.generate(ids3, max_new_tokens=12, use_graph=False))
    mm.kernels.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hidden,intermediate", [(384, 704), (1152, 1984), (2176, 4160), (4096, 8192)])
def test_decode_step_rows_do_not_depend_on_the_batch(mm, dtype, hidden, intermediate):
    """A decode step picks its kernels by the number of sequences (row work inside the contraction, in a kernel of its own,
    or tcgen05 contractions above 16 rows).  All take the same roundings, so a sequence's logits and state are bit-identical
    whatever the batch around it; sizes with partly filled column groups, row tiles and 16-row blocks."""
    from mmfreelm.models import HGRNBitConfig, HGRNBitForCausalLM
    torch.manual_seed(hidden)
    model = HGRNBitForCausalLM(HGRNBitConfig(vocab_size=1003, hidden_size=hidden, num_hidden_layers=2, intermediate_size=intermediate,
                                             use_lower_bound=True)).eval().cuda()
    with torch.no_grad():
        for n, p in model.named_parameters():
            if "lower_bounds" in n or p.dim() == 1: p.add_(0.3 * torch.randn_like(p))
    model.pack_weights()
    model = model.to(dtype)
    g = torch.Generator().manual_seed(7)
    ids, step = torch.randint(0, 1003, (33, 5), generator=g).cuda(), torch.randint(0, 1003, (33, 1), generator=g).cuda()

    def run(B, embeds):
        past = model(ids[:B], use_cache=True).past_key_values
        mask = torch.ones(B, 1, dtype=torch.long, device="cuda")
        mask[B // 2] = 0
        kw = {"inputs_embeds": model.get_input_embeddings()(step[:B])} if embeds else {"input_ids": step[:B]}
        out = model(past_key_values=past, use_cache=True, attention_mask=mask if embeds else None, **kw)
        return out.logits, [s[0].view(B, -1) for s in out.past_key_values]

    ref, ref_states = run(33, False)
    for B in (1, 2, 3, 8, 9, 16):
        logits, states = run(B, False)
        assert torch.equal(logits, ref[:B]), B
        assert all(torch.equal(a, b[:B]) for a, b in zip(states, ref_states)), B
        logits, _ = run(B, True)                     # embeddings given, one sequence's token is padding
        keep = [i for i in range(B) if i != B // 2]
        assert torch.equal(logits[keep], ref[keep]), B


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hidden,intermediate", [(128, 64), (640, 6144), (2048, 6208), (2560, 6912)])
def test_resident_decode_step_at_the_ends_of_its_range(mm, dtype, hidden, intermediate):
    """All blocks of a step in one kernel (up to 16 sequences) against the chain of kernels that 33 sequences take, bit for bit: fewer channel
    pairs than SMs, the longest inner row of eight warps and one beyond it, the widest rows; one row, one tile of eight, a row more."""
    from matmulfreellm_b200 import _lib
    from mmfreelm.models import HGRNBitConfig, HGRNBitForCausalLM
    torch.manual_seed(hidden)
    model = HGRNBitForCausalLM(HGRNBitConfig(vocab_size=300, hidden_size=hidden, num_hidden_layers=3, intermediate_size=intermediate)).eval().cuda()
    with torch.no_grad():
        for n, p in model.named_parameters():
            if "lower_bounds" in n or p.dim() == 1: p.add_(0.3 * torch.randn_like(p))
    model.pack_weights()
    model = model.to(dtype)
    g = torch.Generator().manual_seed(7)
    ids, step = torch.randint(0, 300, (33, 3), generator=g).cuda(), torch.randint(0, 300, (2, 33, 1), generator=g).cuda()

    def run(B):
        past = model(ids[:B], use_cache=True).past_key_values
        for s in step:
            out = model(input_ids=s[:B], past_key_values=past, use_cache=True)
        return out.logits, [s[0].view(B, -1) for s in out.past_key_values]

    ref, ref_states = run(33)
    for B in (1, 2, 8, 9, 16):
        taken = _lib.load().mmf_decode_step_workspace_bytes(B, hidden, intermediate, 3) > 0
        assert taken == ((B <= 8 or hidden < 2560) and (B != 2 or hidden > 1024)), B
        logits, states = run(B)
        assert torch.equal(logits, ref[:B]), B
        assert all(torch.equal(a, b[:B]) for a, b in zip(states, ref_states)), B
    mm.kernels.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K,N", [(64, 1), (704, 130), (2112, 37), (5632, 2048), (8192, 515)])
def test_bitlinear_of_one_and_two_rows_equals_more_rows(mm, dtype, K, N):
    from matmulfreellm_b200.ops.fusedbitnet import FusedBitLinear
    torch.manual_seed(K)
    layer = FusedBitLinear(K, N).cuda()
    layer.pack_weights()
    layer = layer.to(dtype)
    x = torch.randn(40, K, device="cuda").to(dtype)
    ref = layer(x)
    for rows in (x[:1], x[:2], x[::7][:2]):
        pick = ref[:rows.shape[0]] if rows.stride(0) == K or rows.shape[0] == 1 else ref[::7][:2]
        assert torch.equal(layer(rows), pick)


def test_resident_decode_step_whose_waits_give_up(mm):
    """A step whose waits run out ends by itself, sets the status word and leaves the GPU usable: with a limit of one poll every wait that does
    not find its words at once gives up (with several rows most CTAs look for codes long before they are made)."""
    from matmulfreellm_b200 import _lib
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=4), cfg, torch.bfloat16)
    for B in (1, 5, 16):
        prompt, ids = torch.randint(0, 32000, (B, 7), device="cuda"), torch.randint(0, 32000, (B, 1), device="cuda")

        def step():
            past = model(prompt, use_cache=True).past_key_values
            torch.cuda.synchronize()
            with _lib.experiments_library() as lib:
                lib.mmf_tuning(13, limit)
                out = model(input_ids=ids, past_key_values=past, use_cache=True)
                torch.cuda.synchronize()
            return out.logits

        limit = 0
        want = step()
        mm.kernels.check_status()
        limit = 1
        step()
        if B > 1:
            with pytest.raises(_lib.MMFreeError, match="MMF_ERR_TIMEOUT"):
                mm.kernels.check_status()
        else:                                   # (one sequence's words may all be there at the first look)
            mm.kernels._rezero_workspaces()
            _lib.native().take_gave_up()
        limit = 0
        assert torch.equal(step(), want)
        mm.kernels.check_status()


def test_step_that_gave_up_is_reported_by_the_next_call(mm):
    """Without anyone asking for the status word: a forward, a decoder's step (eager and replayed) and `generate` raise once a step of that
    device has given up, and work again afterwards."""
    from matmulfreellm_b200 import _lib
    from matmulfreellm_b200.engine import GreedyDecoder
    cfg = tiny_cfg()
    model = build_gpu_model(O.random_weights(cfg, seed=4), cfg, torch.bfloat16)
    prompt = torch.randint(0, 32000, (5, 7), device="cuda")
    host = torch.zeros(5, 1, dtype=torch.int64).pin_memory(), torch.zeros(5, dtype=torch.int64).pin_memory()
    eager, graph = GreedyDecoder(model, 5, use_graph=False), GreedyDecoder(model, 5)
    calls = {"forward": lambda: model(prompt[:1, :1]), "prompt": lambda: model(prompt), "decoder": eager.step, "graph": graph.step,
             "host buffers": lambda: graph.step_host(*host), "generate": lambda: model.generate(prompt, max_new_tokens=4)}
    for call in calls.values():
        call()
    for name, call in calls.items():
        past = model(prompt, use_cache=True).past_key_values
        with _lib.experiments_library() as lib:
            lib.mmf_tuning(13, 1)
            model(input_ids=prompt[:, :1], past_key_values=past, use_cache=True)
            torch.cuda.synchronize()
        with pytest.raises(_lib.MMFreeError, match="mmf_decode_step failed with MMF_ERR_TIMEOUT"):
            call()
        assert all(not ws[:4].any() for ws in mm.kernels._ws_cache.values()), name
        call()
        torch.cuda.synchronize()
        mm.kernels.check_status()


def _resident_model(resident=True):
    """Ten blocks whose packed weights (33 MB) are larger than what the allocator keeps for the scratch of a few tokens."""
    from mmfreelm.models import HGRNBitConfig, HGRNBitForCausalLM
    torch.manual_seed(5)
    with torch.device("cuda"):
        model = HGRNBitForCausalLM(HGRNBitConfig(vocab_size=1003, hidden_size=1024, num_hidden_layers=10, intermediate_size=2816)).eval()
    model.pack_weights()
    model.resident_step = resident
    return model.bfloat16()


def _one_step(model, ids):
    """(logits, states, kernels launched) of a cached step after a fixed prompt."""
    from matmulfreellm_b200 import _lib
    past = model(torch.arange(ids.shape[0] * 3, device="cuda").view(-1, 3), use_cache=True).past_key_values
    torch.cuda.synchronize()
    before = _lib.launch_count
    out = model(input_ids=ids, past_key_values=past, use_cache=True)
    return out.logits, [s[0].clone() for s in out.past_key_values], _lib.launch_count - before


def _same_step(a, b):
    return torch.equal(a[0], b[0]) and all(torch.equal(x, y) for x, y in zip(a[1], b[1]))


def test_second_copy_of_the_weights_is_made_by_the_first_step_that_reads_it(mm):
    """Prompts, larger batches, two rows of 1024 (which the resident kernel does not take) and a model that was told not to hold no copy."""
    from matmulfreellm_b200.engine import GreedyDecoder
    ids = torch.arange(33, device="cuda").view(33, 1)
    for resident in (False, True):
        model = _resident_model(resident)
        copy = sum(m._packed.packed.numel() for n, m in model.named_modules() if hasattr(m, "_packed") and "lm_head" not in n)

        def held(*batches):
            before = torch.cuda.memory_allocated()
            for b in batches:
                _one_step(model, ids[:b])
            torch.cuda.synchronize()
            return torch.cuda.memory_allocated() - before >= copy

        model(ids[:2])                                       # the runner
        assert copy > 30 << 20 and not held(33, 2, 17)
        assert model.prepare_step(ids[:2]) is False and not held(2)
        assert held(16) == resident and not held(1, 16, 4)
        assert model.prepare_step(ids[:1]) is resident
        steps = [_one_step(model, ids[:b])[2] for b in (1, 16)]
        assert (max(steps) < 10) == resident and (min(steps) > 40) != resident
        if resident:                                         # told not to: the copy goes with the runner
            model.resident_step = False
            dec = GreedyDecoder(model, 4)
            dec.prefill(ids[:4])
            dec.step()
            assert dec.kernels_per_step > 40
        del model


def test_step_without_memory_for_the_second_copy(mm):
    """A step that fitted without the copy of the weights still runs where the copy cannot be allocated, with the same results; a model that is
    told to try again (a new runner) takes the resident kernel."""
    ids = torch.arange(5, device="cuda").view(5, 1)
    want = _one_step(_resident_model(False), ids)
    model = _resident_model()
    _one_step(model, ids.repeat(5, 1))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total, held = torch.cuda.mem_get_info()[1], []
    try:
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
        with pytest.raises(torch.OutOfMemoryError):          # no hole that earlier tests left is as large as the copy (33 MB)
            while True:
                held.append(torch.empty(16 << 20, dtype=torch.uint8, device="cuda"))
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (24 << 20)) / total)
        got = _one_step(model, ids)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        del held
    assert _same_step(got, want) and got[2] == want[2]
    again = _one_step(model, ids)                            # (not tried on every step)
    assert _same_step(again, want) and again[2] == want[2]
    model.resident_step = False
    _one_step(model, ids)
    model.resident_step = True
    again = _one_step(model, ids)
    assert _same_step(again, want) and again[2] < want[2]


def test_first_step_under_capture(mm):
    """A step that a user's own graph captures before any other has run: no allocation and no packing become part of the graph."""
    ids = torch.arange(5, device="cuda").view(5, 1)
    want = _one_step(_resident_model(False), ids)
    model = _resident_model()
    past = model(torch.arange(15, device="cuda").view(5, 3), use_cache=True).past_key_values
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        model(torch.arange(40, device="cuda").view(8, 5))    # this stream's workspace
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = model(input_ids=ids, past_key_values=past, use_cache=True)
    graph.replay()
    assert torch.equal(out.logits, want[0]) and all(torch.equal(s[0], w) for s, w in zip(out.past_key_values, want[1]))
    assert _one_step(model, ids)[2] < 10


def test_first_steps_of_several_threads(mm):
    """Threads on streams of their own that all meet a model without the copy: one makes it, and none reads it before it is complete."""
    import threading
    ids = torch.arange(16, device="cuda").view(16, 1)
    want = {B: _one_step(_resident_model(False), ids[:B]) for B in (1, 3, 8, 16)}
    for _ in range(3):
        model = _resident_model()
        model(ids[:3])
        del model._fused_runner
        model(ids.repeat(3, 1))                              # a new runner
        torch.cuda.synchronize()
        start, wrong = threading.Barrier(4), []

        def thread(B):
            try:
                with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
                    past = model(torch.arange(B * 3, device="cuda").view(-1, 3), use_cache=True).past_key_values
                    torch.cuda.current_stream().synchronize()
                    start.wait()
                    out = model(input_ids=ids[:B], past_key_values=past, use_cache=True)
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(out.logits, want[B][0]): wrong.append(B)
            except Exception as e:                           # noqa: BLE001 - reported by the assertion below
                wrong.append((B, repr(e)))

        threads = [threading.Thread(target=thread, args=(B,)) for B in want]
        for t in threads: t.start()
        for t in threads: t.join()
        assert not wrong


def test_step_whose_cooperative_launch_is_refused(mm):
    """Where the context cannot hold all CTAs of the resident kernel (the refusal is answered by the experiments build; nothing is launched) the
    call runs as the chain of kernels, and so do the later ones of the model, eager and captured."""
    from matmulfreellm_b200 import _lib
    from matmulfreellm_b200.engine import GreedyDecoder
    ids = torch.arange(16, device="cuda").view(16, 1)
    plain = _resident_model(False)
    for B in (1, 16):
        want = _one_step(plain, ids[:B])
        model = _resident_model()
        with _lib.experiments_library() as lib:
            lib.mmf_tuning(14, 1)
            got = _one_step(model, ids[:B])
            dec = GreedyDecoder(model, B)
            dec.prefill(ids[:B])
            dec.step()
        assert _same_step(got, want) and got[2] == want[2] + 1           # the fill in front of the refused launch
        got = _one_step(model, ids[:B])
        assert _same_step(got, want) and got[2] == want[2]
        assert dec.kernels_per_step > 40 and model.prepare_step(ids[:B]) is False
    mm.kernels.check_status()


@pytest.mark.parametrize("bad_weights", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_resident_decode_step_with_infinities_and_nan(mm, dtype, bad_weights):
    """The words that CTAs hand to one another say by their value that they have arrived, so no value that a step can form may look like an
    absent one, which would be waited for in vain.  Embeddings, states and norm weights that are infinite, NaN, as large as the type holds,
    subnormal or zero: every wait ends, and outputs and states are those of the chain of kernels, NaN for NaN."""
    from mmfreelm.models import HGRNBitConfig, HGRNBitForCausalLM
    torch.manual_seed(3)
    D, inf, nan, top = 640, float("inf"), float("nan"), torch.finfo(dtype).max
    model = HGRNBitForCausalLM(HGRNBitConfig(vocab_size=40, hidden_size=D, num_hidden_layers=3, intermediate_size=1984)).eval().cuda()
    model.pack_weights()
    model = model.to(dtype)
    special = [inf, -inf, nan, -nan, top, -top, torch.finfo(dtype).smallest_normal / 4, 0.0, -0.0]
    g = torch.Generator().manual_seed(1)
    with torch.no_grad():
        emb = model.model.embeddings.weight
        for k, v in enumerate(special):
            emb[k, torch.randperm(D, generator=g)[:3].cuda()] = v        # a few entries of a row, a whole row, a row with all of them
            emb[10 + k] = v
        emb[20, :len(special)] = torch.tensor(special, device="cuda").to(dtype)
        if bad_weights:
            for k, (n, p) in enumerate((n, p) for n, p in model.named_parameters() if n.endswith("norm.weight")):
                p[torch.randperm(p.numel(), generator=g)[:2].cuda()] = special[k % len(special)]

    def run(ids, states, resident):
        model.resident_step = resident
        past = model.model.init_cache(len(ids))
        for (s,), v in zip(past.states, states):
            s.copy_(v.view_as(s))
        for _ in range(2):
            out = model(input_ids=ids, past_key_values=past, use_cache=True)
        mm.kernels.check_status()
        return [out.logits, *(s[0] for s in past.states)]

    batches = [[k] for k in range(21)] + [[k, k + 10, 30, 20, 31] for k in range(9)] + [list(range(16)), list(range(5, 21))]
    for rows in batches:
        ids = torch.tensor(rows, device="cuda").view(-1, 1)
        states = [torch.randn(len(rows), D, generator=g).cuda() for _ in range(3)]
        for k, s in enumerate(states):
            s.view(-1)[k::97] = special[(rows[0] + k) % len(special)]
        got, want = (run(ids, states, r) for r in (True, False))
        for a, b in zip(got, want):
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(7.0), b.nan_to_num(7.0)), rows
