"""The work that users of this package have it do, as measurable cases.

A case is a plain dict.  Its `kind` names the public entry point, the other keys are sizes, data types and options:

  bitlinear   FusedBitLinear.forward on `rows` token rows (a layer of a user's own model, or a leaf swapped into the
              reference's files)
  hgrn        chunk_hgrn (`log_gate`) / fused_recurrent_hgrn on [batch, 1, time, width]
  decode      GreedyDecoder.step: one token for every sequence of a serving batch, state resident on the device
  step        HGRNBitForCausalLM.forward with past_key_values: one cached step of a user's own generation loop
  prompt      HGRNBitForCausalLM.forward over a batch of prompts, logits of the last or of all positions
  generate    HGRNBitForCausalLM.generate: prompt pass and decoding, greedy or nucleus sampling

Weights are random (no checkpoint ships with the package) with the distribution the configurations name: latent weights
N(0, 0.02), ternarised and packed once; norm weights near one, lower bounds as training moves them.
"""
import math

import torch

from matmulfreellm_b200.engine import GreedyDecoder
from matmulfreellm_b200.models import HGRNBitConfig, HGRNBitForCausalLM
from matmulfreellm_b200.ops.fusedbitnet import BitLinear, FusedBitLinear
from matmulfreellm_b200.ops.hgrn import chunk_hgrn, fused_recurrent_hgrn

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
VOCAB = 32000
# the three configurations of the repository: hidden, intermediate, blocks
MODELS = {"tiny": (256, 704, 2), "1.3b": (2048, 5632, 24), "2.7b": (2560, 6912, 32)}
# the layers of those models: (in_features, out_features)
LAYERS = ((2048, 2048), (2048, 11264), (5632, 2048), (2560, 2560), (2560, 13824), (6912, 2560), (256, 1408), (704, 256))


def listed():
    return [
        # one attention projection of one new token: the smallest call, all latency and launches
        {"name": "bitlinear_1_row", "kind": "bitlinear", "rows": 1, "k": 2048, "n": 2048, "dtype": "bf16"},
        # the widest layer on a ragged batch of short prompts in half precision
        {"name": "bitlinear_300_rows", "kind": "bitlinear", "rows": 300, "k": 2048, "n": 11264, "dtype": "fp16"},
        # the layer with the longest contraction over a full prompt batch
        {"name": "bitlinear_16384_rows", "kind": "bitlinear", "rows": 16384, "k": 5632, "n": 2048, "dtype": "bf16"},
        # the recurrence over prompts, log-gate convention
        {"name": "chunk_hgrn_2048", "kind": "hgrn", "log_gate": True, "batch": 8, "time": 2048, "width": 2048, "dtype": "bf16", "initial": False},
        # the recurrence continued from a state over an odd number of steps, linear gate, single precision
        {"name": "recurrent_hgrn_777", "kind": "hgrn", "log_gate": False, "batch": 5, "time": 777, "width": 2560, "dtype": "fp32", "initial": True},
        # one user talking to the model
        {"name": "decode_1", "kind": "decode", "model": "1.3b", "batch": 1, "dtype": "bf16"},
        # the serving batch of the benchmark
        {"name": "decode_32", "kind": "decode", "model": "1.3b", "batch": 32, "dtype": "bf16"},
        # the per-GPU share of the high-throughput configuration
        {"name": "decode_64_2.7b", "kind": "decode", "model": "2.7b", "batch": 64, "dtype": "bf16"},
        # a user's own loop around forward(past_key_values=...), as code written for the reference has it
        {"name": "step_4", "kind": "step", "model": "1.3b", "batch": 4, "dtype": "bf16"},
        # scoring a few left-padded texts: logits of every position, half precision
        {"name": "prompt_3x333_all", "kind": "prompt", "model": "1.3b", "batch": 3, "time": 333, "dtype": "fp16", "last_only": False, "masked": True},
        # the prompt pass of the benchmark
        {"name": "prompt_16x2048", "kind": "prompt", "model": "1.3b", "batch": 16, "time": 2048, "dtype": "bf16", "last_only": True, "masked": False},
        # a batch of questions answered with the sampling options of the reference's demo
        {"name": "generate_8", "kind": "generate", "model": "1.3b", "batch": 8, "time": 100, "new": 32, "dtype": "bf16", "sample": True},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _dtype(rng):
    return rng.choice(("bf16", "bf16", "fp16", "fp32"))


def draw(rng):
    kind = rng.choice(("bitlinear", "bitlinear", "hgrn", "decode", "decode", "step", "prompt", "prompt", "generate"))
    if kind == "bitlinear":
        k, n = rng.choice(LAYERS)
        return {"kind": kind, "rows": _log_int(rng, 1, 16384), "k": k, "n": n, "dtype": _dtype(rng)}
    if kind == "hgrn":
        width = rng.choice((256, 2048, 2560))
        batch = _log_int(rng, 1, 256)
        time = _log_int(rng, 1, max(1, min(8192, (8 * 8192 * 2048) // (batch * width))))
        return {"kind": kind, "log_gate": rng.random() < 0.5, "batch": batch, "time": time, "width": width, "dtype": _dtype(rng),
                "initial": rng.random() < 0.5}
    model = rng.choice(("tiny", "1.3b", "1.3b", "2.7b"))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    if kind == "decode":
        return {"kind": kind, "model": model, "batch": _log_int(rng, 1, 256), "dtype": dtype}
    if kind == "step":
        return {"kind": kind, "model": model, "batch": _log_int(rng, 1, 64), "dtype": dtype}
    if kind == "prompt":
        last_only = rng.random() < 0.5
        batch = _log_int(rng, 1, 16)
        rows = 4096 if not last_only else 15360 if model == "2.7b" else 32768
        return {"kind": kind, "model": model, "batch": batch, "time": _log_int(rng, 2, min(2048, rows // batch)), "dtype": dtype,
                "last_only": last_only, "masked": rng.random() < 0.5}
    return {"kind": kind, "model": model, "batch": _log_int(rng, 1, 32), "time": _log_int(rng, 4, 256), "new": rng.randint(8, 24),
            "dtype": dtype, "sample": rng.random() < 0.5}


# -- preparation ---------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda")


def _model(case, gen):
    """A model as a serving program holds it: packed from fp32 latent weights, then cast to the activation dtype."""
    hidden, inner, blocks = MODELS[case["model"]]
    with torch.device("cuda"):
        lm = HGRNBitForCausalLM(HGRNBitConfig(vocab_size=VOCAB, hidden_size=hidden, num_hidden_layers=blocks, intermediate_size=inner)).eval()
    with torch.no_grad():
        for m in lm.modules():
            if isinstance(m, BitLinear):
                m.weight.normal_(0.0, 0.02, generator=gen)
        lm.model.embeddings.weight.normal_(0.0, 0.02, generator=gen)
        lm.model.lower_bounds.normal_(0.0, 0.5, generator=gen)
        for name, p in lm.named_parameters():
            if name.endswith("norm.weight"):
                p.normal_(1.0, 0.05, generator=gen)
    lm.pack_weights()
    return lm.to(DTYPES[case["dtype"]])


def _ids(gen, batch, time):
    return torch.randint(0, VOCAB, (batch, time), generator=gen, device="cuda")


def prepare(case, seed):
    gen = _generator(seed)
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    state = dict(case)
    with torch.no_grad():
        if kind == "bitlinear":
            k, n = case["k"], case["n"]
            with torch.device("cuda"):
                layer = FusedBitLinear(k, n).eval()
            layer.weight.normal_(0.0, 0.02, generator=gen)
            layer.norm.weight.normal_(1.0, 0.05, generator=gen)
            layer.pack_weights()
            x = _randn(gen, case["rows"], k)
            outliers = torch.randperm(k, generator=gen, device="cuda")[: k // 100]     # 1 % of the channels, as activations have them
            x[:, outliers] *= 20.0
            state.update(layer=layer.to(dtype), x=x.to(dtype))
        elif kind == "hgrn":
            shape = (case["batch"], 1, case["time"], case["width"])
            g = torch.nn.functional.logsigmoid(_randn(gen, *shape))
            x = ((1.0 - g.exp()) * torch.nn.functional.silu(_randn(gen, *shape))).to(dtype)
            h0 = _randn(gen, case["batch"], 1, case["width"]) if case["initial"] else None
            state.update(x=x, g=g if case["log_gate"] else g.exp().to(dtype), h0=h0)
        else:
            lm = _model(case, gen)
            state["lm"] = lm
            batch = case["batch"]
            if kind == "decode":
                state["decoder"] = GreedyDecoder(lm, batch)
                state["decoder"].prefill(_ids(gen, batch, 16))
            elif kind == "step":
                out = lm(input_ids=_ids(gen, batch, 16), use_cache=True, last_token_only=True)
                state.update(past=out.past_key_values, ids=_ids(gen, batch, 1))
            else:
                time = case["time"]
                state["ids"] = _ids(gen, batch, time)
                if kind == "prompt" and case["masked"]:     # left padding: the first text is full, the others are shorter
                    pad = torch.randint(0, time // 2 + 1, (batch, 1), generator=gen, device="cuda")
                    pad[0] = 0
                    state["mask"] = (torch.arange(time, device="cuda")[None] >= pad).long()
                if kind == "generate":
                    state["generator"] = gen
    return state


# -- one pass ------------------------------------------------------------------------------------------------------
@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "bitlinear":
        return state["layer"](state["x"])
    if kind == "hgrn":
        op = chunk_hgrn if state["log_gate"] else fused_recurrent_hgrn
        return op(state["x"], state["g"], initial_state=state["h0"], output_final_state=True)
    if kind == "decode":
        dec = state["decoder"]
        token = dec.step()
        return {"token": token, "logits": dec.last_logits, "states": [s for (s,) in dec.cache.states]}
    lm = state["lm"]
    if kind == "generate":
        if state["sample"]:
            return lm.generate(state["ids"], max_new_tokens=state["new"], do_sample=True, top_p=0.4, temperature=0.6,
                               generator=state["generator"])
        return lm.generate(state["ids"], max_new_tokens=state["new"])
    if kind == "step":
        out = lm(input_ids=state["ids"], past_key_values=state["past"], use_cache=True)
    else:
        out = lm(input_ids=state["ids"], attention_mask=state.get("mask"), use_cache=True, last_token_only=state["last_only"])
    return {"logits": out.logits, "states": [s for (s,) in out.past_key_values]}


# -- what a pass cannot do without -----------------------------------------------------------------------------------
def _pass_work(case, rows, head_rows):
    """Bytes and operations of one forward over `rows` token rows with logits for `head_rows` of them: packed weights,
    norm weights, embedding rows, recurrent states (read and written) and logits; activations can stay on the chip."""
    hidden, inner, blocks = MODELS[case["model"]]
    e = BYTES[case["dtype"]]
    per_block = 4 * hidden * hidden + 3 * hidden * inner
    head = hidden * VOCAB
    norms = blocks * (7 * hidden + inner) + 2 * hidden
    data = (blocks * per_block + head) // 4 + norms * e + rows * (8 + hidden * e) + 8 * blocks * case["batch"] * hidden + head_rows * VOCAB * e
    return data, 2 * rows * blocks * per_block + 2 * head_rows * head


def work(case):
    kind, e = case["kind"], BYTES[case["dtype"]]
    if kind == "bitlinear":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": m * k * e + k * n // 4 + 4 * k + m * n * e, "flops": 2 * m * k * n}
    if kind == "hgrn":
        n = case["batch"] * case["time"] * case["width"]
        states = case["batch"] * case["width"] * (4 * case["initial"] + (4 if case["log_gate"] else e))
        return {"bytes": n * (2 * e + (4 if case["log_gate"] else e)) + states, "flops": 2 * n}
    batch = case["batch"]
    if kind in ("decode", "step"):
        data, ops = _pass_work(case, batch, batch)
    elif kind == "prompt":
        rows = batch * case["time"]
        data, ops = _pass_work(case, rows, batch if case["last_only"] else rows)
    else:       # the weights do not fit on the chip, so every new token reads them again
        data, ops = _pass_work(case, batch * case["time"], batch)
        step_data, step_ops = _pass_work(case, batch, batch)
        data, ops = data + (case["new"] - 1) * step_data, ops + (case["new"] - 1) * step_ops
    return {"bytes": data, "flops": ops}


def tolerance(case):
    """Half-precision activations: 1e-2 (2e-3 for the recurrence in fp16).  Single precision: the contraction is over
    integer codes, where an activation at a rounding tie may take either code (1e-4); the recurrence is plain fp32
    arithmetic (1e-5).  A token may differ where two logits are tied."""
    kind, dtype = case["kind"], case["dtype"]
    if kind == "hgrn":
        return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[dtype]}
    if kind == "bitlinear":
        return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-4}[dtype]}
    return {"rel": 1e-2, "differ": 0.01}
