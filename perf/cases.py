"""The work whose speed counts: what users of this framework have it do, through its public entry points.

Three kinds of pass, each as the programs of this repository make it:

* ``train``     one optimizer step as ``Trainer.train_step`` and ``bench.py`` take it: the token batches come from pinned host
                memory, ``accum`` micro-steps of forward + backward, global gradient norm, clip factor, AdamW, read of the loss;
* ``eval``      one batch of ``Trainer.validate`` / ``infer_gpt2.run_eval``: forward with targets, read of the loss;
* ``generate``  one token of ``infer_gpt2.run_infer``: the whole forward pass at batch 1, the softmax of one row, its copy to the
                host (the next token is drawn there, so the program cannot go on without it).

Models are the descriptors of ``config.py`` whose head size is 64 (the GPT-2 ladder d6 ... d48 and the GPT-3 channel ladder up to
c1024); sequences are 16 tokens up to the model's maximum, batches 1 to 64; precisions are those of ``--precision``.
Weights are the model's random initialisation, tokens follow Zipf's law over the vocabulary as text does.  A delayed-scaling fp8
model is in mid-training: its amax histories are full.
"""
import math

import numpy as np
import torch

from llm_mojo_b200 import ops
from llm_mojo_b200.config import PARAM_NAMES, Precision, parse_model_descriptor
from llm_mojo_b200.models import GPT2
from llm_mojo_b200.ops.lowp import AMAX_HISTORY

LR, WEIGHT_DECAY, BETA1, BETA2, EPS, CLIP = 6e-4, 0.1, 0.9, 0.95, 1e-8, 1.0


def _case(name, kind, model, precision, B, T, accum=1, recompute=False, head_chunks=1):
    return {"name": name, "kind": kind, "model": model, "precision": precision, "B": B, "T": T, "accum": accum,
            "recompute": recompute, "head_chunks": head_chunks}


def listed():
    return [
        # sampling from a prompt that fits the smallest window run_infer uses: 64 positions
        _case("generate_d12_64", "generate", "d12", "bf16", 1, 64),
        # sampling late in a long text with a larger model; run_infer rounds the window up to a multiple of 8
        _case("generate_d24_776", "generate", "d24", "bf16", 1, 776),
        # validation and multiple-choice evaluation at infer_gpt2's default batch
        _case("eval_d12_16x1024", "eval", "d12", "bf16", 16, 1024),
        # a small experiment or a test: launches and host work show
        _case("train_d6_2x128", "train", "d6", "bf16", 2, 128),
        # the command line's default batch (-b 4 -t 1024), accumulated over two micro-steps
        _case("train_d12_4x1024_accum2", "train", "d12", "bf16", 4, 1024, accum=2),
        # sizes that no tile divides: an odd batch of an odd length
        _case("train_d12_7x777", "train", "d12", "bf16", 7, 777),
        # the headline configuration's micro-batch
        _case("train_d12_64x1024", "train", "d12", "bf16", 64, 1024),
        # long context of the GPT-3 ladder with the two options that save memory: recomputed GELU, LM head in vocabulary tiles
        _case("train_c1024_6x2048_recompute", "train", "gpt3:c1024", "bf16", 6, 2048, recompute=True, head_chunks=4),
        # fp32 storage: the TF32 tensor path
        _case("train_d12_4x512_tf32", "train", "d12", "tf32", 4, 512),
        # FP8, per-tensor delayed scaling, and FP8 with per-128 block scales on the d36 configuration
        _case("train_d36_8x1024_fp8", "train", "d36", "fp8", 8, 1024),
        _case("train_d36_4x1024_fp8b", "train", "d36", "fp8b", 4, 1024),
        # NVFP4 on the d48 configuration
        _case("train_d48_4x1024_fp4", "train", "d48", "fp4", 4, 1024),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["train", "train", "train", "eval", "generate"])
        model = rng.choice(["d6", "d12", "d12", "d24", "d36", "d48", "gpt3:c384", "gpt3:c768", "gpt3:c1024"])
        precision = rng.choice(["bf16", "bf16", "bf16", "fp8", "fp8b", "fp4", "tf32"]) if kind == "train" else "bf16"
        max_t = parse_model_descriptor(model).max_seq_len
        B = 1 if kind == "generate" else _log_int(rng, 1, 64)
        if precision in ("fp8", "fp8b", "fp4"):          # low-precision training runs at whole 128-row tiles
            T = 128 * rng.randint(1, max_t // 128)
        elif kind == "generate":                         # run_infer's windows are multiples of 8, at least 64
            T = 8 * _log_int(rng, 8, max_t // 8)
        else:
            T = _log_int(rng, 16, max_t)
        case = _case("", kind, model, precision, B, T, accum=rng.choice([1, 1, 1, 2, 3]) if kind == "train" else 1,
                     recompute=kind == "train" and rng.random() < 0.2, head_chunks=rng.choice([1, 1, 1, 4]) if kind == "train" else 1)
        del case["name"]
        if work(case)["flops"] <= most and _state_bytes(case) <= 45e9 and not (precision == "tf32" and B * T > 8192):
            return case


def _state_bytes(case):
    """Device memory of the parameters, optimizer state and activations of one case, roughly."""
    cfg = parse_model_descriptor(case["model"])
    rows, e = case["B"] * case["T"], 4 if case["precision"] == "tf32" else 2
    per_row = cfg.num_layer * cfg.channels * (16 * e + (9 if case["precision"].startswith("f") else 0)) + cfg.padded_vocab_size * e
    return cfg.num_parameters() * 18 + rows * per_row


def _weights(cfg, gen):
    """Flat fp32 parameters with the distributions of the random initialisation, drawn on the GPU."""
    flat = torch.zeros(cfg.num_parameters(), dtype=torch.float32, device="cuda")
    off = 0
    for name, n in zip(PARAM_NAMES, cfg.param_sizes()):
        part = flat[off:off + n]
        if name in ("ln1w", "ln2w", "lnfw"):
            part.fill_(1.0)
        elif name in ("wte", "wpe", "qkvw", "fcw"):
            part.normal_(0.0, 0.02, generator=gen)
        elif name in ("attprojw", "fcprojw"):
            part.normal_(0.0, 0.02 / math.sqrt(2.0 * cfg.num_layer), generator=gen)
        off += n
    flat[cfg.vocab_size * cfg.channels:cfg.padded_vocab_size * cfg.channels] = 0.0      # rows of the padded vocabulary
    return flat


def _tokens(cfg, n, rng):
    """``n`` token ids with Zipf frequencies over a shuffled vocabulary, in pinned host memory."""
    cdf = np.cumsum(1.0 / np.arange(1, cfg.vocab_size + 1))
    ranks = np.searchsorted(cdf, rng.random(n) * cdf[-1]).clip(max=cfg.vocab_size - 1)
    return torch.from_numpy(rng.permutation(cfg.vocab_size)[ranks].astype(np.int32)).pin_memory()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(1000 + seed)
    rng = np.random.default_rng(1000 + seed)
    cfg = parse_model_descriptor(case["model"])
    B, T, accum = case["B"], case["T"], case["accum"]
    model = GPT2(cfg, case["precision"], "cuda", recompute=case["recompute"], params_flat=_weights(cfg, gen),
                 lm_head_chunks=case["head_chunks"])
    batches = []
    for _ in range(accum):
        toks = _tokens(cfg, B * T + 1, rng)
        batches.append((toks[:-1].view(B, T).contiguous().pin_memory(), toks[1:].view(B, T).contiguous().pin_memory()))
    model.allocate_activations(B, T)
    pr = Precision(case["precision"])
    if pr.name == "fp8" and not pr.fp8_block_scales:
        for i in range(-(-AMAX_HISTORY // accum)):
            for micro, (x, y) in enumerate(batches):
                model.forward(x, y, accum, B=B, T=T)
                model.backward(accum, micro)
        model.read_loss()
    return {"kind": case["kind"], "model": model, "batches": batches, "B": B, "T": T, "accum": accum, "step": 0}


def run(state):
    m, B, T = state["model"], state["B"], state["T"]
    if state["kind"] == "generate":
        m.forward(state["batches"][0][0], None, B=B, T=T)
        row = m.acts["logits"][0, T - 1:T]
        probs = ops.softmax_rows(row.reshape(1, -1), m.config.vocab_size, 1.0)[0].float().cpu()
        return {"logits": m.acts["logits"], "probs": probs}
    if state["kind"] == "eval":
        x, y = state["batches"][0]
        m.forward(x, y, 1, B=B, T=T)
        return {"loss": m.read_loss(), "losses": m.acts["losses"]}
    for micro, (x, y) in enumerate(state["batches"]):
        m.forward(x, y, state["accum"], B=B, T=T)
        m.backward(state["accum"], micro)
    norm = m.calculate_grad_norm()
    scale = m.clip_scale_from_norm(norm, CLIP)
    state["step"] += 1
    m.update(state["step"], LR, WEIGHT_DECAY, 1.0, BETA1, BETA2, EPS, dev_scale=scale)
    out = {"loss": m.read_loss(), "norm": norm, "params": m.params}
    if m.master is not None:
        out["master"] = m.master
    return out


def work(case):
    cfg = parse_model_descriptor(case["model"])
    B, T, accum = case["B"], case["T"], case["accum"]
    L, C, Vp, P = cfg.num_layer, cfg.channels, cfg.padded_vocab_size, cfg.num_parameters()
    rows, e = B * T, 4 if case["precision"] == "tf32" else 2
    forward = rows * (2 * (12 * L * C * C + Vp * C) + 2 * L * T * C)      # linear layers and LM head; causal attention
    if case["kind"] == "generate":
        return {"flops": forward, "bytes": P * e + rows * (4 + Vp * e) + 4 * cfg.vocab_size}
    if case["kind"] == "eval":
        return {"flops": forward, "bytes": P * e + rows * 12}
    # parameters, gradients written, and the optimizer's read and write of its moments and of the fp32 weights
    state = P * (4 + 16) + P * (8 if e == 4 else 8 + 2 * e)
    return {"flops": 3 * forward * accum, "bytes": state + accum * rows * 8}


def tolerance(case):
    # Measured against a second implementation at the same precision (library GEMMs and attention, and the single-CTA GEMM with the
    # two-kernel attention backward), two passes: logits 1.4e-2, losses 2.7e-3; weights after two updates 3e-3 to 6e-3 in bf16 and
    # TF32, up to 1.5e-2 in fp8 and NVFP4 (largest element 0.13), gradient norm 1.3e-2.
    if case["kind"] == "eval":
        return {"rel": 0.01, "max": 0.4}
    return {"rel": 0.03, "max": 0.5}
