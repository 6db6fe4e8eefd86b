"""One forward / backward micro-step of GPT-2 through the native launch sequence (``csrc/gpt2_step.cu``).

``forward`` and ``backward`` issue exactly the ops that ``models/gpt2.py`` would issue one by one, over the same buffers and
scratch; ``usable`` says whether a model's state is what the native sequence is written for.  Pointers are read from the
tensors on every call."""
from __future__ import annotations

import ctypes
import functools
import os

import torch

from . import colsum_usable, lowp, scratch, _count, _dw_splits, _splits_for
from ._lib import check, dtype_code, lib, status_word, stream
from ..config import PARAM_NAMES
from .. import ops

ACTS = ("encoded", "ln1", "ln1_mean", "ln1_rstd", "qkv", "atty", "lse", "residual2", "ln2", "ln2_mean", "ln2_rstd", "fch", "fch_gelu",
        "residual3", "lnf", "lnf_mean", "lnf_rstd", "losses", "dres", "dl_btc", "dl_bt4c")          # then: logits or a vocabulary tile, ce_stats
F32_ACTS = frozenset(n for n in ACTS if n.endswith(("_mean", "_rstd"))) | {"lse", "losses"}
P, I, LL = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong


class Gpt2Step(ctypes.Structure):
    _fields_ = [("p", P * len(PARAM_NAMES)), ("g", P * len(PARAM_NAMES)), ("a", P * (len(ACTS) + 2)), ("tokens", P), ("targets", P),
                ("loss_acc", P), ("status", P), ("s_encoder", P), ("s_ln", P), ("s_dbias", P), ("s_stats", P), ("s_dq", P),
                ("s_encoder_bytes", LL), ("s_ln_bytes", LL), ("s_dbias_bytes", LL), ("dloss", ctypes.c_float),
                ("B", I), ("T", I), ("L", I), ("C", I), ("NH", I), ("V", I), ("Vp", I), ("recompute", I), ("tile_width", I), ("fc_colsum", I),
                ("splits_qkv", I), ("splits_att", I), ("splits_fc", I), ("splits_proj", I), ("splits_head", I), ("splits_head_last", I),
                ("vocab_bits", I), ("launches", I), ("dtype", I), ("lowp", I), ("fp4_first", I), ("fp4_end", I), ("fp4_rht", I), ("fp4_sr", I),
                ("lp_splits_qkv", I), ("lp_splits_att", I), ("lp_splits_fc", I), ("lp_splits_proj", I), ("seed", ctypes.c_ulonglong),
                ("micro", LL), ("s_lowp", P), ("kept", P), ("first", I), ("T_max", I)]


PLAIN, FP8B, FP4 = 0, 2, 3      # what the linear sites run in (LP_* of the C side)


def _mode(m):
    """PLAIN (bf16, or TF32 products on fp32 storage), FP8B, FP4, or None where the op-by-op path is taken."""
    pr, cfg, rows = m.precision, m.config, m.B * m.T
    if pr.name == "fp8":           # per-tensor scaling keeps its amax books in Python
        ok = (pr.fp8_block_scales and len(pr.fp8_sites) == 4 and m.dtype == torch.bfloat16 and lowp.FP8B_DUAL and lowp.fp8_block_native()
              and lowp.fp8_block_usable(rows, cfg.channels, cfg.channels))
        return FP8B if ok else None
    if pr.name == "fp4":
        return FP4 if m.dtype == torch.bfloat16 and lowp.nvfp4_native(cfg.channels, rows) else None
    return PLAIN if m.dtype == torch.bfloat16 or ops._tc_kind(m.loss_acc) is not None else None


def usable(m) -> bool:
    """The sequence covers one GPU with the default kernels and 64-wide heads: bf16, TF32, block-scaled FP8, NVFP4; ZeRO engines,
    per-tensor FP8, library comparators and the bias-gradient switches take the op-by-op path."""
    cfg, env = m.config, os.environ
    return (m.device.type == "cuda" and m.zero is None and ops.GEMM_IMPL == "tcgen05" and ops.ATTN_IMPL == "tcgen05"
            and ops.ATTN_BWD == "fused" and cfg.channels == 64 * cfg.num_heads
            and env.get("LLMM_FUSED_LN_DBIAS", "0") == "0" and env.get("LLMM_FUSED_QKV_DBIAS", "1") != "0" and _mode(m) is not None)


@functools.lru_cache(maxsize=64)
def _act_specs(L, C, NH, B, T, Vp, recompute, tile_width, dtype):
    """(name, type, bytes) of the buffers in ``ACTS`` and of the logits or the vocabulary tile, as the sequence indexes them."""
    rows = B * T
    once = {"encoded", "lnf", "lnf_mean", "lnf_rstd", "losses", "dres", "dl_btc", "dl_bt4c"} | ({"fch_gelu"} if recompute else set())
    width = {"qkv": 3 * C, "fch": 4 * C, "fch_gelu": 4 * C, "dl_bt4c": 4 * C, "lse": NH, "losses": 1}
    specs = [(n, torch.float32 if n in F32_ACTS else dtype, (1 if n in once else L) * rows * (1 if n.endswith(("_mean", "_rstd")) else width.get(n, C)))
             for n in ACTS]
    specs += [("logits_tile", dtype, rows * tile_width), ("ce_stats", torch.float32, 4 * rows)] if tile_width else [("logits", dtype, rows * Vp)]
    return tuple((n, t, e * t.itemsize) for n, t, e in specs)


@functools.lru_cache(maxsize=64)
def _param_specs(sizes, dtype):
    return tuple((n, dtype, e * dtype.itemsize) for n, e in zip(PARAM_NAMES, sizes))


def _addresses(tensors, specs):
    """Addresses of the named tensors, or None if one of them is not what the kernels take: they see no strides, read 16 bytes at a time
    and find a layer by its place (a model whose options were changed after its buffers were allocated keeps to the op-by-op path)."""
    out = []
    for name, dtype, nbytes in specs:
        t = tensors[name]
        at = t.data_ptr()
        if t.dtype is not dtype or t.nbytes != nbytes or at & 15 or not (t.is_cuda and t.is_contiguous()):
            return None
        out.append(at)
    return out


def _fill(m, tiled: bool, targets: bool):
    cfg, a = m.config, m.acts
    s = Gpt2Step()
    params = _addresses(m.p, _param_specs(tuple(m.param_sizes), m.dtype))
    acts = _addresses(a, _act_specs(cfg.num_layer, cfg.channels, cfg.num_heads, m.B, m.T, cfg.padded_vocab_size, m.recompute,
                                    m.tile_width if tiled else 0, m.dtype))
    if params is None or acts is None:
        return None
    s.p[:], s.a[:len(acts)] = params, acts
    if tiled:
        s.tile_width = m.tile_width
    s.tokens, s.targets = m.inputs_dev.data_ptr(), m.targets_dev.data_ptr() if targets else None
    s.loss_acc, s.status, s.dloss = m.loss_acc.data_ptr(), status_word(m.device).data_ptr(), m._dloss
    s.B, s.T, s.L, s.C, s.NH, s.V, s.Vp = m.B, m.T, cfg.num_layer, cfg.channels, cfg.num_heads, cfg.vocab_size, cfg.padded_vocab_size
    s.recompute, s.dtype = int(m.recompute), dtype_code(a["encoded"])
    s.lowp = _mode(m)
    if s.lowp:
        pr, L = m.precision, lib()
        s.fp4_first, s.fp4_end, s.fp4_rht, s.fp4_sr = pr.fp4_first, cfg.num_layer - pr.fp4_last_offset, int(pr.fp4_rht), int(pr.fp4_sr)
        s.seed, s.micro = m.rng_seed, m.micro_steps_done
        work = torch.empty(L.llmb_gpt2_lowp_scratch_bytes(ctypes.byref(s)), dtype=torch.uint8, device=m.device)
        s.s_lowp = work.data_ptr()
        s.work = work                                    # (a Python attribute: lives as long as the argument block)
    return s


def forward(m, targets: bool) -> bool:
    """Issues the forward pass; False (nothing issued) if a buffer is not a plain contiguous tensor."""
    s = _fill(m, targets and m.lm_head_chunks > 1, targets)
    if s is None:
        return False
    if s.lowp == FP8B and targets:                       # a backward pass may follow
        m.step_kept = torch.empty(lib().llmb_gpt2_lowp_kept_bytes(ctypes.byref(s)), dtype=torch.uint8, device=m.device)
        s.kept, m.step_kept_stream = m.step_kept.data_ptr(), stream()
    rc = lib().llmb_gpt2_forward(ctypes.byref(s), stream())
    _count(s.launches)
    check(rc, "gpt2_forward")
    return True


def backward(m, first: bool) -> bool:
    """As ``forward``.  ``first``: whatever the gradients hold is discarded."""
    cfg, a, dev = m.config, m.acts, m.device
    tiled = m.lm_head_chunks > 1
    s = _fill(m, tiled, True)
    if s is None:
        return False
    grads = _addresses(m.g, _param_specs(tuple(m.param_sizes), torch.float32))
    if grads is None:
        return False
    s.g[:] = grads
    s.first, s.T_max = int(first), m.config.max_seq_len
    B, T, C, NH, Vp = m.B, m.T, cfg.channels, cfg.num_heads, cfg.padded_vocab_size
    rows, L = B * T, lib()
    s.fc_colsum = int(colsum_usable(a["dl_bt4c"].view(rows, 4 * C), a["fch"][0].view(rows, 4 * C)))
    s.splits_qkv, s.splits_att = _dw_splits(3 * C, C, rows), _dw_splits(C, C, rows)
    s.splits_fc, s.splits_proj = _dw_splits(4 * C, C, rows), _dw_splits(C, 4 * C, rows)
    if tiled:
        s.splits_head, s.splits_head_last = (_dw_splits(w, C, rows) for w in (m.tile_width, Vp - (Vp - 1) // m.tile_width * m.tile_width))
    else:
        s.splits_head = s.splits_head_last = _dw_splits(Vp, C, rows)
    if s.lowp:
        if m.step_kept is not None and m.step_kept.numel() == L.llmb_gpt2_lowp_kept_bytes(ctypes.byref(s)):
            s.kept = m.step_kept.data_ptr()              # of this micro-step's forward pass
            if m.step_kept_stream != stream():           # it is let go below, while this stream may still have to read it
                m.step_kept.record_stream(torch.cuda.current_stream())
        lp = lambda n, k: _splits_for(n, k, rows, bk=128 if s.lowp == FP8B else 256)
        s.lp_splits_qkv, s.lp_splits_att, s.lp_splits_fc, s.lp_splits_proj = lp(3 * C, C), lp(C, C), lp(4 * C, C), lp(C, 4 * C)
    s.vocab_bits = max(1, (Vp - 1).bit_length())
    enc = scratch("encoder_bwd", L.llmb_encoder_bwd_scratch_bytes(rows, C), dev)
    ln = scratch("layernorm_bwd", L.llmb_layernorm_bwd_scratch_bytes(rows, C), dev)
    db = scratch("dbias", L.llmb_dbias_scratch_bytes(rows, 4 * C), dev)
    if m.dtype == torch.bfloat16:
        st = scratch("attn_bwd_stats", L.llmb_attention_bwd_fused_stats_floats(B, T, NH) * 4, dev)
        s.s_dq = scratch("attn_bwd_dq_acc", L.llmb_attention_bwd_fused_acc_floats(B, T, NH) * 4, dev, zero=True).data_ptr()
    else:
        st = scratch("attn_f32_dots", B * NH * T * 4, dev)
    s.s_encoder, s.s_ln, s.s_dbias, s.s_stats = (t.data_ptr() for t in (enc, ln, db, st))
    s.s_encoder_bytes, s.s_ln_bytes, s.s_dbias_bytes = enc.numel(), ln.numel(), db.numel()
    rc = L.llmb_gpt2_backward(ctypes.byref(s), stream())
    m.step_kept = None
    _count(s.launches)
    check(rc, "gpt2_backward")
    return True
