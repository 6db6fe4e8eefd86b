"""One bf16 forward / backward micro-step of GPT-2 through the native launch sequence (``csrc/gpt2_step.cu``).

``forward`` and ``backward`` issue exactly the ops that ``models/gpt2.py`` would issue one by one, over the same buffers and
scratch; ``usable`` says whether a model's state is what the native sequence is written for.  Pointers are read from the
tensors on every call."""
from __future__ import annotations

import ctypes
import os

import torch

from . import _lib, colsum_usable, scratch, _count, _splits_for
from ._lib import check, lib, ptr, status_word, stream
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
                ("vocab_bits", I), ("launches", I)]


def _plain(tensors, dtype) -> bool:
    return all(t.dtype == dtype and t.is_cuda and t.is_contiguous() for t in tensors)


def usable(m) -> bool:
    """The sequence covers bf16 storage and products on one GPU with the default kernels (64-wide heads); ZeRO engines, low-precision
    sites, library comparators and the bias-gradient switches take the op-by-op path."""
    cfg, env = m.config, os.environ
    return (m.device.type == "cuda" and m.zero is None and m.precision.name == "bf16" and m.dtype == torch.bfloat16 and m.lowp is None
            and ops.GEMM_IMPL == "tcgen05" and ops.ATTN_IMPL == "tcgen05" and ops.ATTN_BWD == "fused" and cfg.channels == 64 * cfg.num_heads
            and env.get("LLMM_FUSED_LN_DBIAS", "0") == "0" and env.get("LLMM_FUSED_QKV_DBIAS", "1") != "0"
            and _plain((t for n, t in m.acts.items() if n in ACTS and n not in F32_ACTS), m.dtype)
            and _plain((m.acts[n] for n in F32_ACTS), torch.float32) and _plain(m.p.values(), m.dtype))


def _fill(m, tiled: bool, targets: bool) -> Gpt2Step:
    cfg, a = m.config, m.acts
    s = Gpt2Step()
    s.p[:] = [m.p[n].data_ptr() for n in PARAM_NAMES]
    s.a[:len(ACTS)] = [a[n].data_ptr() for n in ACTS]
    s.a[len(ACTS)] = a["logits_tile" if tiled else "logits"].data_ptr()
    if tiled:
        s.a[len(ACTS) + 1] = a["ce_stats"].data_ptr()
        s.tile_width = m.tile_width
    s.tokens, s.targets = m.inputs_dev.data_ptr(), m.targets_dev.data_ptr() if targets else None
    s.loss_acc, s.status, s.dloss = m.loss_acc.data_ptr(), status_word(m.device).data_ptr(), m._dloss
    s.B, s.T, s.L, s.C, s.NH, s.V, s.Vp = m.B, m.T, cfg.num_layer, cfg.channels, cfg.num_heads, cfg.vocab_size, cfg.padded_vocab_size
    s.recompute = int(m.recompute)
    return s


def forward(m, targets: bool) -> None:
    s = _fill(m, targets and m.lm_head_chunks > 1, targets)
    rc = lib().llmb_gpt2_forward(ctypes.byref(s), stream())
    _count(s.launches)
    check(rc, "gpt2_forward")


def backward(m) -> None:
    cfg, a, dev = m.config, m.acts, m.device
    tiled = m.lm_head_chunks > 1
    s = _fill(m, tiled, True)
    s.g[:] = [m.g[n].data_ptr() for n in PARAM_NAMES]
    B, T, C, NH, Vp = m.B, m.T, cfg.channels, cfg.num_heads, cfg.padded_vocab_size
    rows, L = B * T, lib()
    s.fc_colsum = int(colsum_usable(a["dl_bt4c"].view(rows, 4 * C), a["fch"][0].view(rows, 4 * C)))
    s.splits_qkv, s.splits_att = _splits_for(3 * C, C, rows), _splits_for(C, C, rows)
    s.splits_fc, s.splits_proj = _splits_for(4 * C, C, rows), _splits_for(C, 4 * C, rows)
    if tiled:
        s.splits_head, s.splits_head_last = (_splits_for(w, C, rows) for w in (m.tile_width, Vp - (Vp - 1) // m.tile_width * m.tile_width))
    else:
        s.splits_head = s.splits_head_last = _splits_for(Vp, C, rows)
    s.vocab_bits = max(1, (Vp - 1).bit_length())
    enc = scratch("encoder_bwd", L.llmb_encoder_bwd_scratch_bytes(rows, C), dev)
    ln = scratch("layernorm_bwd", L.llmb_layernorm_bwd_scratch_bytes(rows, C), dev)
    db = scratch("dbias", L.llmb_dbias_scratch_bytes(rows, C if s.fc_colsum else 4 * C), dev)
    st = scratch("attn_bwd_stats", L.llmb_attention_bwd_fused_stats_floats(B, T, NH) * 4, dev)
    dq = scratch("attn_bwd_dq_acc", L.llmb_attention_bwd_fused_acc_floats(B, T, NH) * 4, dev, zero=True)
    s.s_encoder, s.s_ln, s.s_dbias, s.s_stats, s.s_dq = (t.data_ptr() for t in (enc, ln, db, st, dq))
    s.s_encoder_bytes, s.s_ln_bytes, s.s_dbias_bytes = enc.numel(), ln.numel(), db.numel()
    rc = L.llmb_gpt2_backward(ctypes.byref(s), stream())
    _count(s.launches)
    check(rc, "gpt2_backward")
