"""The ctypes side of the kernel library: argument block, argument lists, refusal of a library built from other sources."""
import ctypes
import glob
import os
import re
import subprocess
import sys
import threading

import pytest
import torch

from llm_mojo_b200 import ops
from llm_mojo_b200.config import GPT2Config
from llm_mojo_b200.models import GPT2
from llm_mojo_b200.ops import _lib, step


@pytest.mark.skipif(not _lib.available(), reason="kernel library not built")
def test_step_struct_layout():
    assert ctypes.sizeof(step.Gpt2Step) == _lib.lib().llmb_gpt2_step_bytes()


@pytest.mark.skipif(not _lib.available(), reason="kernel library not built")
@pytest.mark.parametrize("kind", [0, 1])
def test_weight_gradients_are_cut_into_no_more_parts_than_asked_for(kind):
    """Parts of a contraction are added in the order in which they finish: one part is the caller's way to a repeatable sum."""
    L, seen = _lib.lib(), set()
    for M in (64, 384, 768, 3072):
        for N in (64, 768, 1600):
            for K in (64, 777, 2048, 4096):
                for splits in (1, 2, 3, 8):
                    got = L.llmb_gemm_dw_splits(kind, M, N, K, splits)
                    assert 1 <= got <= splits, (M, N, K, splits, got)
                    seen.add(got)
    assert len(seen) > 2
    # a negative number leaves the parts of other tiles than CTA pairs to the rule, and means the same on CTA pairs
    assert L.llmb_gemm_dw_splits(kind, 384, 384, 777, -1) > L.llmb_gemm_dw_splits(kind, 384, 384, 777, 1) == 1
    assert L.llmb_gemm_dw_splits(kind, 3072, 3072, 8192, -2) == L.llmb_gemm_dw_splits(kind, 3072, 3072, 8192, 2) == 2
    assert 1 <= L.llmb_gemm_dw_splits(kind, 384, 384, 64, -(1 << 31)) <= 2


@pytest.mark.parametrize("bwd,sign", [("fused", -1), ("split", 1)])
def test_the_repeatable_choice_holds_weight_gradients_to_their_parts(bwd, sign, monkeypatch):
    monkeypatch.setattr(ops, "ATTN_BWD", bwd)
    for size in ((384, 384, 777), (768, 768, 65536)):
        assert ops._dw_splits(*size) == sign * ops._splits_for(*size)


class _Fn:
    def __init__(self, value):
        self.value = value

    def __call__(self):
        return self.value


class _Library:
    """A stand-in for a loaded library: every entry point is there, ``without`` one of them, with the given answers."""

    def __init__(self, abi=_lib.ABI, step_bytes=ctypes.sizeof(step.Gpt2Step), without=None):
        for name in _lib._SIGS:
            if name != without:
                setattr(self, name, _Fn(0))
        self.llmb_abi, self.llmb_gpt2_step_bytes = _Fn(abi), _Fn(step_bytes)


def test_a_library_of_other_sources_is_refused_at_load():
    _lib._declare(_Library())
    for other in (_Library(abi=_lib.ABI - 1), _Library(step_bytes=ctypes.sizeof(step.Gpt2Step) - 8), _Library(without="llmb_gpt2_forward")):
        with pytest.raises(RuntimeError, match="build it again"):
            _lib._declare(other)


def test_argument_lists_match_the_sources():
    csrc = os.path.join(os.path.dirname(_lib.__file__), os.pardir, "csrc")
    text = "\n".join(open(f).read() for f in sorted(glob.glob(os.path.join(csrc, "*.cu"))))
    declared = {}
    for name, args in re.findall(r"LLMB_API\s+(?:int|long long|void)\s+(\w+)\(([^)]*)\)", text):
        declared.setdefault(name, set()).add(len(args.split(",")) if args.strip() else 0)
    for name, sig in _lib._SIGS.items():
        if name.startswith("llmb_bounds_report"):          # defined by a macro
            continue
        assert declared.get(name) == {len(sig)}, name


@pytest.mark.skipif(not _lib.available(), reason="kernel library not built")
def test_layernorm_backward_of_nothing_is_an_error():
    """In a process of its own: an integer division by zero would end it."""
    code = ("from llm_mojo_b200.ops import _lib\n"
            "for rows, C in ((0, 768), (4, 0), (-1, 768)):\n"
            "    for dtype in (0, 1):\n"
            "        assert _lib.lib().llmb_layernorm_bwd_colsum(*[None] * 5, 1 << 20, *[None] * 5, rows, C, 1, dtype, None) == 2   # BAD_ARG\n")
    root = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__))))
    assert subprocess.run([sys.executable, "-c", code], cwd=root).returncode == 0


@pytest.mark.skipif(not _lib.available(), reason="kernel library not built")
def test_forced_tiles_are_the_calling_threads_own():
    L = _lib.lib()
    parts = lambda: L.llmb_gemm_dw_splits(0, 768, 768, 2048, 15)
    rule, other = parts(), []
    try:
        L.llmb_gemm_force_tile(64, 1)
        assert parts() == 15 != rule                       # a forced tile takes the parts as given
        t = threading.Thread(target=lambda: other.append(parts()))
        t.start()
        t.join()
    finally:
        L.llmb_gemm_force_tile(0, 1)
    assert other == [rule] and parts() == rule


class _Tensor:
    def __init__(self, n, dtype=torch.bfloat16, at=1 << 20, cuda=True, contiguous=True):
        self.nbytes, self.dtype, self.at, self.is_cuda, self.contiguous = n * dtype.itemsize, dtype, at, cuda, contiguous

    data_ptr = lambda self: self.at
    is_contiguous = lambda self: self.contiguous


def test_addresses_of_plain_buffers_only():
    good = {"qkv": _Tensor(12), "lse": _Tensor(4, torch.float32, at=1 << 21)}
    specs = (("qkv", torch.bfloat16, 24), ("lse", torch.float32, 16))
    assert step._addresses(good, specs) == [1 << 20, 1 << 21]
    for bad in (_Tensor(11), _Tensor(6, torch.float32), _Tensor(12, torch.float16), _Tensor(12, at=(1 << 20) + 8), _Tensor(12, cuda=False),
                _Tensor(12, contiguous=False)):
        assert step._addresses({**good, "qkv": bad}, specs) is None


@pytest.mark.parametrize("recompute,chunks", [(False, 1), (True, 1), (False, 3)])
def test_buffer_sizes_are_those_that_the_model_allocates(recompute, chunks):
    cfg = GPT2Config(max_seq_len=16, vocab_size=300, num_layer=3, num_heads=2, channels=128, padded_vocab_size=384)
    m = GPT2(cfg, "fp32", "cpu", recompute=recompute, lm_head_chunks=chunks)
    m.allocate_activations(2, 5)
    specs = lambda r: step._act_specs(3, 128, 2, 2, 5, 384, r, m.tile_width if chunks > 1 else 0, torch.float32)
    sizes = {n: (t.dtype, t.nbytes) for n, t in m.acts.items()}
    assert {n: (t, b) for n, t, b in specs(recompute)} == sizes != {n: (t, b) for n, t, b in specs(not recompute)}
    assert [n for n, _, _ in specs(recompute)][:len(step.ACTS)] == list(step.ACTS)
    assert [(m.p[n].dtype, m.p[n].nbytes) for n, _, _ in step._param_specs(tuple(m.param_sizes), torch.float32)] == \
        [(t, b) for _, t, b in step._param_specs(tuple(m.param_sizes), torch.float32)]


def test_a_forward_pass_lets_go_of_what_the_one_before_left():
    m = GPT2(GPT2Config(max_seq_len=16, vocab_size=60, num_layer=1, num_heads=1, channels=64, padded_vocab_size=64), "fp32", "cpu")
    m.step_kept = torch.zeros(3)              # as a native forward would
    toks = torch.zeros(1, 4, dtype=torch.int32)
    m.forward(toks, toks)                     # op by op
    assert m.step_kept is None
