"""The native launch sequence of a micro-step (bf16, TF32, block-scaled FP8, NVFP4) against the op-by-op sequence of the model: same
kernels, same buffers."""
import pytest
import torch

from llm_mojo_b200 import ops
from llm_mojo_b200.config import GPT2Config
from llm_mojo_b200.models import GPT2
from llm_mojo_b200.models.gpt2 import LAYER_TENSORS
from llm_mojo_b200.ops import _lib, step

pytestmark = pytest.mark.gpu


def run(native, monkeypatch, cfg, B, T, accum, recompute, chunks, targets=True, precision="bf16"):
    g = torch.Generator().manual_seed(3)
    m = GPT2(cfg, precision, "cuda", recompute=recompute, lm_head_chunks=chunks)
    used = []
    if native:
        monkeypatch.setattr(step, "usable", lambda mm, f=step.usable: used.append(f(mm)) or used[-1])
    else:
        monkeypatch.setattr(step, "usable", lambda mm: False)
    n0 = ops.LAUNCHES
    m.grads.fill_(float("nan"))      # the first micro-step discards whatever is there
    for micro in range(accum):
        toks = torch.randint(0, cfg.vocab_size, (B * T + 1,), generator=g, dtype=torch.int32)
        m.forward(toks[:-1].view(B, T), toks[1:].view(B, T) if targets else None, accum)
        if targets:
            m.backward(accum, micro)
    launches = ops.LAUNCHES - n0
    monkeypatch.undo()
    assert all(used) and (used or not native)
    out = {"grads": pieces(m) if targets else {}, "loss": torch.tensor(m.read_loss()), "lnf": m.acts["lnf"].clone()}
    if targets:
        out["losses"] = m.acts["losses"].clone()
    if not targets or chunks == 1:
        out["logits"] = m.acts["logits"].clone()
    assert _lib.read_status() == 0
    return out, launches


def pieces(m):
    """Every gradient by name, those of stacked tensors layer by layer."""
    out = {}
    for name, t in m.g.items():
        for l in range(m.config.num_layer) if name in LAYER_TENSORS else [None]:
            out[name if l is None else f"{name}[{l}]"] = (t if l is None else t[l]).clone()
    return out


# Largest difference of a gradient relative to its own norm.  fp32 atomics add in another order from run to run: fp32 storage passes that
# on as it is, bf16 gradients of earlier layers as single roundings (2^-8 of a value, some of the values), and where they are quantised
# again on the way a last bit can move a value to its neighbour (fp8: 2^-3 to 2^-2 of it, NVFP4: 1/4 to 1/2, a few of the values).  What the
# comparison is for - a gradient left out, added twice or to another layer - differs by its whole norm.
GRAD_TOL = {"tf32": 2.0 ** -12, "bf16": 2.0 ** -7, "fp8b": 2.0 ** -5, "fp4": 2.0 ** -3}


def same_grads(got, want, precision):
    assert got.keys() == want.keys()
    for k, w in want.items():
        assert torch.isfinite(got[k]).all(), k
        assert (got[k] - w).norm() <= GRAD_TOL[precision] * w.norm(), (k, ((got[k] - w).norm() / w.norm()).item())
        # single values may reach zero on one side only
        assert ((got[k] == 0) != (w == 0)).sum() <= 1 + 1e-3 * w.numel(), k


# sequence lengths around the 128-row tiles and the smallest; vocabulary tiles of equal and unequal width; one and several layers
@pytest.mark.parametrize("L,NH,B,T,accum,recompute,chunks", [
    (1, 1, 1, 16, 1, False, 1), (2, 3, 2, 127, 2, False, 1), (3, 2, 1, 129, 1, True, 1), (2, 2, 3, 200, 2, True, 3), (2, 4, 2, 256, 1, False, 4),
    (1, 12, 16, 256, 2, False, 1)])      # the last: head stored, layer weights split
def test_native_step_matches_op_by_op(L, NH, B, T, accum, recompute, chunks, monkeypatch):
    cfg = GPT2Config(max_seq_len=256, vocab_size=1000, num_layer=L, num_heads=NH, channels=64 * NH, padded_vocab_size=1024)
    want, n_want = run(False, monkeypatch, cfg, B, T, accum, recompute, chunks)
    got, n_got = run(True, monkeypatch, cfg, B, T, accum, recompute, chunks)
    assert n_got == n_want
    same_grads(got.pop("grads"), want.pop("grads"), "bf16")
    for k in want:
        assert torch.equal(got[k], want[k]), k


# TF32 on fp32 storage at lengths no tile divides; FP8 with block scales at whole 128-row tiles; NVFP4 in the middle layers only
@pytest.mark.parametrize("precision,L,NH,B,T,accum,recompute,chunks", [
    ("tf32", 2, 2, 2, 77, 2, False, 1), ("tf32", 1, 3, 1, 128, 1, True, 3), ("fp8b", 2, 2, 2, 128, 2, False, 1), ("fp8b", 2, 4, 1, 256, 1, True, 4),
    ("fp4", 6, 2, 2, 48, 2, False, 1), ("fp4", 5, 4, 1, 224, 1, True, 3)])
def test_native_step_in_other_precisions(precision, L, NH, B, T, accum, recompute, chunks, monkeypatch):
    cfg = GPT2Config(max_seq_len=256, vocab_size=1000, num_layer=L, num_heads=NH, channels=64 * NH, padded_vocab_size=1024)
    want, n_want = run(False, monkeypatch, cfg, B, T, accum, recompute, chunks, precision=precision)
    got, n_got = run(True, monkeypatch, cfg, B, T, accum, recompute, chunks, precision=precision)
    assert n_got == n_want
    same_grads(got.pop("grads"), want.pop("grads"), precision)
    for k in want:
        assert torch.equal(got[k], want[k]), k


@pytest.mark.parametrize("precision,NH,T", [("fp8b", 2, 96), ("fp8b", 3, 128), ("fp8", 2, 128), ("fp4", 2, 40)])
def test_other_shapes_and_precisions_stay_op_by_op(precision, NH, T):
    m = GPT2(GPT2Config(max_seq_len=256, vocab_size=1000, num_layer=1, num_heads=NH, channels=64 * NH, padded_vocab_size=1024), precision, "cuda")
    m.allocate_activations(1, T)
    assert not step.usable(m)


def test_native_forward_without_targets(monkeypatch):
    cfg = GPT2Config(max_seq_len=128, vocab_size=1000, num_layer=2, num_heads=2, channels=128, padded_vocab_size=1024)
    for chunks in (1, 4):     # without targets the whole logits are written, whatever the tiling of the loss
        want, n_want = run(False, monkeypatch, cfg, 1, 72, 1, False, chunks, targets=False)
        got, n_got = run(True, monkeypatch, cfg, 1, 72, 1, False, chunks, targets=False)
        assert n_got == n_want and torch.equal(got["logits"], want["logits"])


@pytest.mark.parametrize("n", [1, 3, 1023, 4097, 65536])
def test_loss_accumulate(n):
    x = torch.rand(n + 1, generator=torch.Generator().manual_seed(1)).cuda() * 11
    for off in (0, 1):        # aligned and unaligned
        v = x[off:off + n]
        acc = torch.full((1,), 2.0, device="cuda")
        ops.loss_accumulate(acc, v, 0.25)
        want = 2.0 + 0.25 * v.double().sum().item()
        assert abs(acc.item() - want) <= 2e-6 * want, (n, off)      # at most 64 serial fp32 additions of positive terms, then a tree


@pytest.mark.parametrize("form", ["strided", "transposed", "double", "empty"])
def test_loss_accumulate_takes_what_a_sum_takes(form):
    x = torch.rand(64, 96, generator=torch.Generator().manual_seed(1)).cuda()
    x = {"strided": x[:, ::2], "transposed": x.t(), "double": x.double(), "empty": x[:0]}[form]
    acc = torch.full((1,), 2.0, dtype=x.dtype, device="cuda")
    ops.loss_accumulate(acc, x, 0.25)
    want = 2.0 + 0.25 * x.double().sum().item()
    assert abs(acc.item() - want) <= 2e-6 * want


def test_options_changed_after_the_buffers_take_the_op_by_op_path():
    """One GELU buffer, and a backward pass that would index one per layer."""
    m = GPT2(GPT2Config(max_seq_len=64, vocab_size=1000, num_layer=2, num_heads=1, channels=64, padded_vocab_size=1024), "bf16", "cuda", recompute=True)
    toks = torch.zeros(1, 32, dtype=torch.int32)
    m.forward(toks, toks)
    m.recompute = False
    with pytest.raises(IndexError):
        m.forward(toks, toks)
    m.recompute = True
    m.forward(toks, toks)
    m.backward()
    torch.cuda.synchronize()
    assert _lib.read_status() == 0


def test_operands_kept_for_a_backward_pass_on_another_stream():
    """The forward's stream may not have their memory back while the backward's stream still reads them."""
    cfg = GPT2Config(max_seq_len=128, vocab_size=1000, num_layer=2, num_heads=2, channels=128, padded_vocab_size=1024)
    toks = torch.randint(0, 1000, (2 * 128 + 1,), generator=torch.Generator().manual_seed(5), dtype=torch.int32).cuda()
    x, y = toks[:-1].view(2, 128), toks[1:].view(2, 128)
    grads = []
    for apart in (False, True):
        m = GPT2(cfg, "fp8b", "cuda")
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        first.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(first):
            m.forward(x, y)
        n = m.step_kept.numel()
        second.wait_stream(first)
        with torch.cuda.stream(second if apart else first):
            torch.cuda._sleep(100_000_000)
            m.backward()
        assert m.step_kept is None
        with torch.cuda.stream(first):            # what a program may do next on its own stream
            reused = torch.full((n,), 0x7f, dtype=torch.uint8, device="cuda") if apart else None
        torch.cuda.synchronize()
        grads.append(m.grads.clone())
        del reused
    assert torch.isfinite(grads[1]).all() and (grads[1] - grads[0]).norm() <= 2.0 ** -8 * grads[0].norm()
