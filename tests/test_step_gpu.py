"""The native launch sequence of a bf16 micro-step against the op-by-op sequence of the model: same kernels, same buffers."""
import pytest
import torch

from llm_mojo_b200 import ops
from llm_mojo_b200.config import GPT2Config
from llm_mojo_b200.models import GPT2
from llm_mojo_b200.ops import _lib, step

pytestmark = pytest.mark.gpu


def run(native, monkeypatch, cfg, B, T, accum, recompute, chunks, targets=True):
    g = torch.Generator().manual_seed(3)
    m = GPT2(cfg, "bf16", "cuda", recompute=recompute, lm_head_chunks=chunks)
    used = []
    if native:
        monkeypatch.setattr(step, "usable", lambda mm, f=step.usable: used.append(f(mm)) or used[-1])
    else:
        monkeypatch.setattr(step, "usable", lambda mm: False)
    n0 = ops.LAUNCHES
    for micro in range(accum):
        toks = torch.randint(0, cfg.vocab_size, (B * T + 1,), generator=g, dtype=torch.int32)
        m.forward(toks[:-1].view(B, T), toks[1:].view(B, T) if targets else None, accum)
        if targets:
            m.backward(accum, micro)
    launches = ops.LAUNCHES - n0
    monkeypatch.undo()
    assert all(used) and (used or not native)
    out = {"grads": m.grads.clone(), "loss": torch.tensor(m.read_loss()), "lnf": m.acts["lnf"].clone()}
    if targets:
        out["losses"] = m.acts["losses"].clone()
    if not targets or chunks == 1:
        out["logits"] = m.acts["logits"].clone()
    assert _lib.read_status() == 0
    return out, launches


# sequence lengths around the 128-row tiles and the smallest; vocabulary tiles of equal and unequal width; one and several layers
@pytest.mark.parametrize("L,NH,B,T,accum,recompute,chunks", [
    (1, 1, 1, 16, 1, False, 1), (2, 3, 2, 127, 2, False, 1), (3, 2, 1, 129, 1, True, 1), (2, 2, 3, 200, 2, True, 3), (2, 4, 2, 256, 1, False, 4)])
def test_native_step_matches_op_by_op(L, NH, B, T, accum, recompute, chunks, monkeypatch):
    cfg = GPT2Config(max_seq_len=256, vocab_size=1000, num_layer=L, num_heads=NH, channels=64 * NH, padded_vocab_size=1024)
    want, n_want = run(False, monkeypatch, cfg, B, T, accum, recompute, chunks)
    got, n_got = run(True, monkeypatch, cfg, B, T, accum, recompute, chunks)
    assert n_got == n_want
    for k in want:
        if k == "grads":      # fp32 atomics add in another order from run to run, which bf16 gradients of earlier layers carry on
            assert (got[k] - want[k]).norm() <= 2.0 ** -8 * want[k].norm(), k
            assert ((got[k] == 0) == (want[k] == 0)).float().mean() > 0.999, k
        else:
            assert torch.equal(got[k], want[k]), k


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
