"""fp32 attention on the GPU (forward, log-sum-exp, backward) against the same formulas in 64 bits."""
import math

import pytest
import torch

from llm_mojo_b200 import ops

pytestmark = pytest.mark.gpu


def reference(qkv, dout, NH):
    """out, lse (log2 domain) and dqkv in float64."""
    B, T, C3 = qkv.shape
    q, k, v = (t.view(B, T, NH, 64).transpose(1, 2) for t in qkv.double().split(C3 // 3, dim=2))
    do = dout.double().view(B, T, NH, 64).transpose(1, 2)
    s = (q @ k.transpose(-1, -2) / 8).masked_fill(~torch.ones(T, T, dtype=torch.bool, device=qkv.device).tril(), float("-inf"))
    lse = torch.logsumexp(s, dim=-1)
    p = torch.exp(s - lse.unsqueeze(-1))
    o = p @ v
    ds = p * (do @ v.transpose(-1, -2) - (do * o).sum(-1, keepdim=True)) / 8
    back = lambda t: t.transpose(1, 2).reshape(B, T, C3 // 3)
    return back(o), lse * math.log2(math.e), torch.cat([back(ds @ k), back(ds.transpose(-1, -2) @ q), back(p.transpose(-1, -2) @ do)], dim=2)


def rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-300)).item()


# one row, part of a tile, tiles of 64 rows exactly and one more, several tiles with a ragged last one; one and several heads
@pytest.mark.parametrize("B,T,NH", [(1, 1, 1), (2, 16, 3), (1, 63, 2), (1, 64, 1), (2, 65, 2), (1, 128, 5), (3, 200, 2), (1, 1000, 2)])
@pytest.mark.parametrize("scale", [1.0, 6.0])
def test_attention_f32(B, T, NH, scale):
    g = torch.Generator().manual_seed(T)
    C = 64 * NH
    qkv = (torch.randn(B, T, 3 * C, generator=g) * scale).cuda()
    dout = torch.randn(B, T, C, generator=g).cuda()
    out, lse = torch.empty(B, T, C, device="cuda"), torch.empty(B, NH, T, device="cuda")
    dqkv = torch.full((B, T, 3 * C), 7.0, device="cuda")
    dbias = torch.ones(3 * C, device="cuda")
    assert ops._attn_f32(NH, qkv, out, lse, dqkv, dout)
    ops.attention_fwd(out, lse, qkv, NH)
    ops.attention_bwd(dqkv, dout, qkv, out, lse, NH, dbias=dbias)
    o, l, d = reference(qkv, dout, NH)
    # a score is a sum of 64 products of size scale^2 (error of order 2^-24 * 8 * scale^2), which the exponential passes on; the sums that
    # follow add a few 2^-24 each
    tol = 2.0 ** -24 * (16 + 16 * scale * scale)
    assert rel(out, o) < tol and rel(dqkv, d) < 2 * tol if T > 1 else rel(out, o) < tol
    # largest single error of a score: 64 serial additions, each off by at most 2^-24 of a partial sum of the |q k| (mean below scale^2),
    # in the units of lse
    assert (lse.double() - l).abs().max() < 64 * 2.0 ** -24 * 64 * scale * scale * math.log2(math.e) / 8 + 2.0 ** -22
    if T == 1:
        # one key: dq and dk vanish and dv is dout times a probability of 1, recomputed as 2^(score - lse) from two roundings of the same
        # score, so off by up to 2^-23 of the score, which is of order 8 * scale^2
        assert rel(dqkv[..., 2 * C:], dout.double()) < tol and dqkv[..., :2 * C].abs().max() < 1e-4 * scale
    assert (dbias.double() - 1 - d.sum((0, 1))).abs().max() < 1e-3 * scale


def test_layouts_outside_the_kernel_keep_the_library_path():
    qkv = torch.randn(1, 32, 3 * 64, device="cuda")
    out, lse = torch.empty(1, 32, 64, device="cuda"), torch.empty(1, 1, 32, device="cuda")
    assert ops._attn_f32(1, qkv, out, lse)
    assert not ops._attn_f32(2, qkv, out, lse)                       # 32-wide heads
    assert not ops._attn_f32(1, qkv.double(), out, lse)
    assert not ops._attn_f32(1, torch.randn(1, 32, 6 * 64, device="cuda")[..., ::2], out, lse)
    wide = torch.empty(1, 32, 128, device="cuda")
    assert not ops._attn_f32(1, qkv, wide[..., :64], lse)
    ops.attention_fwd(wide[..., :64], lse, qkv, 1)
    ops.attention_fwd(out, lse, qkv, 1)
    assert (wide[..., :64] - out).abs().max() < 1e-4                 # fp32 rounding of either path


def _inputs(B=2, T=80, NH=2):
    g = torch.Generator().manual_seed(4)
    qkv, dout = torch.randn(B, T, 192 * NH, generator=g).cuda(), torch.randn(B, T, 64 * NH, generator=g).cuda()
    return qkv, dout, torch.empty(B, T, 64 * NH, device="cuda"), torch.full((B, NH, T), float("nan"), device="cuda")


TOL = 2.0 ** -24 * 64          # as in test_attention_f32 at scale 1, either path


# the forward and the backward choose their path by their own tensors: each form of the forward, followed by the backward kernel
@pytest.mark.parametrize("form", ["plain", "strided out", "strided qkv", "unaligned qkv", "strided lse", "unaligned lse", "bf16 out", "recorded"])
def test_backward_after_every_form_of_the_forward(form):
    qkv, dout, out, lse = _inputs()
    B, T, C = out.shape
    o, l, x = out, lse, qkv
    if form == "strided out":
        o = torch.empty(B, T, 2 * C, device="cuda")[..., :C]
    elif form == "bf16 out":
        o = torch.empty(B, T, C, device="cuda", dtype=torch.bfloat16)
    elif form == "strided qkv":
        x = torch.empty(B, T, 6 * C, device="cuda")[..., ::2].copy_(qkv)
    elif form == "unaligned qkv":
        x = torch.empty(qkv.numel() + 1, device="cuda")[1:].view(qkv.shape).copy_(qkv)
    elif form == "strided lse":
        l = torch.empty(*lse.shape, 2, device="cuda")[..., 0]
    elif form == "unaligned lse":
        l = torch.empty(lse.numel() + 1, device="cuda")[1:].view(lse.shape)
    elif form == "recorded":
        x = qkv.clone().requires_grad_(True)
    assert ops._attn_f32(2, x, o, l) == (form == "plain")
    ops.attention_fwd(o, l, x, 2)
    want_o, want_l, want_d = reference(qkv, dout, 2)
    assert rel(o.detach(), want_o) < (2.0 ** -8 if form == "bf16 out" else TOL)
    assert (l.double() - want_l).abs().max() < 1e-5
    if form == "recorded":        # autograd saw the forward
        o.backward(dout)
        assert rel(x.grad, want_d) < 2 * TOL
    saved, lse = o.detach().float().contiguous(), l.clone(memory_format=torch.contiguous_format)
    dqkv = torch.empty_like(qkv)
    assert ops._attn_f32(2, qkv, saved, lse, dqkv, dout)
    ops.attention_bwd(dqkv, dout, qkv, saved, lse, 2)
    # a rounded output enters through sum(dO * O) only
    assert rel(dqkv, want_d) < (2.0 ** -8 if form == "bf16 out" else 2 * TOL)


# what the library path took without looking at lse or out: no lse, one of another size, gradients over their inputs, nothing at all
@pytest.mark.parametrize("form", ["no lse", "short lse", "no out", "in place", "empty"])
def test_calls_that_need_no_saved_statistics(form):
    qkv, dout, out, lse = _inputs()
    want_o, _, want_d = reference(qkv, dout, 2)
    dqkv = torch.empty_like(qkv)
    if form == "no lse":
        lse = None
    elif form == "short lse":
        lse = torch.full((4,), 9.0, device="cuda")
    elif form == "in place":
        dqkv = qkv
    elif form == "empty":
        qkv, dout, out, lse, dqkv = qkv[:0], dout[:0], out[:0], lse[:0], dqkv[:0]
    ops.attention_fwd(out, lse, qkv, 2)
    saved = None if form == "no out" else out
    ops.attention_bwd(dqkv, dout, qkv, saved, lse, 2)
    if form == "empty":
        return
    assert rel(out, want_o) < TOL and rel(dqkv, want_d) < 2 * TOL
    if form == "short lse":
        assert bool((lse == 9.0).all())


@pytest.mark.parametrize("B,T,NH", [(1, 1, 1), (1, 64, 1), (2, 65, 2), (3, 200, 2), (1, 1000, 2), (4, 512, 12)])
def test_split_backward_repeats_itself(B, T, NH, monkeypatch):
    """LLMB_ATTN_BWD=split: the fp32 backward without additions in arrival order."""
    monkeypatch.setattr(ops, "ATTN_BWD", "split")
    qkv, dout, out, lse = _inputs(B, T, NH)
    ops.attention_fwd(out, lse, qkv, NH)
    got = []
    for _ in range(3):
        dqkv = torch.full_like(qkv, float("nan"))
        ops.attention_bwd(dqkv, dout, qkv, out, lse, NH)
        got.append(dqkv)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    want = reference(qkv, dout, NH)[2]
    if T == 1:                     # dq and dk vanish
        assert rel(got[0][..., 128 * NH:], dout.double()) < TOL and got[0][..., :128 * NH].abs().max() < 1e-4
    else:
        assert rel(got[0], want) < 2 * TOL
