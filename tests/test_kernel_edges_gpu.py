"""Edges of the kernels' tiles and dispatch rules on the GPU, against the fp32 PyTorch statement of the same op."""
import math

import pytest
import torch

from llm_mojo_b200 import ops
from llm_mojo_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, dtype=torch.bfloat16, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + 7 * sum(shape))
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


def assert_close(a, b, atol, rtol, what):
    a, b = a.float().cpu(), b.float().cpu()
    assert torch.isfinite(a).all(), f"{what}: non-finite output"
    worst = ((a - b).abs() - (atol + rtol * b.abs())).max().item()
    assert worst <= 0, f"{what}: out of tolerance by {worst:.3g}"


# one vector, part of a warp, several warps per row, the widest rows; one row, partial chunks, several chunks per group
@pytest.mark.parametrize("C", [8, 264, 384, 1600, 4096])
@pytest.mark.parametrize("rows", [1, 5, 446, 3001])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_layernorm_bwd_edges(rows, C, dtype):
    if dtype == torch.float32:
        C = min(C, 2048)
    x, d, r0 = rnd(rows, C, dtype=dtype), rnd(rows, C, dtype=dtype, seed=1), rnd(rows, C, dtype=dtype, seed=2)
    w = (1 + 0.1 * rnd(C, dtype=dtype, seed=3)).to(dtype)
    mean = x.float().mean(1)
    rstd = torch.rsqrt(x.float().var(1, unbiased=False) + 1e-5)
    ref, rw, rb = r0.float().clone(), torch.full((C,), 0.25), torch.full((C,), -0.5)
    ops.layernorm_bwd(ref, rw, rb, d.float(), x.float(), w.float(), mean, rstd)
    got = []
    for _ in range(2):
        dres, dw, db = r0.to(DEV).clone(), torch.full((C,), 0.25, device=DEV), torch.full((C,), -0.5, device=DEV)
        ops.layernorm_bwd(dres, dw, db, d.to(DEV), x.to(DEV), w.to(DEV), mean.to(DEV), rstd.to(DEV))
        got.append((dres, dw, db))
    # one rounding to the storage type (2^-9 / fp32 sums of C terms); column sums of `rows` fp32 terms of size ~1
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-5
    assert_close(got[0][0], ref, eps * 4, eps, "dres")
    assert_close(got[0][1], rw, 1e-5 * math.sqrt(rows) + 1e-4, 1e-4, "dgamma")
    assert_close(got[0][2], rb, 1e-5 * math.sqrt(rows) + 1e-4, 1e-4, "dbeta")
    assert all(torch.equal(a, b) for a, b in zip(*got)), "LayerNorm backward must be bitwise repeatable"
