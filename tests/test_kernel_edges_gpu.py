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


# whole vectors, a straddling last vector, a tile that ends beyond the vocabulary, a tile without any real column
@pytest.mark.parametrize("rows,width,col0", [(1, 1024, 0), (37, 1000, 128), (5, 517, 3), (64, 1024, 29990), (3, 256, 30016)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_chunked_ce_edges(rows, width, col0, dtype):
    V, ld = 30011, 1024
    x = rnd(rows, ld, dtype=dtype, scale=3.0)
    t = torch.randint(0, V, (rows,), dtype=torch.int32, generator=torch.Generator().manual_seed(1))
    t[0] = col0 if col0 < V else 0
    st0 = torch.tensor([2.0, 5.0, 0.5, 0.0]).repeat(rows, 1)
    for first in (True, False):
        ref, got = st0.clone(), st0.to(DEV)
        ops.chunked_ce_pass1(ref, x[:, :width].float(), t, col0, width, V, first)
        ops.chunked_ce_pass1(got, x.to(DEV)[:, :width], t.to(DEV), col0, width, V, first)
        if first and col0 >= V:
            assert bool((got[:, 1] == 0).all())
            continue
        assert_close(got[:, :3], ref[:, :3], 1e-6, 1e-5, f"statistics first={first}")
    tile = x.to(DEV)
    ops.chunked_ce_pass2(tile[:, :width], got, t.to(DEV), col0, width, V, 0.125)
    ref_tile = x.float()[:, :width].clone()
    ops.chunked_ce_pass2(ref_tile, ref, t, col0, width, V, 0.125)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    assert_close(tile[:, :width], ref_tile, 1e-7, eps, "dlogits")
    assert torch.equal(tile[:, width:].cpu(), x[:, width:]), "columns beyond the tile must stay"


@pytest.mark.parametrize("rows", [1, 63, 64])          # a cluster of CTAs per row / one CTA per row
@pytest.mark.parametrize("V", [1, 9, 4097, 50257])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_softmax_rows_edges(rows, V, dtype):
    x = rnd(rows, (V + 15) // 8 * 8, dtype=dtype, scale=4.0)
    got = ops.softmax_rows(x.to(DEV), V, 0.7)
    assert_close(got, ops.softmax_rows(x, V, 0.7), 1e-7, 2e-5, "softmax")
    assert _lib.read_status() == 0


def test_gemm_residual_right_edge_many_tiles():
    """Several tiles per CTA pair with a right edge that leaves one 64-column slab in a warp's half of the tile: the slab's buffer is
    refilled with the next tile's residual, which must wait for the store that still reads it."""
    M, N, K = 256 * 74 * 3 + 40, 320, 64
    x, w, r = rnd(M, K), rnd(N, K, scale=0.1, seed=1), rnd(M, N, seed=2)
    ref = x.float() @ w.float().t() + r.float()
    X, W, Rs = x.to(DEV), w.to(DEV), r.to(DEV)
    for _ in range(5):
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        ops.matmul_fwd(out, X, W, torch.zeros(N, dtype=torch.bfloat16, device=DEV), residual=Rs)
        assert_close(out, ref, 2.0 ** -6, 2.0 ** -8, "residual at the right edge")
