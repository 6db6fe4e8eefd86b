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


@pytest.fixture
def force_tile():
    yield lambda bn, cl: _lib.lib().llmb_gemm_force_tile(bn, cl)
    _lib.lib().llmb_gemm_force_tile(0, 1)


# 256: CTA-pair kernel; 64 / 128: one tile per CTA, with 1, 2 or 4 CTAs sharing the contraction
@pytest.mark.parametrize("bn,cl", [(256, 1), (128, 1), (128, 2), (64, 1), (64, 2), (64, 4)])
# one row, a partial band, a partial tile; column counts that end inside a slab / inside a pair of slabs; odd numbers of k-blocks
@pytest.mark.parametrize("M,N,K", [(1, 64, 320), (37, 200, 264), (300, 1608, 456), (129, 320, 1288)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemm_tile_configurations(bn, cl, M, N, K, dtype, force_tile):
    """Every epilogue and operand layout on every tile configuration, at sizes that leave partial tiles, slabs and k-blocks."""
    force_tile(bn, cl)
    x, w, b, r = rnd(M, K, dtype=dtype), rnd(N, K, dtype=dtype, scale=0.05, seed=1), rnd(N, dtype=dtype, seed=2), rnd(M, N, dtype=dtype, seed=3)
    X, W, Bi, Rs = (t.to(DEV) for t in (x, w, b, r))
    # operands: bf16 exact, fp32 rounded to tf32 (2^-11 each, K terms of size ~0.05); results rounded once to the storage type
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10
    tol = dict(atol=eps * 4, rtol=eps)
    y = x.float() @ w.float().t()
    out, pre = torch.full((M, N), 7.0, dtype=dtype, device=DEV), torch.full((M, N), 7.0, dtype=dtype, device=DEV)
    ops.matmul_fwd(out, X, W)
    assert_close(out, y, what="none", **tol)
    ops.matmul_fwd(out, X, W, Bi)
    assert_close(out, y + b.float(), what="bias", **tol)
    ops.matmul_fwd(out, X, W, Bi, residual=Rs)
    assert_close(out, y + b.float() + r.float(), what="residual", **tol)
    ops.matmul_fwd(out, X, W, Bi, pre_gelu=pre)
    assert_close(pre, y + b.float(), what="pre-GELU", **tol)
    assert_close(out, torch.nn.functional.gelu(pre.float(), approximate="tanh"), 2 * eps, eps, "GELU")
    # backward: dinp [M, K] contracted over N, dW [N, K] contracted over M (added to what is there), column sums of dinp
    d = rnd(M, N, dtype=dtype, seed=4)
    D = d.to(DEV)
    g = d.float() @ w.float()
    tol_b = dict(atol=eps * 8, rtol=eps)
    dinp = torch.empty(M, K, dtype=dtype, device=DEV)
    ops.matmul_bwd(dinp, None, None, D, X, W)
    assert_close(dinp, g, what="dinp", **tol_b)
    cs = torch.full((K,), 0.5, device=DEV)
    ops.matmul_bwd(dinp, None, None, D, X, W, gelu_pre=X, dinp_colsum=cs)
    xg = x.float().requires_grad_(True)
    torch.nn.functional.gelu(xg, approximate="tanh").backward(g)
    assert_close(dinp, xg.grad, eps * 16, 2 * eps, "dGELU")
    assert_close(cs, 0.5 + dinp.float().sum(0).cpu(), 1e-4 * math.sqrt(M), 1e-4, "column sums")
    dw = torch.full((N, K), 0.25, device=DEV)
    ops.matmul_bwd(None, dw, None, D, X, W)
    assert_close(dw, 0.25 + d.float().t() @ x.float(), (1e-4 if dtype == torch.bfloat16 else 4 * eps) * math.sqrt(M), 1e-4 if dtype == torch.bfloat16 else eps, "dW")
    f32 = torch.empty(M, K, device=DEV)
    ops.gemm(f32, D, W, b_mn=True, epi=ops.EPI_STORE_F32, kind=0 if dtype == torch.bfloat16 else 1)
    assert_close(f32, g, 1e-4 if dtype == torch.bfloat16 else eps * 8, 1e-4 if dtype == torch.bfloat16 else eps, "fp32 store")
    torch.cuda.synchronize()
    assert _lib.read_status() == 0


@pytest.mark.parametrize("bn,cl", [(256, 1), (128, 1), (128, 2)])
def test_gemm_fp8_tile_configurations(bn, cl, force_tile):
    force_tile(bn, cl)
    M, N, K = 200, 336, 272
    a = rnd(M, K, dtype=torch.float32).to(torch.float8_e4m3fn)
    w = rnd(N, K, dtype=torch.float32, seed=1).to(torch.float8_e4m3fn)
    d = rnd(M, N, dtype=torch.float32, seed=2).to(torch.float8_e5m2)
    A, W, D = (t.view(torch.uint8).to(DEV) for t in (a, w, d))
    alpha = torch.full((1,), 0.125, device=DEV)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.gemm(out, A, W, kind=2, alpha=alpha)
    assert_close(out, 0.125 * a.float() @ w.float().t(), 2.0 ** -7, 2.0 ** -8, "fp8 forward")
    dinp = torch.empty(M, K, dtype=torch.bfloat16, device=DEV)
    ops.gemm(dinp, D, W, b_mn=True, kind=2, a_fmt=1, alpha=alpha)
    assert_close(dinp, 0.125 * d.float() @ w.float(), 2.0 ** -7, 2.0 ** -8, "fp8 dinp")
    dw = torch.zeros(N, K, device=DEV)
    ops.gemm(dw, D, A, a_mn=True, b_mn=True, epi=ops.EPI_ACC_F32, splits=2, kind=2, a_fmt=1, alpha=alpha)
    assert_close(dw, 0.125 * d.float().t() @ a.float(), 2e-3, 1e-4, "fp8 dW")
    assert _lib.read_status() == 0


# columns in the last 256-wide tile: its first warps' halves hold 1, 2, 3 (and 4, then 1) boxes of 32 columns; 1 and 2 slabs of 64
@pytest.mark.parametrize("N", [288, 320, 352, 416])
@pytest.mark.parametrize("epi", ["residual", "dgelu"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])      # 8 warps with two boxes each / two buffers for four boxes
def test_gemm_residual_right_edge_many_tiles(dtype, epi, N, force_tile):
    """Several tiles per CTA pair, the right edge leaving part of a warp's boxes: a buffer is refilled with the next tile's auxiliary
    input, which must wait for the store that still reads it."""
    force_tile(256, 1)
    M, K = 256 * 74 * 3 + 40, 64
    x, w, r = rnd(M, K, dtype=dtype), rnd(N, K, dtype=dtype, scale=0.1, seed=1), rnd(M, N, dtype=dtype, seed=2)
    ref = x.float() @ w.float().t()
    if epi == "residual":
        ref += r.float()
    else:
        xg = r.float().requires_grad_(True)
        torch.nn.functional.gelu(xg, approximate="tanh").backward(ref)
        ref = xg.grad
    X, W, Rs = x.to(DEV), w.to(DEV), r.to(DEV)
    zero = torch.zeros(N, dtype=dtype, device=DEV)
    # bf16: one rounding of the result, GELU' by a tanh within 2^-11; fp32: operands rounded to tf32 (2^-11 each, 64 terms of size ~0.1)
    tol = (2.0 ** -6, 2.0 ** -7 if epi == "dgelu" else 2.0 ** -8) if dtype == torch.bfloat16 else (2.0 ** -8, 2.0 ** -9)
    for _ in range(3):
        out = torch.empty(M, N, dtype=dtype, device=DEV)
        if epi == "residual":
            ops.matmul_fwd(out, X, W, zero, residual=Rs)
        else:
            ops.gemm(out, X, W, epi=ops.EPI_DGELU, aux=Rs, kind=0 if dtype == torch.bfloat16 else 1)
        assert_close(out, ref, *tol, f"{epi} at the right edge")
    assert _lib.read_status() == 0


# a thread of the classifier holds 7 or 8 vectors of a row: widths around whole and partial last vectors, the switch and the largest
@pytest.mark.parametrize("V,Vp", [(3, 8), (7930, 7936), (7944, 7944), (50257, 50304), (55546, 55552), (55553, 55560), (57344, 57344)])
@pytest.mark.parametrize("rows", [1, 3, 400])
def test_fused_classifier_row_widths(V, Vp, rows):
    x = rnd(rows, Vp, scale=3.0)
    tgt = torch.randint(0, V, (rows,), generator=torch.Generator().manual_seed(rows), dtype=torch.int32)
    tgt[0], tgt[-1] = 0, V - 1
    got, losses = x.to(DEV), torch.empty(rows, device=DEV)
    ops.fused_classifier(got, losses, tgt.to(DEV), 0.5, V)
    p = torch.softmax(x[:, :V].float(), dim=1)
    at = (torch.arange(rows), tgt.long())
    # the target column is a difference: absolute error of the bf16 exponential (p <= 1) and of the result
    assert_close(got.cpu()[at], 0.5 * (p[at] - 1), 0.5 * 2.0 ** -8, 0.0, "dlogits of the targets")
    got = got.cpu()
    got[at], p[at] = 0, 0
    assert_close(got[:, :V], 0.5 * p, 1e-7, 2.0 ** -7, "dlogits")        # two bf16 roundings: of the exponential and of the result
    assert bool((got[:, V:] == 0).all())
    want = torch.nn.functional.cross_entropy(x[:, :V].float(), tgt.long(), reduction="none")
    assert_close(losses, want, 1e-4, 1e-4, "losses")
    assert _lib.read_status() == 0


# one CTA, clusters of 2, 4 and 8 with even and uneven slabs, the last row count of the single launch and the first of the pair
@pytest.mark.parametrize("rows", [1, 511, 513, 1025, 3001, 8192, 8193])
@pytest.mark.parametrize("OC", [8, 72, 776])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_dbias_edges(rows, OC, dtype):
    x = rnd(rows, OC, dtype=dtype)
    got = torch.full((OC,), 3.0, device=DEV)
    ops.dbias_reduce(got, x.to(DEV))
    want = 3.0 + x.double().sum(0)
    assert_close(got, want, 2.0 ** -24 * 4 * rows ** 0.5 * 16, 1e-5, "dbias")      # fp32 sums of unit normals in short chains
    again = torch.full((OC,), 3.0, device=DEV)
    ops.dbias_reduce(again, x.to(DEV))
    assert torch.equal(got, again)


# segments of 16 positions, 4 segments and 32 channel vectors per CTA; a token that fills several segments, every token once
@pytest.mark.parametrize("BT,C,V", [(1, 8, 8), (15, 256, 40), (65, 264, 40), (300, 768, 7), (513, 384, 5000), (64, 1600, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("off", [0, 1])
def test_encoder_bwd_edges(BT, C, V, dtype, off):
    tok = torch.randint(0, V, (1, BT), generator=torch.Generator().manual_seed(BT), dtype=torch.int32)
    d = rnd(1, BT, C, dtype=dtype)
    store = torch.full((V * C + 1,), 0.5, device=DEV)
    dwte, dwpe = store[off:off + V * C].view(V, C), torch.full((BT, C), 0.25, device=DEV)      # off = 1: not 16-byte aligned
    ops.encoder_bwd(dwte, dwpe, d.to(DEV), tok.to(DEV))
    want = torch.full((V, C), 0.5, dtype=torch.float64).index_add_(0, tok[0].long(), d[0].double())
    assert_close(dwte, want, 1e-5, 1e-5, "dwte")
    assert_close(dwpe, 0.25 + d[0].double(), 1e-6, 1e-6, "dwpe")


# the forward takes one query tile per CTA up to as many tiles as the chip has SMs and pairs beyond: both sides of the switch, one tile,
# even and odd tile counts, ragged ends
@pytest.mark.parametrize("B,T,NH", [(1, 64, 12), (1, 128, 1), (1, 776, 16), (1, 1024, 18), (1, 1100, 16), (2, 1024, 9), (1, 1024, 19), (3, 300, 49), (3, 300, 50)])
def test_attention_fwd_tiles_per_item(B, T, NH):
    qkv = rnd(B, T, 3 * 64 * NH)
    ref, lse_ref = torch.empty(B, T, 64 * NH), torch.empty(B, NH, T)
    ops.attention_fwd(ref, lse_ref, qkv.float(), NH)
    out, lse = torch.empty(B, T, 64 * NH, dtype=torch.bfloat16, device=DEV), torch.empty(B, NH, T, device=DEV)
    ops.attention_fwd(out, lse, qkv.to(DEV), NH)
    assert_close(out, ref, 2.0 ** -7, 2.0 ** -7, "out")          # bf16 probabilities and output, values of order one
    assert_close(lse, lse_ref, 1e-3, 1e-4, "lse")
    assert _lib.read_status() == 0


# NaN and -infinity where a whole vector, a thread's whole share, a scalar tail or a row holds nothing else; masks of -infinity
@pytest.mark.parametrize("rows", [3, 64])              # softmax: a cluster of CTAs per row / one CTA per row
@pytest.mark.parametrize("V", [9, 4099])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_nan_reaches_every_denominator(rows, V, dtype):
    ld = (V + 15) // 8 * 8
    for where in (slice(0, 8), slice(V - 1, V), slice(0, V), slice(V // 2, V // 2 + 1)):
        for around in (0.5, float("-inf")):
            x = rnd(rows, ld, dtype=dtype)
            x[1] = around
            x[1, where] = float("nan")
            got = ops.softmax_rows(x.to(DEV), V).cpu()
            assert bool(torch.isnan(got[1]).all()), (where, around)
            assert_close(got[[0, 2]], torch.softmax(x[[0, 2], :V].float(), dim=-1), 1e-7, 2e-5, "rows beside it")
            stats, losses = torch.empty(rows, 4, device=DEV), torch.empty(rows, device=DEV)
            tgt = torch.zeros(rows, dtype=torch.int32, device=DEV)
            for c0 in range(0, ld, 2048):                  # several tiles: the NaN has to last
                w = min(2048, ld - c0)
                ops.chunked_ce_pass1(stats, x.to(DEV)[:, c0:c0 + w], tgt, c0, w, V, c0 == 0)
            ops.chunked_ce_loss(losses, stats)
            assert bool(torch.isnan(losses[1])), (where, around)
            assert_close(losses[[0, 2]], torch.nn.functional.cross_entropy(x[[0, 2], :V].float(), torch.zeros(2, dtype=torch.long), reduction="none"),
                         1e-5, 1e-5, "losses beside it")


@pytest.mark.parametrize("mask", [float("-inf"), "lowest"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_masked_logits_count_as_nothing(mask, dtype):
    rows, V = 5, 3001
    x = rnd(rows, 3008, dtype=dtype, scale=3.0)
    x[:, 100:2900] = torch.finfo(dtype).min if mask == "lowest" else mask
    assert_close(ops.softmax_rows(x.to(DEV), V), torch.softmax(x[:, :V].double(), dim=-1), 1e-7, 2e-5, "softmax")
    stats, losses = torch.empty(rows, 4, device=DEV), torch.empty(rows, device=DEV)
    tgt = torch.tensor([0, 99, 2900, 3000, 5], dtype=torch.int32)
    for c0 in (0, 1000, 2000):                             # the middle tile is masked as a whole
        ops.chunked_ce_pass1(stats, x.to(DEV)[:, c0:c0 + 1008 if c0 == 2000 else c0 + 1000], tgt.to(DEV), c0, 1008 if c0 == 2000 else 1000, V, c0 == 0)
    ops.chunked_ce_loss(losses, stats)
    want = torch.nn.functional.cross_entropy(x[:, :V].double(), tgt.long(), reduction="none")
    assert_close(losses, want, 1e-5, 1e-5, "losses")


def test_chunked_ce_exponentials_do_not_depend_on_the_storage_type():
    """The same logits as a bf16 and as an fp32 tile: the fp32 dlogits, rounded, are the bf16 dlogits."""
    rows, V = 200, 4096
    x = rnd(rows, V, scale=6.0).to(DEV)
    tgt = torch.randint(0, V, (rows,), dtype=torch.int32, generator=torch.Generator().manual_seed(2)).to(DEV)
    both = [x.clone(), x.float()]
    stats = [torch.empty(rows, 4, device=DEV) for _ in both]
    for t, s in zip(both, stats):
        ops.chunked_ce_pass1(s, t, tgt, 0, V, V, True)
    # two orders of 4096 additions of terms up to 1, the longest chain 32 of them; each exponential within 2^-23
    assert_close(stats[0], stats[1].cpu(), 0.0, 2.0 ** -21, "statistics")
    for t in both:
        ops.chunked_ce_pass2(t, stats[1], tgt, 0, V, V, 0.125)
    assert torch.equal(both[0], both[1].bfloat16())


# sizes at which the rule takes one CTA per tile, two and four CTAs per tile, and CTA pairs
@pytest.mark.parametrize("M,N,K", [(776, 1024, 1024), (64, 768, 768), (64, 768, 3072), (4096, 2304, 768)])
def test_gemm_armed_for_the_pair_kernel(M, N, K, force_tile):
    """The armed call, and only that one, gives the bits of the CTA-pair kernel."""
    x, w, b, r = rnd(M, K).to(DEV), rnd(N, K, scale=0.05, seed=1).to(DEV), rnd(N, seed=2).to(DEV), rnd(M, N, seed=3).to(DEV)

    def product():
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        ops.matmul_fwd(out, x, w, b, residual=r)
        return out

    rule = product()
    force_tile(256, 1)
    pair = product()
    force_tile(0, 1)
    _lib.lib().llmb_gemm_set_pair()
    assert torch.equal(product(), pair)
    assert torch.equal(product(), rule)
    if (M, K) == (64, 3072):
        assert not torch.equal(rule, pair)           # four CTAs add their parts of K: another order


@pytest.mark.parametrize("M,N,K", [(384, 384, 777), (768, 768, 2048), (1536, 384, 1024)])      # the rule alone would cut K into 3, 4 and 4 parts
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_weight_gradient_in_one_part_repeats_itself(M, N, K, dtype):
    a, b = rnd(K, M, dtype=dtype).to(DEV), rnd(K, N, dtype=dtype, seed=1).to(DEV)
    start = rnd(M, N, dtype=torch.float32, seed=2).to(DEV)
    got = []
    for _ in range(4):
        d = start.clone()
        ops.gemm(d, a, b, a_mn=True, b_mn=True, epi=ops.EPI_ACC_F32, splits=1, kind=0 if dtype == torch.bfloat16 else 1)
        got.append(d)
    assert all(torch.equal(got[0], d) for d in got[1:])
    want = start.double() + a.double().t() @ b.double()
    assert_close(got[0], want, (1e-4 if dtype == torch.bfloat16 else 2.0 ** -8) * math.sqrt(K), 1e-4 if dtype == torch.bfloat16 else 2.0 ** -10, "dW")
