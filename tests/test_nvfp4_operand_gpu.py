"""Both orientations of an NVFP4 operand from one call, byte for byte against the kernels that make one orientation at a time."""
import pytest
import torch

from llm_mojo_b200.ops import _lib, lowp

pytestmark = pytest.mark.gpu


def part(op, addr, n):
    at = addr - op.buf.data_ptr()
    return op.buf[at:at + n]


def same(got, want):
    return torch.equal(got.view(torch.uint8), want.view(torch.uint8))


# one 16 x 16 block; a whole tile; ragged tiles in both directions; partial scale atoms; several tiles
@pytest.mark.parametrize("rows,cols", [(16, 16), (128, 128), (144, 80), (272, 208), (48, 1600), (512, 400)])
@pytest.mark.parametrize("mode", ["nearest", "stochastic", "transform", "both", "block16"])
@pytest.mark.parametrize("special", ["normal", "zeros", "nan", "inf"])
def test_operand_bytes(rows, cols, mode, special):
    if special != "normal" and (rows, cols) not in ((144, 80), (128, 128)):
        pytest.skip("special values at two sizes")
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows + cols)).mul(3).bfloat16()
    x[rows // 2, cols // 3] = {"normal": 40.0, "zeros": 0.0, "nan": float("nan"), "inf": float("inf")}[special]
    if special == "zeros":
        x[: rows // 2] = 0
    x = x.cuda()
    sr, rht, b16 = mode in ("stochastic", "both"), mode in ("transform", "both"), mode == "block16"
    other = torch.full((1,), 0.75, device="cuda")
    op = lowp.Fp4Operand(x, True, True, block16=b16, rht=rht, sr=sr, seed=7, streams=(18, 19), step=5, other0=other.data_ptr(),
                         other1=other.data_ptr(), factor1=1.0 / 16)
    br = 16 if b16 else 1
    for axis in (1, 0):
        deq, ts, q, sc = lowp.nvfp4_fake_quant(x, axis=axis, block_rows=br, rht=rht and axis == 0, sr=sr, seed=7,
                                               stream_id=18 if axis else 19, step=5, want_packed=True)
        aq, asf, ats, aal = (op.q0, op.sf0, op.ts0, op.alpha0) if axis else (op.q1, op.sf1, op.ts1, op.alpha1)
        assert same(part(op, ats, 4), ts), "tensor scale"
        assert same(part(op, aal, 4), ts * other * (1.0 if axis else 1.0 / 16)), "product factor"
        assert same(part(op, asf, sc.numel()), sc), f"block scales, axis {axis}"
        assert same(part(op, aq, q.numel()), q), f"values, axis {axis}"
        single = lowp.Fp4Operand(x, axis == 1, axis == 0, block16=b16, rht=rht, sr=sr, seed=7, streams=(18, 19), step=5)
        assert same(part(single, single.q0 if axis else single.q1, q.numel()), q) and \
            same(part(single, single.sf0 if axis else single.sf1, sc.numel()), sc), f"one orientation, axis {axis}"
    assert _lib.read_status() == 0


def test_layouts_outside_the_tiles_take_the_general_path():
    x = torch.zeros(64, 64, dtype=torch.bfloat16, device="cuda")
    assert lowp._fp4_tiled(x, x[16:])
    assert not lowp._fp4_tiled(x.float())
    assert not lowp._fp4_tiled(x[:, :32])                  # row pitch beyond the row
    assert not lowp._fp4_tiled(x.t()[:, :32])
    assert not lowp._fp4_tiled(x[:24])                     # rows not in whole blocks
    assert not lowp._fp4_tiled(x.view(-1)[1:1 + 48 * 64].view(48, 64))   # alignment
