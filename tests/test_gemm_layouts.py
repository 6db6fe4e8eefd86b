"""Layouts that the GEMM entry points refuse on the host, before anything is launched."""
import pytest
import torch

from llm_mojo_b200.ops import EPI_ACC_F32, EPI_BIAS, EPI_BIAS_GELU, EPI_BIAS_RESID, EPI_DGELU, EPI_NONE, EPI_STORE_F32, _lib

pytestmark = pytest.mark.skipif(not _lib.available(), reason="kernel library not built")
M, N, K = 512, 264, 256
AT = 1 << 40                                             # made-up addresses: every call below ends on the host
BAD_ARG, NO_ENCODER = 2, 999


def call(which, epi, *, M=M, ldd=N, ldaux=N, aux=AT, bias=AT):
    L = _lib.lib()
    if which in ("nvfp4", "mxfp8"):
        fmts = (0, 0) if which == "mxfp8" else ()
        return getattr(L, f"llmb_gemm_{which}")(AT, AT, AT, AT, AT, bias, aux, None, M, N, K, *fmts, ldd, ldaux, epi, 1, AT, None)
    kind = {"bf16": 0, "tf32": 1, "fp8": 2}[which]
    return L.llmb_gemm(AT, AT, AT, bias, aux, None, M, N, K, K, K, ldd, ldaux, 0, 0, kind, 0, 0, epi, 1, AT, None)


ANY = ("bf16", "fp8", "nvfp4", "mxfp8", "tf32")
BF16 = ANY[:4]
REFUSED = [(w, e, dict(ldd=N + d)) for w in ANY for e in (EPI_ACC_F32, EPI_STORE_F32) for d in (1, 2, 3)]
REFUSED += [(w, e, dict(ldd=N + d)) for w in ANY for e in (EPI_NONE, EPI_BIAS, EPI_DGELU) for d in (1, 2, 6)]
REFUSED += [(w, e, dict(aux=None)) for w in ANY for e in (EPI_BIAS_GELU, EPI_DGELU, EPI_BIAS_RESID)]
REFUSED += [(w, e, dict(ldaux=N + 2)) for w in ANY for e in (EPI_BIAS_GELU, EPI_DGELU, EPI_BIAS_RESID)]
REFUSED += [(w, EPI_DGELU, dict(aux=AT + 4)) for w in ANY] + [("tf32", EPI_DGELU, dict(aux=AT + 8))]
REFUSED += [(w, e, dict(ldd=N + 4, bias=AT + 2)) for w in BF16 for e in (EPI_BIAS, EPI_BIAS_GELU, EPI_BIAS_RESID)]


@pytest.mark.parametrize("which,epi,layout", REFUSED)
def test_layouts_that_the_register_epilogue_would_access_misaligned_are_refused(which, epi, layout):
    """Without a tensor map the results leave by 16-byte (fp32) and 8-byte (bf16) accesses from registers; a row pitch, auxiliary tensor or bias
    that does not allow these, or a missing auxiliary tensor, is an argument error and not an access."""
    assert call(which, epi, **layout) == BAD_ARG


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up: only where no tensor map can be encoded and nothing is launched")
@pytest.mark.parametrize("which,epi,layout", [(w, e, {}) for w in ANY for e in range(7)] + [(w, e, dict(ldd=N + 4)) for w in ANY for e in range(7)]
                         + [(w, EPI_DGELU, dict(aux=AT + 8, ldaux=N + 4)) for w in BF16] + [(w, EPI_BIAS, dict(bias=None, ldd=N + 4)) for w in ANY]
                         + [(w, e, dict(bias=AT + 2, aux=AT + 2, ldaux=1)) for w in ANY for e in (EPI_NONE, EPI_ACC_F32, EPI_STORE_F32)]
                         + [(w, e, dict(M=1, ldd=N + 1, ldaux=1)) for w in ANY for e in range(7)])
def test_layouts_that_either_epilogue_can_access_are_taken(which, epi, layout):
    """They get as far as the operands' tensor maps, which this machine cannot encode."""
    assert call(which, epi, **layout) == NO_ENCODER
