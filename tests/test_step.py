"""The ctypes mirror of the native step's argument block has the layout of the C struct."""
import ctypes

import pytest

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
