"""The ctypes mirror of the native step's argument block has the layout of the C struct."""
import ctypes

import pytest

from llm_mojo_b200.ops import _lib, step


@pytest.mark.skipif(not _lib.available(), reason="kernel library not built")
def test_step_struct_layout():
    assert ctypes.sizeof(step.Gpt2Step) == _lib.lib().llmb_gpt2_step_bytes()
