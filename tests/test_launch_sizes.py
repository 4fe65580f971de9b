"""How large the launches of a shape are, where the host decides it alone (no GPU)."""
import ctypes

import pytest

from synaptix_b200.csrc.build import load_library
from synaptix_b200.ops.moe import MODE_GATE_UP, MODE_PLAIN


def library(name):
    import shutil
    if shutil.which("nvcc") is None:
        pytest.skip("no compiler for the kernels")
    return load_library(name)


@pytest.mark.parametrize("rows,E,N", [(1, 1, 8), (4, 16, 96), (8, 128, 768), (16, 1024, 130), (128, 16, 2432)])
def test_streamed_experts(rows, E, N):
    """No more blocks than the chosen experts' tiles, as far as that is known: a pair has one expert, so there are at most
    min(E, rows) of them."""
    blocks = library("moe").sx_moe_stream_blocks
    blocks.restype = ctypes.c_longlong
    for mode, tile in ((MODE_GATE_UP, 8), (MODE_PLAIN, 16)):
        assert blocks(rows, E, N, mode) == min(E, rows) * ((N + tile - 1) // tile)
