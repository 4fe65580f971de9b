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


def plan(lib, name, *args):
    out = (ctypes.c_int * 2)()
    f = getattr(library(lib), name)
    f.restype = None
    f(*args, out)
    return tuple(out)


@pytest.mark.parametrize("sms", [74, 108, 148, 160, 296])
def test_float32_launches_follow_the_sms(sms):
    """Float32 products: 64-row tiles from two a SM on; else blocks that share a tile's K until there is about one a SM.  Float32
    attention: blocks that share a token's keys until there is one a SM."""
    for M, N, K in ((17, 1024, 4096), (263, 1024, 3072), (263, 4096, 1024), (1024, 6144, 1024), (600, 2048, 300), (9000, 2048, 64)):
        rows, cluster = plan("generic", "sx_gemm_f32_plan", M, N, K, sms)
        columns = -(-N // 128)
        assert rows == (64 if -(-M // 64) * columns >= 2 * sms else 32)
        tiles, few = -(-M // rows) * columns, sms - sms // 18
        assert cluster in (1, 2, 4, 8) and (cluster == 1 or (tiles * cluster // 2 < few and K >= 128 * cluster))
        assert cluster == 8 or tiles * cluster >= few or K < 256 * cluster
    for n, nh, nkv, pages in ((1, 16, 8, 40), (2, 16, 8, 3), (20, 16, 8, 64), (263, 16, 8, 5), (40, 4, 4, 9), (9, 32, 4, 64), (400, 8, 8, 8)):
        tokens, cluster = plan("generic", "sx_attn_f32_plan", n, nh, nkv, pages, sms)
        heads = nh // nkv
        rows = 2 if heads <= 2 else 4
        blocks = nkv * -(-heads // rows) * n
        assert cluster == 8 or blocks * cluster >= sms or pages < 2 * cluster
        assert cluster == 1 or (blocks * cluster // 2 < sms and tokens == 1)
        assert tokens == (rows // heads if cluster == 1 and heads < rows and blocks >= sms * (rows // heads) else 1)


@pytest.mark.parametrize("lens", [[40], [500, 1, 1, 5], [1, 500], [3, 64, 2, 20, 5, 6], [6, 6, 6, 6, 6, 6, 6], [30, 70, 5, 8, 6, 200], [1] * 40, [200, 5, 7, 7, 7]])
@pytest.mark.parametrize("past", [0, 300, 5000])
def test_float32_attention_of_long_and_short_portions(lens, past):
    """Sequences that bring less than the others' tiles are worth lie within the range that is handed on, and the rest has tiles."""
    f = library("generic").sx_attn_f32_mix
    f.restype = None
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    out = (ctypes.c_int * 4)()
    array = lambda x: (ctypes.c_int * len(x))(*x)  # noqa: E731
    f(array(cu), array([past if n < 40 else 0 for n in lens]), cu[-1], len(lens), 64, 8, 148, out)
    tiles, few, first, last = out

    def worth(rest):
        per = sum(rest) // len(rest) if rest else 0
        return per >= 16 and -(-sum(rest) // 32) * 64 * min(per, 32) >= 32 * 148 // 3
    assert bool(tiles) == any(worth([n for n in lens if n >= k]) for k in ((0,) if len(lens) == 1 else (6, 17, 33)))
    if tiles:
        small = [(a, b) for a, b in zip(cu, cu[1:]) if b - a < few]
        assert (first, last) == ((small[0][0], small[-1][1]) if small else (0, 0)) and worth([n for n in lens if n >= few])
        assert few in ((6, 17, 33) if small else (0,)) and (past < 5000 or few > 8 or not any(6 <= n <= 8 for n in lens))
    f(None, None, cu[-1], len(lens), 64, 8, 148, out)        # (where the lengths are not known, any may be short)
    assert list(out) == [int(worth(lens))] + ([6, 0, cu[-1]] if len(lens) > 1 else [0, 0, 0])
