"""Python face of ``csrc/layers.cu``: all layers of a dense decoder in one kernel, single-token steps (bfloat16, one or two rows)."""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from ._lib import KernelError, c_int, check, fn, launcher, raw_stream, require_cuda

# Rows a step: with more, every block's share of the activations (tagged words, twice their size) costs more than the kernel saves.
# Measured with forms for four and eight rows, ms a step at 4B sizes and 1,100 keys: 4 rows 2.02 to 2.07 against 2.07 with five kernels
# a layer, 8 rows 2.62 against 2.20 (0.6B: 0.72 to 0.80 against 0.76, 0.99 against 0.82).  One and two rows are shorter at every size
# measured: 0.6B, 1.7B, 4B, 8B and models of two layers, 30 to 7,000 keys (figures in the source).
MAX_ROWS = 2
NO_ROOM = 10006       # the library's code for a stream whose share of the SMs does not hold all blocks at once
RECORD = 9            # 8-byte numbers a layer: q/k/v, o, gate and up, down; gains of norm1, norm2, q and k heads; first cache row

_WORDS = {}


def decode_layers_words(T: int, W: int, nh: int, nkv: int, hd: int, ff: int, n_layers: int) -> int:
    """The workspace of a step of ``T`` rows in 8-byte words, or 0 where the kernel does not take these sizes."""
    key = (torch.cuda.current_device(), T, W, nh, nkv, hd, ff, n_layers)
    n = _WORDS.get(key)
    if n is None:
        f = fn("layers", "sx_decode_layers_plan")
        n = _WORDS[key] = int(f(*(c_int(v) for v in key[1:])))
    return n


def decode_layers(layers: torch.Tensor, words: torch.Tensor, h: torch.Tensor, seq_lens: torch.Tensor, block_table: torch.Tensor,
                  k_rows: torch.Tensor, v_rows: torch.Tensor, n_pages: int, inv_freq: Optional[torch.Tensor], nh: int, nkv: int, hd: int,
                  ff: int, scale: float, eps: float, qk_eps: float) -> bool:
    """``h [T, W]`` (float32, in place) through the layers of ``layers`` (int64 ``[n, RECORD]`` on the device).

    ``k_rows`` / ``v_rows [rows, hd]``: the cache of all layers as rows, a layer's from its record's last number on;
    ``words``: ``decode_layers_words`` zeros (int64) that no launch running at the same time uses.  ``False``: the blocks
    cannot run at once on the current stream (it has a part of the SMs only), and nothing was launched."""
    require_cuda(layers, words, h, seq_lens, block_table, k_rows, v_rows, inv_freq)
    T, W = h.shape
    if h.dtype != torch.float32 or layers.dtype != torch.int64 or layers.dim() != 2 or layers.shape[1] != RECORD:
        raise KernelError("decode_layers: float32 rows, int64 [n, 9] records")
    need = decode_layers_words(T, W, nh, nkv, hd, ff, layers.shape[0])
    if need <= 0 or words.numel() < need or words.dtype != torch.int64:
        raise KernelError("decode_layers: sizes the kernel does not take, or too small a workspace")
    if k_rows.dtype != torch.bfloat16 or v_rows.dtype != torch.bfloat16 or k_rows.shape != v_rows.shape or k_rows.shape[1] != hd:
        raise KernelError("decode_layers: the cache is bfloat16 [rows, head size]")
    if seq_lens.numel() < T or block_table.dim() != 2 or block_table.shape[0] < T or seq_lens.dtype != torch.int32 or block_table.dtype != torch.int32:
        raise KernelError("decode_layers: int32 lengths and block tables of every row")
    if inv_freq is not None and (inv_freq.dtype != torch.float32 or inv_freq.numel() != hd // 2):
        raise KernelError("decode_layers: float32 frequencies of the whole head")
    code = launcher("layers", "sx_decode_layers")(
        layers.data_ptr(), layers.shape[0], words.data_ptr(), h.data_ptr(), h.data_ptr(), seq_lens.data_ptr(), block_table.data_ptr(),
        block_table.shape[1], n_pages, k_rows.data_ptr(), v_rows.data_ptr(), k_rows.shape[0], None if inv_freq is None else inv_freq.data_ptr(),
        T, W, nh, nkv, hd, ff, scale, eps, qk_eps, raw_stream())
    if code == NO_ROOM:
        return False
    check(code, "decode_layers")
    return True


def decode_layers_status(reset: bool = False) -> int:
    """0, or which bounded wait of the kernel ran out (a value in host memory: no device call)."""
    out = (ctypes.c_int * 1)()
    check(fn("layers", "sx_decode_layers_status")(out, c_int(1 if reset else 0)), "decode_layers_status", launches=0)
    return int(out[0])
