"""Single-token steps of a dense decoder: all its layers as one kernel (``ops.decode_layers``).

What the kernel computes is what ``PreNormBlock`` of RMS norms, plain grouped-query attention and SwiGLU launches as five kernels
a layer, for one or two rows in bfloat16.  A step is handed to it only if every layer is exactly that: the parts' classes, numbers and
tensors are looked at (``repeat.form_of``) in every step that is not replayed, so that a layer that was put in or a ``forward`` that
was wrapped is walked.
"""
from __future__ import annotations

import torch

from .. import ops
from ..parts.attention import Attention
from ..parts.block import PreNormBlock
from ..parts.linear import Linear
from ..parts.mlp import SwiGLU
from ..parts.norm import RMSNorm
from ..parts.rope import RotaryHalf
from .repeat import form_of


def _is_plain_dense(layer) -> bool:
    """A layer the kernel computes, going by its first example (the others are compared with its form)."""
    if type(layer) is not PreNormBlock or type(layer.mixer) is not Attention or type(layer.ffn) is not SwiGLU:
        return False
    a, f = layer.mixer, layer.ffn
    if not all(type(n) is RMSNorm for n in (layer.norm1, layer.norm2)) or layer.norm1.eps != layer.norm2.eps:
        return False
    if not all(type(p) is Linear and p.bias is None and p.weight is not None for p in (a.qkv, a.o, f.gate_up, f.down)):
        return False
    if not a.is_plain or not a.own_kv or a.shared or a.window is not None or a.sinks is not None or a._order is not None:
        return False
    if type(a.position) is not RotaryHalf or a.position.scaling is not None or a.position.rotary_dim != a.hd:
        return False
    W, ff = a.width, f.intermediate
    shapes = ((a.qkv, (a.nh + 2 * a.nkv) * a.hd, W), (a.o, W, a.nh * a.hd), (f.gate_up, 2 * ff, W), (f.down, W, ff))
    return (all(tuple(p.weight.shape) == (n, k) and p.weight.dtype == torch.bfloat16 for p, n, k in shapes)
            and f.width == W == layer.norm1.width == layer.norm2.width and (a.wq is None) == (a.wk is None))


def _records(model, cache, h: torch.Tensor):
    """``(records, the cache's keys and values as rows, cache group)``, or ``None`` if some layer is not like the first."""
    runs = model.steps
    first = model.layers[runs[0].layer]
    if not _is_plain_dense(first) or first.mixer.width != h.shape[1]:
        return None
    form = form_of(first)
    if form is None:
        return None
    views = [cache.view(r.cache_entry) for r in runs]
    k0, v0 = views[0].k, views[0].v
    stores = (k0.untyped_storage().data_ptr(), v0.untyped_storage().data_ptr())
    hd = first.mixer.hd
    lowest = min(views, key=lambda v: v.k.data_ptr())
    base = lowest.k.data_ptr(), lowest.v.data_ptr()
    records = []
    for run, view in zip(runs, views):
        layer = model.layers[run.layer]
        if layer is not first and form[0].tensors(layer) is None:
            return None
        if (view.group != views[0].group or view.window is not None or view.k.shape != k0.shape or view.v.shape != k0.shape
                or view.k.dtype != torch.bfloat16 or not view.k.is_contiguous() or not view.v.is_contiguous()
                or (view.k.untyped_storage().data_ptr(), view.v.untyped_storage().data_ptr()) != stores):
            return None
        at = view.k.data_ptr() - base[0]
        if view.v.data_ptr() - base[1] != at:
            return None
        a, f = layer.mixer, layer.ffn
        records.append([a.qkv.weight.data_ptr(), a.o.weight.data_ptr(), f.gate_up.weight.data_ptr(), f.down.weight.data_ptr(),
                        layer.norm1.weight.data_ptr(), layer.norm2.weight.data_ptr(), 0 if a.wq is None else a.wq.data_ptr(),
                        0 if a.wk is None else a.wk.data_ptr(), at // (2 * hd)])
    if any(p % 16 for r in records for p in r[:4]) or any(p % 8 for r in records for p in r[6:8]):
        return None
    rows = max(r[-1] for r in records) + k0.numel() // hd
    return records, lowest.k.as_strided((rows, hd), (hd, 1)), lowest.v.as_strided((rows, hd), (hd, 1)), views[0].group


def run_layers(model, h: torch.Tensor, ctx, cache) -> bool:
    """Run all layers on ``h`` (in place) if one kernel computes them; ``False`` (nothing launched) otherwise."""
    T = h.shape[0]
    o = ops.OPTIONS
    if not (o.decode_layers and o.attn_prep and o.attn_tma and o.gemm_ws and o.fused_residual):      # (those ask for other kernels)
        return False
    if (not ctx.all_single or T > ops.DECODE_LAYERS_MAX_ROWS or ctx.n_seqs != T or ctx.runtime.dtype != torch.bfloat16
            or h.dtype != torch.float32 or not h.is_contiguous() or not model.runs_each_layer_once or ops.current_gate() != (0.0, 0.0, 0)):
        return False
    first = model.layers[model.steps[0].layer]
    if type(first) is not PreNormBlock or type(first.mixer) is not Attention or type(first.ffn) is not SwiGLU:
        return False
    a, ff = first.mixer, first.ffn.intermediate
    need = ops.decode_layers_words(T, h.shape[1], a.nh, a.nkv, a.hd, ff, len(model.steps))
    found = _records(model, cache, h) if need > 0 else None
    if found is None:
        return False
    records, k_rows, v_rows, group = found
    # The records and the workspace belong to the step's arrays: a captured step keeps them for its replays, any other one
    # makes them anew.
    kept = ctx.scratch.get("decode_layers")
    if kept == "no room":
        return False
    if kept is None or kept[0] != records or kept[2].numel() < need:
        if torch.cuda.is_current_stream_capturing():
            return False
        kept = ctx.scratch["decode_layers"] = (records, torch.tensor(records, dtype=torch.int64).to(h.device, non_blocking=True),
                                               torch.zeros(need, dtype=torch.int64, device=h.device))
    inv_freq, _ = a._rotation()
    if ops.decode_layers(kept[1], kept[2], h, ctx.seq_lens, ctx.block_tables[group], k_rows, v_rows,
                         cache.view(model.steps[0].cache_entry).k.shape[0], inv_freq, a.nh, a.nkv, a.hd, ff, a.scale, first.norm1.eps,
                         a.qk_norm_eps if a.qk_norm_eps is not None else 0.0):
        return True
    ctx.scratch["decode_layers"] = "no room"       # (so that the step is walked when it is captured, too)
    return False
