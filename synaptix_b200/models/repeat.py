"""A prompt step's launches for layers of one form, made again with other pointers.

The layers of a decoder are mostly the same parts with other weights: what differs between two neighbouring layers' launches
are the pointers of their parameters, of their cache entries and of the branch that travels from one to the next.  A prompt
step of a few hundred tokens is bound by the host, which walks the parts and makes some twenty arguments for each of two
hundred launches (17 us a launch at 0.6B sizes, more than the kernels take); so the step walks the first two layers of a
stretch, records what the second one launched, and makes the same launches for the others with their pointers put in (5 us).
Nothing of a step outlasts it: the layers' forms are taken anew in every step (20 us a layer), so that a layer that was put in, a
number that was changed or a ``forward`` that was wrapped since the last one counts as it does where every layer is walked.

Only parts whose class says ``repeatable`` in its own body are asked (their ``forward`` launches kernels through ``ops.launch``
and does nothing else on the device, and depends on nothing but their sizes, the step and their inputs; strings other than the
tensors' names, ``name_attributes``, belong to the form), and only a recording that holds everything that was launched is used;
any other layer is simply walked.
"""
from __future__ import annotations

import bisect
import ctypes
import itertools
from typing import List, Optional, Tuple

import torch

from ..parts.base import Part, PendingLinear

MIN_LAYERS = 4                 # a stretch shorter than this is walked


class _Unlike(Exception):
    pass


_VALUES = frozenset((type(None), bool, int, float, torch.dtype, torch.device))


def _walk_part(part: Part, form: list, places: list) -> None:
    """Append what ``part`` is, its tensors' names aside, to ``form`` and the place of every tensor in it to ``places``."""
    cls = type(part)
    if not cls.__dict__.get("repeatable", False):
        raise _Unlike
    held = vars(part)
    form += (cls, tuple(held))
    for key in cls.shared_attributes:              # (what a step makes of such a tensor has a place of its own in the launches)
        t = held[key]
        form.append(None if t is None else t.data_ptr())
    _walk(held, held.items(), form, places, cls.name_attributes)


def _walk(where, items, form: list, places: list, names) -> None:
    """The values of ``where``.  ``names``: the keys whose strings are names of tensors (``True``: all)."""
    put = form.append
    for key, value in items:
        kind = type(value)
        put(kind)
        if kind in _VALUES:
            put(value)
        elif kind is str:
            if names is not True and key not in names:
                put(value)
        elif kind is torch.Tensor or kind is torch.nn.Parameter:
            put((value.shape, value.dtype, value.device, value.is_contiguous()))
            places.append((where, key))
        elif issubclass(kind, Part):
            _walk_part(value, form, places)
        elif kind is dict:
            named = names is True or key in names
            put(len(value) if named else tuple(value))
            _walk(value, value.items(), form, places, named or ())
        elif kind is list or issubclass(kind, tuple):
            put(len(value))
            _walk(value, enumerate(value), form, places, names is True or key in names or ())
        else:
            raise _Unlike


def form_of(layer: Part) -> Optional[Tuple[tuple, list]]:
    """``(form, places of its tensors)`` of a layer, or ``None`` if it holds anything that is not repeatable."""
    form, places = [], []
    try:
        _walk_part(layer, form, places)
    except _Unlike:
        return None
    return tuple(form), places


def _tensors(places: list) -> List[torch.Tensor]:
    return [where[key] for where, key in places]


def _at(tensors: List[torch.Tensor], t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else next((i for i, x in enumerate(tensors) if x is t), -1)


def repeat(recording, before, after, places: list, views: list):
    """Make the launches of ``recording`` again for the layers behind the recorded one.

    ``places[0]`` and ``places[1]`` are the tensors' places of the layer before the recorded one and of the recorded one,
    ``places[2:]`` those of the layers to come; ``views[1:]`` are the cache views of the recorded and the coming ones.
    ``before`` and ``after`` are the branches the recorded layer was handed and handed on (``PendingLinear``).  Returns the
    branch that the last layer hands on, or ``None`` if the recording cannot be used (nothing has been launched then)."""
    from ..ops._lib import check, use_gate
    if not recording.whole or type(before) is not PendingLinear or type(after) is not PendingLinear:
        return None
    if before.x.shape != after.x.shape or before.x.dtype != after.x.dtype or (before.bias is None) != (after.bias is None):
        return None
    first, second = _tensors(places[0]), _tensors(places[1])
    weight, bias = _at(second, after.weight), _at(second, after.bias)
    if weight == -1 or bias == -1 or first[weight] is not before.weight or (bias is not None and first[bias] is not before.bias):
        return None
    if any(v.group != views[1].group or v.window != views[1].window for v in views[2:]):
        return None
    # What a recorded pointer can be, as (row, column) of the table that a layer makes of its own: (the layer before, the branch
    # that comes in) and (the layer, its cache, the branch that goes out).
    def table(above, mine, view, x_in, x_out):
        k, v = (0 if t is None else t.data_ptr() for t in (view.k, view.v))
        return above + [x_in.data_ptr()], mine + [k, v, x_out.data_ptr()]
    x_in, x_out = before.x, after.x
    above, mine = [t.data_ptr() for t in first], [t.data_ptr() for t in second]
    source = {}
    for row, pointers in enumerate(table(above, mine, views[1], x_in, x_out)):
        for i, a in enumerate(pointers):
            source.setdefault(a, []).append((row, i))
    source.pop(0, None)
    tables = []
    for p, view in zip(places[2:], views[2:]):
        x_in, x_out = x_out, x_in                  # the branch a layer hands on is the next one's
        above, mine = mine, [where[key].data_ptr() for where, key in p]
        tables.append(table(above, mine, view, x_in, x_out))
    # one pointer for several things (tied weights): they have to be one in every layer
    for at in source.values():
        if len(at) > 1 and any(t[row][i] != t[at[0][0]][at[0][1]] for t in tables for row, i in at[1:]):
            return None
    # (a pointer into the middle of one of these has no place to come from in the next layer)
    spans = sorted((t.data_ptr(), t.data_ptr() + t.numel() * t.element_size())
                   for t in first + second + [before.x, after.x] + [t for t in (views[1].k, views[1].v) if t is not None])
    starts, ends = [a for a, _ in spans], list(itertools.accumulate((b for _, b in spans), max))

    def inside(a: int) -> bool:
        i = bisect.bisect_right(starts, a)
        return i > 0 and a < ends[i - 1]
    calls = []
    for f, args, what, launches, gated in recording.calls:
        if any(kind is ctypes.c_void_p and a and a not in source and inside(a) for a, kind in zip(args, f.argtypes)):
            return None
        put = [(j,) + source[a][0] for j, (a, kind) in enumerate(zip(args, f.argtypes))
               if kind is ctypes.c_void_p and a in source]
        calls.append((f, list(args), put, what, launches, gated))
    for t in tables:
        for f, args, put, what, launches, gated in calls:
            for j, row, i in put:
                args[j] = t[row][i]
            if gated is not None:                  # (a library's activation may be another thread's since)
                use_gate(gated)
            check(f(*args), what, launches)
    last = _tensors(places[-1])
    return PendingLinear(x_out, last[weight], None if bias is None else last[bias])
