"""A prompt step's launches for layers of one form, made again with other pointers.

The layers of a decoder are mostly the same parts with other weights: what differs between two neighbouring layers' launches
are the pointers of their parameters, of their cache entries and of the branch that travels from one to the next.  A prompt
step of a few hundred tokens is bound by the host, which walks the parts and makes some twenty arguments for each of two
hundred launches (17 us a launch at 0.6B sizes, more than the kernels take); so the step walks the first two layers of a
stretch, records what the second one launched, and makes the same launches for the others with their pointers put in (5 us).
Nothing of a step outlasts it: the layers' forms are compared anew in every step (10 us a layer), so that a layer that was put in, a
number that was changed or a ``forward`` that was wrapped since the last one counts as it does where every layer is walked.

Only parts whose class says ``repeatable`` in its own body are asked (their ``forward`` launches kernels through ``ops.launch``
and does nothing else on the device, and depends on nothing but their sizes, the step and their inputs; strings other than the
tensors' names, ``name_attributes``, belong to the form), and only a recording that holds everything that was launched is used;
any other layer is simply walked.
"""
from __future__ import annotations

import bisect
import ctypes
import functools
import itertools
import operator
from typing import Iterable, List, Optional, Tuple

import torch

from ..parts.base import Part, PendingLinear

class _Unlike(Exception):
    pass


_VALUES = frozenset((type(None), bool, int, float, str, torch.dtype, torch.device))


def _plain(value) -> bool:
    """Whether ``value`` holds nothing but numbers, strings and the like."""
    kind = type(value)
    if kind in _VALUES:
        return True
    if kind is dict:
        return _plain(tuple(value)) and _plain(tuple(value.values()))
    return (kind is list or issubclass(kind, tuple)) and all(_plain(v) for v in value)


@functools.lru_cache(maxsize=256)
def _getter(names: tuple):
    """The attributes ``names`` (with dots) of a layer, as a tuple."""
    if len(names) > 1:
        return operator.attrgetter(*names)
    return (lambda layer: (operator.attrgetter(names[0])(layer),)) if names else (lambda layer: ())


class Form:
    """What a layer is, its tensors' names and contents aside: the classes, numbers and strings of its parts and their tensors'
    sizes, each found by its path from the layer, so that another layer is compared in a few calls (10 us) and not value by
    value (25).  Equal forms, like layers."""

    def __init__(self, layer: Part):
        self._values, self._tensors, self._dicts, self._shared = [], [], [], []
        self._walk(layer, "")
        paths = [tuple(x) for x in (self._values, self._tensors, self._dicts, self._shared)]
        self.names = tuple(paths)
        self._values, self._tensors, self._dicts, self._shared = map(_getter, paths)
        self.values = self._values(layer)
        self.kinds = tuple(map(type, self.values))
        self.counts = tuple(map(len, self._dicts(layer)))
        self.shared = self._shared(layer)
        if self.tensors(layer) is None:
            raise _Unlike

    def _walk(self, part: Part, path: str) -> None:
        cls = type(part)
        if not cls.__dict__.get("repeatable", False):
            raise _Unlike
        self._values.append(path + "__class__")
        self._dicts.append(path + "__dict__")
        self._shared += [path + key for key in cls.shared_attributes]
        for key, value in vars(part).items():
            if key in cls.name_attributes:
                continue
            name, kind = path + key, type(value)
            if kind in _VALUES:
                self._values.append(name)
            elif kind is torch.Tensor or kind is torch.nn.Parameter:
                self._tensors.append(name)
                self._values += (name + ".shape", name + ".dtype", name + ".device")
            elif issubclass(kind, Part):
                self._walk(value, name + ".")
            elif _plain(value):
                self._values.append(name)
            else:
                raise _Unlike

    def tensors(self, layer: Part) -> Optional[List[torch.Tensor]]:
        """The tensors of ``layer``, or ``None`` if it has not this form."""
        try:
            values, counts = self._values(layer), tuple(map(len, self._dicts(layer)))
            # (kinds before values: nothing but plain values is ever compared by value)
            if counts != self.counts or tuple(map(type, values)) != self.kinds or values != self.values:
                return None
            tensors = self._tensors(layer)
            same = all(map(operator.is_, self._shared(layer), self.shared)) and all(map(torch.Tensor.is_contiguous, tensors))
        except (AttributeError, TypeError, RuntimeError):
            return None
        return list(tensors) if same else None

    def __eq__(self, other):
        return (isinstance(other, Form) and (self.names, self.kinds, self.counts) == (other.names, other.kinds, other.counts)
                and self.values == other.values and all(map(operator.is_, self.shared, other.shared)))

    def __hash__(self):
        return hash((self.names, self.kinds, self.counts))


def _as_places(tensors: list) -> list:
    return [(tensors, i) for i in range(len(tensors))]


def form_of(layer: Part) -> Optional[Tuple[Form, list]]:
    """``(form, places of its tensors)`` of a layer, or ``None`` if it holds anything that is not repeatable."""
    try:
        form = Form(layer)
    except _Unlike:
        return None
    return form, _as_places(form.tensors(layer))


def places_of_like(layers: Iterable[Part], form: Form):
    """The places of the layers' tensors, as long as they have the form."""
    for layer in layers:
        tensors = form.tensors(layer)
        if tensors is None:
            return
        yield _as_places(tensors)


def _tensors(places: list) -> List[torch.Tensor]:
    return [where[key] for where, key in places]


def _at(tensors: List[torch.Tensor], t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else next((i for i, x in enumerate(tensors) if x is t), -1)


def repeat(recording, before, after, places: Iterable, views: list):
    """Make the launches of ``recording`` again for the layers behind the recorded one, in turn.

    ``places`` gives the tensors' places of the layer before the recorded one, of the recorded one, and of the layers to come as
    long as they have its form (it is asked for a layer's when the one before has been launched, so that the GPU is busy
    meanwhile); ``views[1:]`` are the cache views of the recorded and the coming
    ones.  ``before`` and ``after`` are the branches the recorded layer was handed and handed on (``PendingLinear``).  Returns the
    branch that the last layer hands on, ``recording.repeats`` of them having been launched; or ``None`` if the recording cannot be
    used (nothing has been launched then)."""
    from ..ops._lib import check, use_gate
    if not recording.whole or type(before) is not PendingLinear or type(after) is not PendingLinear:
        return None
    if before.x.shape != after.x.shape or before.x.dtype != after.x.dtype or (before.bias is None) != (after.bias is None):
        return None
    if any(v.group != views[1].group or v.window != views[1].window for v in views[2:]):
        return None
    places = iter(places)
    both = [_tensors(p) for p in itertools.islice(places, 2)]
    if len(both) < 2:                              # the recorded layer is not like the one before it
        return None
    first, second = both
    weight, bias = _at(second, after.weight), _at(second, after.bias)
    if weight == -1 or bias == -1 or first[weight] is not before.weight or (bias is not None and first[bias] is not before.bias):
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
    shared = [at for at in source.values() if len(at) > 1]
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
    last = None
    for view, p in zip(views[2:], places):
        x_in, x_out = x_out, x_in                  # the branch a layer hands on is the next one's
        above, mine = mine, [where[key].data_ptr() for where, key in p]
        t = table(above, mine, view, x_in, x_out)
        # one pointer for several things (tied weights): they have to be one in this layer, too
        if any(t[row][i] != t[at[0][0]][at[0][1]] for at in shared for row, i in at[1:]):
            break
        for f, args, put, what, launches, gated in calls:
            for j, row, i in put:
                args[j] = t[row][i]
            if gated is not None:                  # (a library's activation may be another thread's since)
                use_gate(gated)
            check(f(*args), what, launches)
        recording.repeats += 1
        last = PendingLinear(x_out, p[weight][0][p[weight][1]], None if bias is None else p[bias][0][p[bias][1]])
    return last
