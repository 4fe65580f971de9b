"""Launches of layers of one form made again with other pointers: which layers are alike, which pointers are put in, and (on the
GPU) that a prompt step gives the same bits as one that walks every layer."""
import ctypes
import sys
import threading
import types

import pytest
import torch

import tiny
from synaptix_b200.models import model_skeleton
from synaptix_b200.models.repeat import form_of, repeat
from synaptix_b200.ops import _lib
from synaptix_b200.parts import Linear, RMSNorm
from synaptix_b200.parts.base import Part, PendingLinear

QWEN3 = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=7, hidden_size=256, num_attention_heads=4,
             num_key_value_heads=2, head_dim=128, intermediate_size=320, vocab_size=997, rope_theta=10000.0, rms_norm_eps=1e-6,
             tie_word_embeddings=True, max_position_embeddings=4096, hidden_act="silu", attention_bias=False, use_sliding_window=False)


def skeleton(**more):
    from synaptix_b200.config import Qwen3Config
    return model_skeleton(Qwen3Config.from_dict(dict(QWEN3, **more)))


def test_forms():
    layers = skeleton().layers
    assert len({form_of(x)[0] for x in layers}) == 1
    windowed = skeleton(use_sliding_window=True, sliding_window=64, max_window_layers=3).layers
    forms = [form_of(x)[0] for x in windowed]
    assert len(set(forms[:3])) == 1 and len(set(forms[3:])) == 1 and forms[2] != forms[3]

    class Other(RMSNorm):           # says nothing of itself: never repeated
        pass
    layers[0].norm1.__class__ = Other
    assert form_of(layers[0]) is None and form_of(layers[1]) is not None
    layers[1].extra = object()
    assert form_of(layers[1]) is None


def test_strings_of_a_form():
    """Names of tensors differ between like layers; any other string may decide what a part does."""
    forms = [form_of(x)[0] for x in skeleton().layers]
    assert len(set(forms)) == 1

    class Scored(RMSNorm):
        repeatable = True

        def __init__(self, name, scoring):
            super().__init__(name, 8, 1e-6)
            self.scoring, self.by_kind = scoring, {scoring: 1}
    a, b, c = form_of(Scored("a", "softmax"))[0], form_of(Scored("b", "softmax"))[0], form_of(Scored("a", "sigmoid"))[0]
    assert a == b and a != c
    d = Scored("a", "softmax")
    d.by_kind = {"sigmoid": 1}
    assert form_of(d)[0] != a
    a, b = (form_of(Linear(n, 4, 4, kind=k))[0] for n, k in (("a", "matrix"), ("b", "embedding")))
    assert a != b


def test_tensors_that_a_step_makes_something_of():
    """Layers that rotate by another tensor of frequencies are not alike, whatever its sizes: a step's tables of cosines and sines
    belong to the tensor they were made of."""
    for part, key in ((lambda x: x.mixer.position, "inv_freq"), (lambda x: x.mixer, "_inv_freq")):
        layers, one = skeleton().layers, torch.ones(64)
        for x in layers:
            setattr(part(x), key, one)
        assert len({form_of(x)[0] for x in layers}) == 1
        setattr(part(layers[4]), key, torch.ones(64))
        forms = [form_of(x)[0] for x in layers]
        assert forms[4] != forms[0] and len(set(forms)) == 2


def test_pointers_are_put_in():
    n, made = 5, []

    class Launch:
        argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]

        def __call__(self, *args):
            made.append(args)
            return 0
    launch = Launch()
    weights = [[torch.zeros(4, 4), torch.zeros(4)] for _ in range(n)]
    views = [types.SimpleNamespace(k=torch.zeros(2), v=torch.zeros(2), group=0, window=None) for _ in range(n)]
    places = [[(w, 0), (w, 1)] for w in weights]
    z = [torch.zeros(3, 4), torch.zeros(3, 4)]
    inside = torch.zeros(3, 4)

    def calls(i, read, write):      # what layer i launches
        return [(read.data_ptr(), weights[i - 1][0].data_ptr(), inside.data_ptr(), 7),
                (weights[i][1].data_ptr(), views[i].k.data_ptr(), views[i].v.data_ptr(), 8),
                (inside.data_ptr(), write.data_ptr(), None, 9)]

    def record(whole=True):
        with _lib.recording() as r:
            for a in calls(1, z[0], z[1]):
                _lib.launch(launch, a, "test")
            if not whole:
                _lib.check(0, "a launch of another kind")
        return r
    before, after = PendingLinear(z[0], weights[0][0]), PendingLinear(z[1], weights[1][0])
    r = record()
    made.clear()
    done = repeat(r, before, after, places, views)
    want = [a for i in range(2, n) for a in calls(i, z[(i + 1) % 2], z[i % 2])]
    assert made == want
    assert done.weight is weights[n - 1][0] and done.bias is None and done.x is z[(n - 1) % 2]
    made.clear()
    assert repeat(record(whole=False), before, after, places, views) is None
    assert repeat(record(), PendingLinear(z[0], torch.zeros(4, 4)), after, places, views) is None
    with _lib.recording() as r:      # a pointer into the middle of a weight
        _lib.launch(launch, (weights[1][0].data_ptr() + 16, None, None, 7), "test")
    assert repeat(r, before, after, places, views) is None
    views[3].group = 1
    assert repeat(record(), before, after, places, views) is None
    with _lib.gate_activation(form="gelu_tanh"):
        assert not record().whole
    with _lib.late_launch():
        assert not record().whole


# ---- a decoder of layers that launch nothing real: what a prompt step launches, walked and repeated ----

class Launches:
    """Stands for a library's function: notes what it is called with."""
    argtypes = [ctypes.c_void_p] * 6 + [ctypes.c_int]

    def __init__(self):
        self.made = []

    def __call__(self, *args):
        self.made.append(args)
        return 0


class Toy(Part):
    """One launch a layer: the branch before, its weight, this layer's vector and cache, the branch handed on, a number."""
    repeatable = True
    takes_pending_product = True

    def __init__(self, window=7):
        self.weight, self.vector, self.window = torch.zeros(4, 4), torch.zeros(4), window

    def forward(self, h, pending, ctx, view, write_cache=True):
        z = torch.zeros(3, 4)
        x, w = (None, None) if pending is None else (pending.x.data_ptr(), pending.weight.data_ptr())
        _lib.launch(ctx.f, (x, w, self.vector.data_ptr(), view.k.data_ptr(), view.v.data_ptr(), z.data_ptr(), self.window), "toy", 1, (z,))
        return h, PendingLinear(z, self.weight)


def toy_model(layers):
    from synaptix_b200.models.decoder import DecoderModel
    embedding = types.SimpleNamespace(forward_step=lambda ctx, view=None: torch.zeros(3, 4))
    norm = types.SimpleNamespace(takes_pending_product=True, add_forward=lambda h, pending, rows=None: pending.weight)
    return DecoderModel(None, embedding, layers, norm, types.SimpleNamespace(forward=lambda x: x))


def toy_step(model, views, on=True):
    """What the step launched, without the branches' places, and the weight of the branch it ended with."""
    from synaptix_b200 import ops
    f = Launches()
    ctx = types.SimpleNamespace(all_single=False, host={}, want_rows=None, observe=None, want_all=False, f=f)
    with ops.options(repeat_layers=on):
        last = model.forward(ctx, types.SimpleNamespace(view=lambda i: views[i]))
    assert [a[0] for a in f.made[1:]] == [a[5] for a in f.made[:-1]]          # each reads what the one before wrote
    return [a[1:5] + a[6:] for a in f.made], last.data_ptr()


def toy_views(n):
    return [types.SimpleNamespace(k=torch.zeros(2), v=torch.zeros(2), group=0, window=None) for _ in range(n)]


def toy(n=8):
    views = toy_views(n)
    model = toy_model([Toy() for _ in range(n)])
    walked = [0]
    forward = Toy.forward

    def counted(self, *args):
        walked[0] += 1
        return forward(self, *args)
    return model, views, walked, counted


def test_steps_after_a_change(monkeypatch):
    """A layer put in, a number changed, a ``forward`` wrapped or a model loaded anew between two prompt steps count in the next."""
    model, views, walked, counted = toy()
    monkeypatch.setattr(Toy, "forward", counted)

    def same(expected):
        want, walked[0] = toy_step(model, views, on=False), 0
        assert toy_step(model, views) == want
        assert walked[0] == expected
    same(2)                                       # the first two layers; the other six are repeated
    model.layers[5] = Toy()
    same(2)
    model.layers[6].window = 64
    same(4)                                       # ... the seventh is another, and the last is too short a stretch
    model.layers[6].window = 7
    same(2)
    seen, inner = [], model.layers[7].forward
    model.layers[7].forward = lambda *args: seen.append(1) or inner(*args)
    same(3)
    assert len(seen) == 2
    del model.layers[7].forward
    for layer in model.layers:
        layer.weight, layer.vector = torch.zeros(4, 4), torch.zeros(4)
    same(2)



def test_one_tensor_in_two_places(monkeypatch):
    """Where a pointer of the recorded layer stands for two of its tensors, or for one of the layer before, too, and the other
    layers' do not, the launches are not made again with it."""
    model, views, walked, counted = toy()
    monkeypatch.setattr(Toy, "forward", counted)
    plain = [(x.weight, x.vector) for x in model.layers]

    def same(expected):
        want, walked[0] = toy_step(model, views, on=False), 0
        assert toy_step(model, views) == want and walked[0] == expected
        for x, (w, v) in zip(model.layers, plain):
            x.weight, x.vector = w, v
    same(2)
    model.layers[1].weight = model.layers[0].weight
    same(3)                                       # the third layer is walked, and what it launched is made again
    model.layers[1].vector = model.layers[1].weight.view(-1)[:4]
    same(4)                                       # (the second layer is the one before the third, too)
    for x in model.layers:                        # in every layer: one pointer for both
        x.vector = x.weight.view(-1)[:4]
    same(2)
    for x in model.layers:                        # one tensor for all layers
        x.vector = plain[0][1]
    same(2)


def test_pointers_into_the_middle():
    """A pointer into the middle of the branch that comes in or goes out, or of a weight behind a tensor that lies in it, has
    another one in its place in the next layer."""
    z = [torch.zeros(3, 4), torch.zeros(3, 4)]
    w = [[x, x[0], torch.zeros(4)] for x in (torch.zeros(4, 4) for _ in range(5))]
    for a in (z[0], z[1], w[1][0]):
        with _lib.recording() as r:
            _lib.launch(Launches(), (a.data_ptr() + 32, w[1][2].data_ptr(), None, None, None, None, 0), "test")
        assert repeat(r, PendingLinear(z[0], w[0][0]), PendingLinear(z[1], w[1][0]), [[(x, i) for i in range(3)] for x in w], toy_views(5)) is None



def test_activation_is_told_again(monkeypatch):
    """Between two of the launches that are made again, another thread may tell the library another activation."""
    told = []
    lib = types.SimpleNamespace(sx_set_gate_act=lambda alpha, limit, form: told.append(form.value))
    monkeypatch.setitem(_lib._LIBS, "toy", lib)
    monkeypatch.setitem(_lib._LIB_GATE, "toy", None)
    seen = []

    def others():
        with _lib.gate_activation(form="gelu_tanh"):
            _lib.use_gate("toy")

    class Shared(Launches):
        def __call__(self, *args):
            seen.append(told[-1])
            t = threading.Thread(target=others)
            t.start()
            t.join()
            return super().__call__(*args)
    n, forward = 8, Toy.forward

    def gated(self, h, pending, ctx, view, write_cache=True):
        _lib.use_gate("toy")
        return forward(self, h, pending, ctx, view, write_cache)
    monkeypatch.setattr(Toy, "forward", gated)
    monkeypatch.setattr(sys.modules[__name__], "Launches", Shared)
    toy_step(toy_model([Toy() for _ in range(n)]), toy_views(n))
    assert seen == [0] * n


@pytest.mark.gpu
@pytest.mark.parametrize("more", [{}, dict(head_dim=64), dict(use_sliding_window=True, sliding_window=64, max_window_layers=2)])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_same_bits(more, dtype):
    from synaptix_b200 import ops
    from synaptix_b200.api import LLM
    from synaptix_b200.engine import Entry
    from synaptix_b200.parts import Runtime
    from synaptix_b200.weights import RandomSource
    model = skeleton(**more)
    model.load(RandomSource(model.all_tensor_specs(), seed=1, device="cuda:0"),
               Runtime(torch.device("cuda:0"), torch.bfloat16 if dtype == "bf16" else torch.float32))
    engine = LLM.from_model(model, max_tokens=4096, max_batch=8).engine

    def run(on, lens):
        with ops.options(repeat_layers=on):
            slots = [engine.open() for _ in lens]
            before = engine.kernel_launches
            out = [engine.step([Entry(s, tiny.random_tokens(997, n, n), [0, n - 1]) for s, n in zip(slots, lens)])]
            launches = engine.kernel_launches - before
            out.append(engine.step([Entry(s, tiny.random_tokens(997, 3, n), [2]) for s, n in zip(slots, lens)]))   # behind a cache
            out.append(engine.step([Entry(s, [5], [0]) for s in slots]))
            for s in slots:
                engine.close(s)
        return out, launches
    for lens in ([2], [17], [100, 33], [161], [300, 5, 260], [1000]):
        (a, n), (b, m) = run(False, lens), run(True, lens)
        assert n == m and all(torch.equal(x, y) for x, y in zip(a, b)), lens


def attention_with_everything(old, i):
    """A layer's attention again, with biases, sinks and a rotation of a quarter of each head."""
    from synaptix_b200.parts import Attention, RotaryHalf
    return Attention(old.prefix, old.width, old.nh, old.nkv, old.hd, position=RotaryHalf(old.hd, 10000.0, old.hd // 4),
                     qk_norm_eps=old.qk_norm_eps, window=old.window, bias_suffix=".b", sinks=True)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype,repeats", [("plain", "bf16", True), ("windows", "bf16", True), ("everything", "bf16", True),
                                                ("heads of 64", "bf16", False), ("plain", "f32", False)])
def test_which_steps_repeat(kind, dtype, repeats, monkeypatch):
    """Prompt steps of bfloat16 layers with heads of 128 make the launches again (and give the bits of a walk); where an operation
    does not note its launches every layer is walked.  A model that is loaded anew runs with its new weights."""
    from synaptix_b200 import ops
    from synaptix_b200.api import LLM
    from synaptix_b200.engine import Entry
    from synaptix_b200.models import decoder
    from synaptix_b200.parts import Runtime, SwiGLU
    from synaptix_b200.weights import RandomSource
    model = skeleton(**{"heads of 64": dict(head_dim=64), "windows": dict(use_sliding_window=True, sliding_window=64, max_window_layers=0)}.get(kind, {}))
    if kind == "everything":
        for i, layer in enumerate(model.layers):
            layer.mixer = attention_with_everything(layer.mixer, i)
            layer.ffn = SwiGLU("model.layers.%d.mlp." % i, 256, 320, bias_suffix=".b")
    made = []

    def noted(*args):
        done = repeat(*args)
        made.append(done is not None)
        return done
    monkeypatch.setattr(decoder, "repeat", noted)

    def load(seed):
        model.load(RandomSource(model.all_tensor_specs(), seed=seed, device="cuda:0"),
                   Runtime(torch.device("cuda:0"), torch.bfloat16 if dtype == "bf16" else torch.float32))
    load(1)
    engine = LLM.from_model(model, max_tokens=4096, max_batch=8).engine

    def run(on, lens):
        del made[:]
        with ops.options(repeat_layers=on):
            slots = [engine.open() for _ in lens]
            out = [engine.step([Entry(s, tiny.random_tokens(997, n, n), [0, n - 1]) for s, n in zip(slots, lens)]) for _ in range(1)]
            for s in slots:
                engine.close(s)
        return out, sum(made)
    run(True, [300])                  # what a part makes of its own when it first runs is made
    first = None
    for seed in (1, 2):
        if seed == 2:
            load(2)
            run(True, [300])
        for lens in ([161], [300, 5, 260], [1000]):
            (a, none), (b, n) = run(False, lens), run(True, lens)
            assert none == 0 and n == (1 if repeats else 0), lens
            assert all(torch.equal(x, y) for x, y in zip(a, b)) and all(torch.isfinite(x).all() for x in a), lens
        assert first is None or not torch.equal(first, a[0])
        first = a[0]
