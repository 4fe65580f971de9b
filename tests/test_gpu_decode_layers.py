"""Single-token steps with all layers in one kernel: against the plain implementation and against the same step walked, at the edges
of pages, of rounds and shares of attention, of groups of rows and of chunks; which models take it."""
import threading

import pytest
import torch

import plain_qwen3 as P
import tiny
from helpers import assert_close, poison_cache
from tiny import random_tokens

BASE = dict(tiny.TINY_F, max_position_embeddings=8192)
# name: (sizes, layers, weight scale).  Heads a kv head: 1, 3, 2, 4; columns of the stream a block: 2 or 4 (chunks side by side) to
# 18 (a group of 16 and one of 2); inputs of one chunk of 1,024, of parts of one and of ten (several passes at two rows)
SIZES = {
    "g1": dict(BASE, num_hidden_layers=2, hidden_size=384, num_attention_heads=8, num_key_value_heads=8, intermediate_size=384),
    "g3": dict(BASE, num_hidden_layers=3, hidden_size=640, num_attention_heads=6, num_key_value_heads=2, intermediate_size=1152,
               tie_word_embeddings=False, rms_norm_eps=1e-5),
    "g2": dict(BASE, num_hidden_layers=2, hidden_size=1024, num_attention_heads=16, num_key_value_heads=8, intermediate_size=3072),
    "g4": dict(tiny.WIDE, num_hidden_layers=2),
}
INIT = dict(seed=31, std_matrix=0.03, std_embedding=0.04, std_gain=0.1)


def config(name):
    tiny.CONFIGS.setdefault("layers_" + name, (SIZES[name], dict(INIT, std_matrix=0.02) if name == "g4" else INIT))
    return "layers_" + name


@pytest.fixture(scope="module")
def engines():
    from helpers import folder
    from synaptix_b200.engine import Engine
    from synaptix_b200.models import load_model
    made = {}

    def get(name, use_graphs=True):
        if (name, use_graphs) not in made:
            made.clear()
            eng = made[(name, use_graphs)] = Engine(load_model(folder(config(name)), dtype="bfloat16"), max_tokens=8192, use_graphs=use_graphs)
            poison_cache(eng)
        return made[(name, use_graphs)]
    return get


def steps(eng, prompts, given):
    """Logits of the single-token steps behind the prompts, and how many kernels one took."""
    from synaptix_b200.engine import Entry
    slots = [eng.open() for _ in prompts]
    for s, p in zip(slots, prompts):
        if p:
            eng.step([Entry(s, p, [len(p) - 1])])
    out, n = [], 0
    for row in zip(*given):
        before = eng.kernel_launches
        out.append(eng.step([Entry(s, [t], [0]) for s, t in zip(slots, row)]))
        n = eng.kernel_launches - before
    for s in slots:
        eng.close(s)
    torch.cuda.synchronize()
    eng.check_kernels()
    return torch.stack(out, 1), n


def fresh(eng):
    eng._captured.clear()
    eng._captured_decode.clear()


CASES = [("g1", (0,)), ("g1", (15, 16)), ("g1", (63,)), ("g1", (64, 0)), ("g1", (700,)), ("g3", (62, 127)), ("g3", (128,)), ("g3", (254, 255)), ("g3", (256,)),
         ("g3", (257, 3)), ("g3", (1300,)), ("g2", (40,)), ("g2", (254, 319)), ("g2", (1153, 64)), ("g4", (33,)), ("g4", (191, 320))]


@pytest.mark.gpu
@pytest.mark.parametrize("name,lens", CASES)
def test_against_the_plain_implementation_and_the_walked_step(engines, name, lens):
    from helpers import oracle
    from synaptix_b200 import ops
    eng = engines(name)
    cfg, W = oracle(config(name))
    toks = [random_tokens(cfg["vocab_size"], n + 4, 70 + i) for i, n in enumerate(lens)]
    fresh(eng)
    got, n = steps(eng, [t[:-4] for t in toks], [t[-4:] for t in toks])
    assert n <= 6                              # (the embedding, the layers, the norm, the head and what it takes)
    with ops.options(decode_layers=False):
        fresh(eng)
        walked, m = steps(eng, [t[:-4] for t in toks], [t[-4:] for t in toks])
    fresh(eng)
    assert m > n
    for i, t in enumerate(toks):
        ref = P.forward(cfg, W, t)[-4:]
        assert_close(got[i], ref, "bfloat16", f"{name} {lens} row {i}")
        # no further from the 32-bit values than the walked step, up to the scatter of two roundings of the same size
        err, other = ((x[i].float().cpu() - ref).norm() for x in (got, walked))
        assert err <= 1.3 * other + 1e-3 * ref.norm()


# the page numbers that the producers hold, 32 at a time, change at every 2,048 keys, within a share and between shares; shares
# of more pages than the ring has stages; two rows of unequal length.  Scores are made large, so that a few keys count and the others' pages tell
@pytest.mark.gpu
@pytest.mark.parametrize("lens", [(2045,), (2047,), (2050,), (4100, 60), (2049, 5000), (7950,)])
@pytest.mark.parametrize("name", ["g1", "g3"])
def test_long_contexts_against_the_walked_step(name, lens):
    from helpers import folder
    from synaptix_b200 import ops
    from synaptix_b200.engine import Engine
    from synaptix_b200.models import load_model
    model = load_model(folder(config(name)), dtype="bfloat16")
    for layer in model.layers:
        layer.mixer.scale *= 2
    eng = Engine(model, max_tokens=8192)
    poison_cache(eng)
    toks = [random_tokens(SIZES[name]["vocab_size"], n + 4, 20 + i) for i, n in enumerate(lens)]
    run = lambda: steps(eng, [t[:-4] for t in toks], [t[-4:] for t in toks])  # noqa: E731
    got, n = run()
    fresh(eng)
    with ops.options(decode_layers=False):
        want, m = run()
    assert n <= 6 < m
    for i in range(len(lens)):
        assert_close(got[i], want[i], "bfloat16", f"{name} {lens} row {i}")


@pytest.mark.gpu
@pytest.mark.parametrize("name,lens", [("g3", (100, 66)), ("g1", (20,))])
def test_without_graphs(engines, name, lens):
    from helpers import oracle
    toks = [random_tokens(oracle(config(name))[0]["vocab_size"], n + 3, 9 + n) for n in lens]
    run = lambda eng: steps(eng, [t[:-3] for t in toks], [t[-3:] for t in toks])  # noqa: E731
    want, n = run(engines(name))
    got, m = run(engines(name, use_graphs=False))
    assert torch.equal(got, want) and m == n       # every sum has one order


@pytest.mark.gpu
def test_two_engines_on_streams_of_their_own():
    from helpers import folder
    from synaptix_b200.engine import DecodeRow, Engine, Entry
    from synaptix_b200.models import load_model
    engs = [Engine(load_model(folder(config("g3")), dtype="bfloat16"), max_tokens=2048) for _ in range(2)]

    def generate(eng, seed, out):
        with torch.cuda.stream(torch.cuda.Stream()):
            s = eng.open()
            p = random_tokens(1000, 90, seed)
            eng.step([Entry(s, p, [89])])
            ses = eng.start_decode([DecodeRow(s, p[0], 0, 1)])
            for k in range(40):
                if ses.in_flight >= 2:
                    out += ses.collect()
                ses.launch()
            while ses.in_flight:
                out += ses.collect()
            ses.drop([0])
            eng.close(s)
            torch.cuda.current_stream().synchronize()
            eng.check_kernels()
    alone = [[], []]
    for i in range(2):
        generate(engs[i], i, alone[i])             # (captures, too: not while another thread works)
    both = [[], []]
    threads = [threading.Thread(target=generate, args=(engs[i], i, both[i])) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert both == alone and len(both[0]) == 40


@pytest.mark.gpu
def test_what_the_kernel_refuses():
    from synaptix_b200.ops import decode_layers_words
    assert decode_layers_words(1, 2560, 32, 8, 128, 9728, 36) > 0
    assert decode_layers_words(2, 2560, 32, 8, 128, 9728, 64) > 0
    for sizes in [(3, 2560, 32, 8, 128, 9728, 36), (0, 2560, 32, 8, 128, 9728, 36), (1, 2560, 32, 8, 64, 9728, 36), (1, 2560, 40, 8, 128, 9728, 36),
                  (1, 2560, 30, 8, 128, 9728, 36), (1, 2600, 32, 8, 128, 9728, 36), (1, 2560, 32, 8, 128, 9700, 36), (1, 256, 4, 2, 128, 384, 2),
                  (1, 2560, 32, 8, 128, 9728, 65), (1, 16384, 32, 8, 128, 9728, 2), (2, 2560, 320, 80, 128, 9728, 2)]:
        assert decode_layers_words(*sizes) == 0


def _model(name="g3", **changed):
    """A model and its cache on the CPU: what decides whether a step's layers are handed over looks at nothing else."""
    from synaptix_b200.cache import Cache
    from synaptix_b200.config import Qwen3Config
    from synaptix_b200.models import model_skeleton
    from synaptix_b200.parts import Runtime

    class Zeros:
        def __init__(self, specs):
            self.specs = specs

        def shapes(self):
            return {n: s.shape for n, s in self.specs.items()}

        def get(self, n):
            return torch.zeros(self.specs[n].shape, dtype=torch.bfloat16)
    model = model_skeleton(Qwen3Config.from_dict(dict(SIZES[name], **changed)))
    model.load(Zeros(model.all_tensor_specs()), Runtime(torch.device("cpu"), torch.bfloat16))
    cache = Cache(model.cache_requests(), max_tokens=256, max_seqs=2, dtype=torch.bfloat16, device="cpu")
    return model, cache, torch.zeros(1, SIZES[name]["hidden_size"])


def test_records_of_a_plain_model():
    from synaptix_b200.models.whole import _records
    model, cache, h = _model()
    records, k_rows, v_rows, group = _records(model, cache, h)
    assert model.runs_each_layer_once and group == 0 and len(records) == 3
    for i, r in enumerate(records):
        layer, view = model.layers[i], cache.view(i)
        assert r[:6] == [t.data_ptr() for t in (layer.mixer.qkv.weight, layer.mixer.o.weight, layer.ffn.gate_up.weight, layer.ffn.down.weight,
                                                layer.norm1.weight, layer.norm2.weight)]
        assert k_rows[r[8]:].data_ptr() == view.k.data_ptr() and v_rows[r[8]:].data_ptr() == view.v.data_ptr()
        assert r[8] + view.k.numel() // 128 <= k_rows.shape[0]


def _wrap(model):
    layer = model.layers[1]
    forward = layer.forward
    layer.forward = lambda *a, **k: forward(*a, **k)


@pytest.mark.parametrize("change", [
    _wrap,
    lambda m: setattr(m.layers[2].norm2, "eps", 1e-3),
    lambda m: setattr(m.layers[1].mixer, "scale", 0.5),
    lambda m: setattr(m.layers[1].mixer, "window", 64),
    lambda m: setattr(m.layers[0].mixer, "sinks", torch.zeros(6)),
    lambda m: setattr(m.layers[2].mixer.position, "inv_freq", m.layers[2].mixer.position.inv_freq.clone()),
    lambda m: setattr(m.layers[1].ffn.down, "bias", torch.zeros(640)),
    lambda m: setattr(m.layers[1].ffn.down, "weight", m.layers[1].ffn.down.weight.float()),
    lambda m: setattr(m.layers[2].mixer, "wq", None),
    lambda m: m.layers[0].mixer.qkv.__setattr__("weight", m.layers[0].mixer.qkv.weight.t().contiguous().t()),
])
def test_other_layers_are_walked(change):
    from synaptix_b200.models.whole import _records
    model, cache, h = _model()
    change(model)
    assert _records(model, cache, h) is None


def test_where_the_blocks_have_no_room(monkeypatch):
    """A launch that the device refuses for want of SMs leaves the step to the walk, also when it is captured; any other error is raised."""
    from synaptix_b200.models import whole
    from synaptix_b200.ops import KernelError, layers
    from synaptix_b200.parts import Runtime
    from synaptix_b200.parts.base import StepContext
    model, cache, h = _model()
    codes, calls = [10006], []
    monkeypatch.setattr(whole.ops, "decode_layers_words", lambda *a: 64)
    monkeypatch.setattr(layers, "decode_layers_words", lambda *a: 64)
    monkeypatch.setattr(layers, "require_cuda", lambda *a: None)
    monkeypatch.setattr(layers, "raw_stream", lambda: 0)
    monkeypatch.setattr(layers, "launcher", lambda *a: lambda *args: calls.append(args) or codes[0])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)

    def ctx():
        i32 = lambda *x: torch.zeros(*x, dtype=torch.int32)  # noqa: E731
        return StepContext(all_single=True, n_seqs=1, runtime=Runtime(torch.device("cpu"), torch.bfloat16), seq_lens=i32(1), block_tables=[i32(1, 4)])
    c = ctx()
    assert not whole.run_layers(model, h, c, cache) and len(calls) == 1
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert not whole.run_layers(model, h, c, cache) and len(calls) == 1
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    codes[0] = 0
    assert whole.run_layers(model, h, ctx(), cache) and len(calls) == 2
    codes[0] = 700
    with pytest.raises(KernelError):
        whole.run_layers(model, h, ctx(), cache)


def test_other_models_are_walked():
    from synaptix_b200.models.whole import _records
    assert _records(*_model(use_sliding_window=True, sliding_window=64, max_window_layers=1)) is None
    model, cache, h = _model()
    assert _records(model, cache, torch.zeros(1, 512)) is None
    model.steps = model.steps[:1] + model.steps[:1]
    assert not model.runs_each_layer_once
