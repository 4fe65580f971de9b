"""Workloads of the library on one B200, for measuring it: prompt steps and generation with whole models.

Every case is what a program does that keeps a loaded model and is handed token ids: prompts of a batch run as one step
of the engine, then single-token steps run as a decode session (what ``LLM.generate`` does: sampling and the move to the
next token on the device, tokens read back one step behind), then one more step whose logits are kept, and the slots are
given back.  The tokens that run in the single-token steps are GIVEN, as the replay program gives them, so that two
implementations that differ by rounding run the same sequences; the session samples all the same.  A pass returns the
logits at the prompts' ends and those of the last step, which see everything the cache holds.

Models: the Qwen3 dense decoder at its published sizes with all its layers, and the Pidutar hybrid decoder (matrix
memories, windowed attention over a cached latent, layers that read another layer's cache, mixture of experts) with eight
layers, the sizes of ``bench.py``.  Weights are random and belong to the case's model, not to the seed: a program loads a
model once.  The seed draws the prompts and the given tokens.
"""
import gc
import hashlib
import math
import random

import torch

QWEN3 = {  # name: layers, width, query heads, feed-forward, output head shares the embedding (8 kv heads, head size 128)
    "qwen3-0.6b": (28, 1024, 16, 3072, True),
    "qwen3-1.7b": (28, 2048, 16, 6144, True),
    "qwen3-4b": (36, 2560, 32, 9728, True),
}
QWEN3_VOCAB, KV_HEADS, HEAD = 151936, 8, 128
PIDUTAR = {  # name: width, feed-forward weights a token uses (4 experts of a quarter), heads, head size, memory heads
    "pidutar-1k": (1024, 4096, 16, 64, 8),
    "pidutar-2.5k": (2560, 9728, 32, 128, 8),
}
PIDUTAR_LAYERS, PIDUTAR_VOCAB, EXPERTS, TOP, WINDOW = 8, 32000, 16, 4, 1000

TOP_P = "temperature 0.8, top-k 50, top-p 0.9"


def listed():
    def case(name, model, batch, prompt, new, dtype="bf16", sampling="greedy"):
        return {"name": name, "model": model, "dtype": dtype, "batch": batch, "prompt": prompt, "new": new, "sampling": sampling}
    return [
        # one short question to a small model: every step is a few dozen microseconds of work, launches and latency count
        case("small_chat", "qwen3-0.6b", 1, 19, 24),
        # the true 32-bit path (reference runs, debugging a model): two short prompts and a few tokens
        case("float32", "qwen3-0.6b", 2, 150, 8, dtype="f32"),
        # a middling prompt to a middling model: a few hundred rows, fewer tiles than the GPU has SMs
        case("prompt_611", "qwen3-1.7b", 1, 611, 0),
        # short prompts of several users in one step (64 to 127 tokens each), no decoding: time to the first token
        case("short_prompts", "qwen3-4b", 5, 127, 0),
        # the benchmark's prompt step
        case("prompt_2048", "qwen3-4b", 1, 2048, 0),
        # a long document
        case("prompt_8191", "qwen3-4b", 1, 8191, 0),
        # one user, a few pages of context: decoding bound by reading the weights
        case("decode_b1", "qwen3-4b", 1, 1500, 64),
        # the benchmark's batch, prompts of unequal lengths, sampled
        case("decode_b8", "qwen3-4b", 8, 1100, 48, sampling=TOP_P),
        # a busy server: many short sequences
        case("decode_b48", "qwen3-4b", 48, 200, 32),
        # the hybrid with experts: its prompt step and its decoding
        case("hybrid_prompt", "pidutar-2.5k", 1, 2048, 0),
        case("hybrid_decode", "pidutar-2.5k", 8, 700, 48),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """A prompt step or a generation: models, batches and lengths between the listed ones', at most 8,192 prompt tokens."""
    dtype = "f32" if rng.random() < 0.1 else "bf16"
    model = "qwen3-0.6b" if dtype == "f32" else rng.choice(["qwen3-0.6b", "qwen3-1.7b", "qwen3-4b", "qwen3-4b", "pidutar-1k", "pidutar-2.5k"])
    generate = rng.random() < 0.55
    batch = _log(rng, 1, 2 if dtype == "f32" else 48) if generate else _log(rng, 1, 6)
    most = 300 // batch if dtype == "f32" else min(8191, 8192 // batch)
    prompt = _log(rng, 16, min(most, 1500) if generate else most)
    new = rng.randint(4, 8 if dtype == "f32" else 48) if generate else 0
    return {"model": model, "dtype": dtype, "batch": batch, "prompt": prompt, "new": new,
            "sampling": rng.choice(["greedy", TOP_P]) if generate else "greedy"}


def _lengths(case):
    """Prompt lengths of the batch: the longest is ``prompt``, the others between half of it and all of it."""
    n, p = case["batch"], case["prompt"]
    return [p - (i * 37) % (p // 2 + 1) for i in range(n)]


# ---- models and weights ---------------------------------------------------------------------------------------------

def _config(name):
    if name in QWEN3:
        layers, width, heads, ff, tied = QWEN3[name]
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=layers, hidden_size=width,
                    num_attention_heads=heads, num_key_value_heads=KV_HEADS, head_dim=HEAD, intermediate_size=ff,
                    vocab_size=QWEN3_VOCAB, rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=tied,
                    max_position_embeddings=40960, hidden_act="silu", attention_bias=False, use_sliding_window=False)
    width, ff, heads, hd, mem = PIDUTAR[name]
    mlp = dict(kind="moe", expert=dict(ff=ff // 4), router=dict(experts=EXPERTS, top=TOP, scale=1.0))
    att = dict(heads=heads, dim=hd // 2, rot_dim=hd // 2, vdim=hd, q_rank=width // 2, kv_rank=width // 8, scale=hd ** -0.5,
               mask=dict(size=WINDOW), rot=dict(dims=hd // 2, base=1.0e6))
    kinds = [dict(type="mlstm", mixer=dict(heads=mem, dim=hd, vdim=hd, gate_cap=15.0), mlp=mlp),
             dict(type="latent_attention", mixer=att, mlp=mlp), None, dict(type="latent_attention", mixer=att, mlp=mlp)]
    layers = [kinds[i % 4] or dict(type="latent_attention", mixer=dict(att, kv_from=i - 1), mlp=mlp) for i in range(PIDUTAR_LAYERS)]
    return dict(architecture="Pidutar", vocab=PIDUTAR_VOCAB, width=width, norm=dict(eps=1e-5), embedding=dict(scale=1.0),
                residual_mult=0.5, logit_scale=1.0, layers=layers)


def _shapes(name):
    """Every tensor of the model: name -> (shape, mean, standard deviation).  What ends a branch is drawn smaller the more
    layers there are, and the embedding is a good part of the stream, so that rounding does not grow through the layers as
    it would in a stack of equally loud random layers (trained models are as steady)."""
    cfg, out = _config(name), {}

    def put(key, *shape, std=0.02, mean=0.0):
        out[key] = (shape, mean, std)

    if name in QWEN3:
        w, ff = cfg["hidden_size"], cfg["intermediate_size"]
        q, kv = cfg["num_attention_heads"] * HEAD, KV_HEADS * HEAD
        quiet = 0.02 / math.sqrt(2 * cfg["num_hidden_layers"])
        put("model.embed_tokens.weight", QWEN3_VOCAB, w, std=0.05)
        for i in range(cfg["num_hidden_layers"]):
            p = "model.layers.%d." % i
            for key, shape in (("self_attn.q_proj", (q, w)), ("self_attn.k_proj", (kv, w)), ("self_attn.v_proj", (kv, w)),
                               ("self_attn.o_proj", (w, q)), ("mlp.gate_proj", (ff, w)), ("mlp.up_proj", (ff, w)), ("mlp.down_proj", (w, ff))):
                put(p + key + ".weight", *shape, std={"self_attn.o_proj": quiet, "mlp.down_proj": 0.2 * quiet}.get(key, 0.02))
            for key, n in (("input_layernorm", w), ("post_attention_layernorm", w), ("self_attn.q_norm", HEAD), ("self_attn.k_norm", HEAD)):
                put(p + key + ".weight", n, mean=1.0, std=0.05)
        put("model.norm.weight", w, mean=1.0, std=0.05)
        return out
    w, v = cfg["width"], cfg["vocab"]
    quiet = 0.02 / math.sqrt(2 * PIDUTAR_LAYERS)
    put("embed", v, w, std=1.0)
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = "l%d." % i, layer["mixer"], layer["mlp"]
        for key in ("ls1", "ls2"):
            put(p + key, w, mean=1.0, std=0.05)
        for key in ("norm1", "norm2"):
            put(p + key, w, std=0.05)
        if layer["type"] == "mlstm":
            h, d, dv = m["heads"], m["dim"], m["vdim"]
            for key, n in (("q", h * d), ("k", h * d), ("v", h * dv), ("g", h * dv), ("i", h), ("f", h)):
                put(p + "mix." + key, n, w)
            put(p + "mix.i.b", h, std=0.1)
            put(p + "mix.f.b", h, mean=3.0, std=0.1)     # (memories that last tens of tokens)
            put(p + "mix.norm", h * dv, mean=1.0, std=0.05)
            put(p + "mix.o", w, h * dv, std=quiet)
        else:
            h, d, r, dv, qr, kr = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["q_rank"], m["kv_rank"]
            put(p + "mix.dq", qr, w)
            put(p + "mix.dq.norm", qr, mean=1.0, std=0.05)
            put(p + "mix.uq", h * (d + r), qr)
            if m.get("kv_from") is None:
                put(p + "mix.dkv", kr + r, w)
                put(p + "mix.dkv.norm", kr, mean=1.0, std=0.05)
            put(p + "mix.uk", h * d, kr)
            put(p + "mix.uv", h * dv, kr)
            put(p + "mix.g", h, w)
            put(p + "mix.o", w, h * dv, std=quiet)
        put(p + "mlp.router", EXPERTS, w, std=0.06)      # (logits of a few units, as trained routers have them)
        for e in range(EXPERTS):
            put(p + "mlp.e%d.gate" % e, f["expert"]["ff"], w)
            put(p + "mlp.e%d.up" % e, f["expert"]["ff"], w)
            put(p + "mlp.e%d.down" % e, w, f["expert"]["ff"], std=quiet)
    put("final.norm", w, std=0.05)
    put("head", v, w)
    return out


class _Weights:
    """The model's weights by name, drawn on the GPU in bfloat16, each tensor from a stream of its own."""

    def __init__(self, model):
        self.model, self.specs = model, _shapes(model)

    def shapes(self):
        return {n: s[0] for n, s in self.specs.items()}

    def get(self, name):
        shape, mean, std = self.specs[name]
        g = torch.Generator(device="cuda")
        g.manual_seed(int.from_bytes(hashlib.sha256(("%s:%s" % (self.model, name)).encode()).digest()[:6], "little"))
        return (torch.randn(shape, generator=g, device="cuda") * std + mean).to(torch.bfloat16)


_loaded = {}  # the loaded model of the case at hand: a program keeps one


def _engine(case):
    from synaptix_b200.api import LLM
    from synaptix_b200.config import PidutarConfig, Qwen3Config
    from synaptix_b200.models import model_skeleton
    from synaptix_b200.parts import Runtime
    key = (case["model"], case["dtype"])
    if key not in _loaded:
        _loaded.clear()
        gc.collect()
        torch.cuda.empty_cache()
        cfg = (Qwen3Config if case["model"] in QWEN3 else PidutarConfig).from_dict(_config(case["model"]))
        model = model_skeleton(cfg)
        model.load(_Weights(case["model"]), Runtime(torch.device("cuda:0"), torch.float32 if case["dtype"] == "f32" else torch.bfloat16))
        _loaded[key] = LLM.from_model(model, max_tokens=4096 if case["dtype"] == "f32" else 16384, max_batch=64)
    return _loaded[key].engine


def _tokens(case, seed):
    """(prompts, given): token ids of each sequence's prompt, and of its single-token steps (the last one's logits are kept)."""
    rng = random.Random(seed)
    vocab = QWEN3_VOCAB if case["model"] in QWEN3 else PIDUTAR_VOCAB
    prompts = [[rng.randrange(vocab) for _ in range(n)] for n in _lengths(case)]
    given = [[rng.randrange(vocab) for _ in range(case["new"] + 1 if case["new"] else 0)] for _ in prompts]
    return prompts, given


# ---- one pass -------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    from synaptix_b200.sampling import SamplingParams
    prompts, given = _tokens(case, seed)
    params = SamplingParams(temperature=0.8, top_k=50, top_p=0.9) if case["sampling"] == TOP_P else SamplingParams()
    return {"engine": _engine(case), "prompts": prompts, "given": given, "params": params}


def run(state):
    from synaptix_b200.engine import DecodeRow, Entry
    from synaptix_b200.sampling import Sampler
    engine, prompts, given, params = (state[k] for k in ("engine", "prompts", "given", "params"))
    slots = [engine.open() for _ in prompts]
    out = {"prompt": engine.step([Entry(s, p, [len(p) - 1]) for s, p in zip(slots, prompts)])}
    if given[0]:
        # the prompt step's draw is read back before decoding starts
        Sampler(params, engine.device).sample_to_host(out["prompt"], list(range(len(slots))), [0] * len(slots), None)
        session = engine.start_decode([DecodeRow(s, t[0], i, 1) for i, (s, t) in enumerate(zip(slots, given))], params)
        session.launch()
        for k in range(1, len(given[0]) - 1):
            if session.in_flight >= 2:
                session.collect()
            session.launch([t[k] for t in given])
        while session.in_flight:
            session.collect()
        session.drop(list(range(len(slots))))
        out["last"] = engine.step([Entry(s, [t[-1]], [0]) for s, t in zip(slots, given)])
    for s in slots:
        engine.close(s)
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def work(case):
    """Bytes: every matrix that a step uses once a step, the cached tokens read once a layer and single-token step, the
    logits written.  Flops: the products and the attention of every token."""
    size = 4 if case["dtype"] == "f32" else 2
    cfg, shapes = _config(case["model"]), _shapes(case["model"])
    lens, steps, n = _lengths(case), case["new"] + 1 if case["new"] else 0, case["batch"]
    head_key = "model.embed_tokens.weight" if case["model"] in QWEN3 else "head"
    total = lambda keys: sum(math.prod(shapes[k][0]) for k in keys)  # noqa: E731
    expert = [k for k in shapes if ".mlp.e" in k]
    fixed = total(k for k in shapes if k not in (head_key, "embed", "model.embed_tokens.weight") and k not in expert)
    head, experts = total([head_key]), total(expert)
    if case["model"] in QWEN3:
        layers = cfg["num_hidden_layers"]
        per_key = layers * 2 * KV_HEADS * HEAD                       # cached elements a token
        key_flops = layers * 4 * cfg["num_attention_heads"] * HEAD   # a (query, key) pair
        seen, state = None, 0
        active = fixed
    else:
        width, _, heads, hd, mem = PIDUTAR[case["model"]]
        attention = [x for x in cfg["layers"] if x["type"] == "latent_attention"]
        per_key = len(attention) * (width // 8 + hd // 2)
        key_flops = len(attention) * 4 * heads * hd
        seen, state = WINDOW, (PIDUTAR_LAYERS - len(attention)) * mem * hd * hd
        active = fixed + experts * TOP / EXPERTS

    def pairs(length):     # (query, key) pairs of a whole prompt
        if seen is None or length <= seen:
            return length * (length + 1) / 2
        return seen * (seen + 1) / 2 + (length - seen) * seen

    def used(tokens):      # share of the experts that so many tokens choose among them
        return 1 - (1 - TOP / EXPERTS) ** tokens

    flops = sum(2 * active * t + key_flops * pairs(t) + 4 * state * t + 2 * head for t in lens)
    nbytes = size * (fixed + experts * used(sum(lens)) + head + per_key * sum(lens)) + 4 * n * shapes[head_key][0][0]
    for k in range(steps):
        keys = [min(t + k + 1, seen or t + k + 1) for t in lens]
        nbytes += size * (fixed + experts * used(n) + head + per_key * sum(keys)) + 2 * 4 * state * n
        flops += n * (2 * (active + head) + 4 * state) + key_flops * sum(keys)
    return {"bytes": nbytes + (4 * n * shapes[head_key][0][0] if steps else 0), "flops": flops}


def tolerance(case):
    # float32: 1.3e-6 off the 64-bit values was measured; two orders of the sums differ by as much.  bfloat16: 0.0018 (hybrid)
    # to 0.0048 off the 64-bit values, so two implementations differ by up to 0.007 (a tie in a router may fall the other way)
    return {"rel": 1e-5, "max": 1e-4} if case["dtype"] == "f32" else {"rel": 0.02, "max": 0.2}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------

def exact(case, seed):
    """Whole sequences without a cache, in 64 bits, from the equations."""
    prompts, given = _tokens(case, seed)
    seqs = [p + g for p, g in zip(prompts, given)]
    ends = [0]
    for s in seqs:
        ends.append(ends[-1] + len(s))
    with torch.no_grad():
        ids = torch.tensor([t for s in seqs for t in s], device="cuda")
        spans = list(zip(ends, ends[1:]))
        rows = [a + len(p) - 1 for (a, _), p in zip(spans, prompts)] + ([b - 1 for _, b in spans] if case["new"] else [])
        logits = (_qwen3 if case["model"] in QWEN3 else _pidutar)(case["model"], ids, spans, torch.tensor(rows, device="cuda"))
    out = {"prompt": logits[:len(seqs)]}
    if case["new"]:
        out["last"] = logits[len(seqs):]
    return out


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window=None):
    """One sequence: q [T, H, d], k and v [T, G, d] with H / G query heads a key head; causal, the last ``window`` keys."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    i = torch.arange(T, device=q.device)
    hidden = (i[None, :] > i[:, None]) | (i[None, :] <= i[:, None] - (window or T + 1))
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        out[:, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v[:, h * G // H]
    return out


def _qwen3(model, ids, spans, rows):
    cfg, src = _config(model), _Weights(model)
    W = lambda name: src.get(name).double()  # noqa: E731
    eps, heads = cfg["rms_norm_eps"], cfg["num_attention_heads"]
    x = W("model.embed_tokens.weight")[ids]
    pos = torch.cat([torch.arange(b - a, device="cuda") for a, b in spans]).double()
    angle = pos[:, None] * cfg["rope_theta"] ** (-torch.arange(HEAD // 2, device="cuda").double() * 2 / HEAD)
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def turned(y):
        u, v = y[..., :HEAD // 2], y[..., HEAD // 2:]
        return torch.cat([u * cos - v * sin, u * sin + v * cos], -1)

    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        h = _unit(x, eps) * W(p + "input_layernorm.weight")
        q, k, v = ((h @ W(p + "self_attn.%s_proj.weight" % c).T).view(len(ids), -1, HEAD) for c in "qkv")
        q = turned(_unit(q, eps) * W(p + "self_attn.q_norm.weight"))
        k = turned(_unit(k, eps) * W(p + "self_attn.k_norm.weight"))
        a = torch.cat([_attend(q[s:e], k[s:e], v[s:e], HEAD ** -0.5) for s, e in spans])
        x = x + a.reshape(len(ids), heads * HEAD) @ W(p + "self_attn.o_proj.weight").T
        h = _unit(x, eps) * W(p + "post_attention_layernorm.weight")
        z = torch.nn.functional.silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)
        x = x + z @ W(p + "mlp.down_proj.weight").T
    return (_unit(x[rows], eps) * W("model.norm.weight")) @ W("model.embed_tokens.weight").T


def _pidutar(model, ids, spans, rows):
    cfg, src = _config(model), _Weights(model)
    W = lambda name: src.get(name).double()  # noqa: E731
    eps, T = cfg["norm"]["eps"], len(ids)
    pos = torch.cat([torch.arange(b - a, device="cuda") for a, b in spans]).double()
    x = W("embed")[ids] * cfg["embedding"]["scale"]
    kept = {}

    def turned(y, dims, base):     # neighbouring elements are a pair
        angle = pos[:, None] * base ** (-torch.arange(dims // 2, device="cuda").double() * 2 / dims)
        c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
        u, v = y[..., 0::2], y[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

    def memory(h, p, m):
        H, D, Dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q = (h @ W(p + "q").T).view(T, H, D) * D ** -0.5
        k, v = (h @ W(p + "k").T).view(T, H, D), (h @ W(p + "v").T).view(T, H, Dv)
        capped = lambda z: cap * torch.tanh(z / cap)  # noqa: E731
        gi = capped(h @ W(p + "i").T + W(p + "i.b"))
        gf = torch.nn.functional.logsigmoid(capped(h @ W(p + "f").T + W(p + "f.b")))
        out = torch.empty(T, H, Dv, dtype=h.dtype, device=h.device)
        for s, e in spans:
            past = torch.ones(e - s, e - s, dtype=torch.bool, device=h.device).tril()
            for hh in range(H):
                b = gf[s:e, hh].cumsum(0)
                g = (b[:, None] - b[None, :] + gi[s:e, hh][None, :]).masked_fill(~past, -math.inf)
                top = torch.maximum(g.amax(1), b)              # (the running maximum starts at 0)
                a = torch.exp(g - top[:, None]) * (q[s:e, hh] @ k[s:e, hh].T)
                out[s:e, hh] = (a @ v[s:e, hh]) / (torch.maximum(a.sum(1).abs(), torch.exp(-top)) + 1e-6)[:, None]
        return (_unit(out, eps).reshape(T, H * Dv) * W(p + "norm") * torch.sigmoid(h @ W(p + "g").T)) @ W(p + "o").T

    def latent(h, p, m, i):
        H, D, R, Dv, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        if m.get("kv_from") is None:
            d = h @ W(p + "dkv").T
            kept[i] = (_unit(d[:, :rank], eps) * W(p + "dkv.norm"), turned(d[:, None, rank:], m["rot"]["dims"], m["rot"]["base"]))
        c, kr = kept[i if m.get("kv_from") is None else m["kv_from"]]
        q = ((_unit(h @ W(p + "dq").T, eps) * W(p + "dq.norm")) @ W(p + "uq").T).view(T, H, D + R)
        q = torch.cat([q[..., :D], turned(q[..., D:], m["rot"]["dims"], m["rot"]["base"])], -1)
        k = torch.cat([(c @ W(p + "uk").T).view(T, H, D), kr.expand(T, H, R)], -1)
        v = (c @ W(p + "uv").T).view(T, H, Dv)
        a = torch.cat([_attend(q[s:e], k[s:e], v[s:e], m["scale"], m["mask"]["size"]) for s, e in spans])
        return (a * torch.sigmoid(h @ W(p + "g").T)[:, :, None]).reshape(T, H * Dv) @ W(p + "o").T

    def experts(h, p, f):
        r = f["router"]
        top, idx = torch.topk(torch.softmax(h @ W(p + "router").T, -1), r["top"], -1)
        w = top / (top.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = torch.zeros_like(h)
        for e in range(r["experts"]):
            t, j = (idx == e).nonzero(as_tuple=True)
            z = torch.nn.functional.silu(h[t] @ W(p + "e%d.gate" % e).T) * (h[t] @ W(p + "e%d.up" % e).T)
            out.index_add_(0, t, w[t, j][:, None] * (z @ W(p + "e%d.down" % e).T))
        return out

    for i, layer in enumerate(cfg["layers"]):
        p, unit = "l%d." % i, _unit(x, eps)
        h = unit * (1 + W(p + "norm1"))
        a = memory(h, p + "mix.", layer["mixer"]) if layer["type"] == "mlstm" else latent(h, p + "mix.", layer["mixer"], i)
        f = experts(unit * (1 + W(p + "norm2")), p + "mlp.", layer["mlp"])
        x = x + cfg["residual_mult"] * (a * W(p + "ls1") + f * W(p + "ls2"))
    return (_unit(x[rows], eps) * (1 + W("final.norm"))) @ W("head").T * cfg["logit_scale"]
