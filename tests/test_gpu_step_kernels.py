"""The kernels of single-token steps for attention over a cached latent and for experts, against 64-bit sums, at the sizes where
they change form.  A sum of n 32-bit products in any order is off by at most (n + 2) 2^-24 times the sum of their magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24
BF16 = 2.0 ** -8        # rounding to bfloat16 (8 bits of significand) moves a value by at most this share


class Step:
    """What the kernels' faces read of a step's context: single tokens, one a sequence."""

    def __init__(self, positions, maxp):
        self.positions = torch.tensor(positions, dtype=torch.int32, device="cuda")
        self.seq_of_token = torch.arange(len(positions), dtype=torch.int32, device="cuda")
        self.n_tokens, self.all_single, self.max_len = len(positions), True, maxp * 64


def latent_cache(lens, E, seed):
    """Pages [P, 1, 64, E] in bfloat16 of sequences with random rows, their tables, and the rows in 64-bit.  Every row that no
    sequence owns is NaN."""
    g = torch.Generator().manual_seed(seed)
    maxp = max((n + 63) // 64 for n in lens)
    ids = torch.randperm(len(lens) * maxp, generator=g) + 1
    pages = torch.full((len(lens) * maxp + 1, 1, 64, E), float("nan"), dtype=torch.bfloat16)
    table = torch.zeros((len(lens), maxp), dtype=torch.int32)
    rows = []
    for s, n in enumerate(lens):
        r = torch.randn(n, E, generator=g).to(torch.bfloat16)
        for p in range((n + 63) // 64):
            table[s, p] = ids[s * maxp + p]
            part = r[p * 64:(p + 1) * 64]
            pages[table[s, p], 0, :part.shape[0]] = part
        rows.append(r.double())
    return pages.cuda(), table.cuda(), rows, maxp


@pytest.mark.parametrize("H,R,Dr", [(1, 16, 0), (9, 32, 16), (16, 128, 32), (32, 320, 64), (17, 512, 64), (4, 400, 48)])
@pytest.mark.parametrize("lens,window", [([1], None), ([32, 33, 700], None), ([31, 64, 97, 700, 1100], 130)])
@pytest.mark.parametrize("parts,cluster", [(None, None), (1, 1), (3, 1), (1, 8), (2, 4), (5, 2), (1, 0)])
def test_latent_attention(H, R, Dr, lens, window, parts, cluster):
    from synaptix_b200 import ops
    from synaptix_b200.ops._lib import c_float, c_int, check, dt_code, fn, ptr, stream
    from synaptix_b200.ops.latent import WeightedLatents
    E, T, scale = R + Dr, len(lens), 0.1
    pages, table, rows, maxp = latent_cache(lens, E, H + R)
    qa = torch.randn(T, H, E, generator=torch.Generator().manual_seed(1)).cuda()
    ctx = Step([n - 1 for n in lens], maxp)
    if parts is None:
        got = ops.latent_attention(qa, pages, ctx, table, H, R, Dr, scale, window)
    else:
        out, ml = torch.full((T, H, parts, R), 7.0, device="cuda"), torch.full((T, H, parts, 2), 7.0, device="cuda")
        check(fn("latent", "sx_latent_attention")(ptr(qa), ptr(pages), ptr(ctx.positions), ptr(ctx.seq_of_token), ptr(table), c_int(maxp),
                                                  c_int(H), c_int(R), c_int(Dr), c_float(scale), c_int(window or 0), ptr(out), ptr(ml),
                                                  c_int(parts), c_int(cluster), c_int(T), c_int(dt_code(torch.bfloat16)), stream()), "latent_attention")
        got = WeightedLatents(out, ml, parts)
    got = got.merged().double().cpu()
    for s, n in enumerate(lens):
        k = rows[s][max(0, n - (window or n)):]
        z = qa[s].double().cpu() @ k.T * scale
        want = torch.softmax(z, -1) @ k[:, :R]
        # scores off by (E + 8) 2^-24 |q| |k| scale at most, weights by twice that and a few roundings, the mean by (keys + 16) more
        off = (E + 8) * ULP * float(qa[s].norm(dim=-1).max()) * float(k.norm(dim=-1).max()) * scale
        assert (got[s] - want).abs().max() <= (2 * off + (n + 32) * ULP) * float(k.abs().max())


def test_latent_attention_of_the_largest_floats():
    """Queries between the largest bfloat16 and the largest float32, against cache elements so small that the scores are ordinary."""
    from synaptix_b200 import ops
    H, R, Dr, n, scale = 3, 32, 16, 100, 0.25
    E, g = R + Dr, torch.Generator().manual_seed(0)
    pages, table, rows, maxp = latent_cache([n], E, 0)
    small = ((0.5 + torch.rand(n, generator=g)) * torch.randn(n, generator=g).sign() * 2.0 ** -124).to(torch.bfloat16)
    rows[0][:, 5] = small.double()
    for p in range(maxp):
        part = small[p * 64:(p + 1) * 64]
        pages[table[0, p], 0, :len(part), 5] = part.cuda()
    qa = torch.zeros(1, H, E)
    qa[0, :, 5] = torch.tensor([3.4e38, -3.4028234e38, 3.3961e38])
    got = ops.latent_attention(qa.cuda(), pages, Step([n - 1], maxp), table, H, R, Dr, scale, None).merged().double().cpu()[0]
    z = qa[0].double() @ rows[0].T * scale                  # one product a score
    want = torch.softmax(z, -1) @ rows[0][:, :R]
    assert ((got - want).abs() <= (4 * float(z.abs().max()) + n + 32) * ULP * float(rows[0].abs().max())).all()


@pytest.mark.parametrize("n,window", [(100, None), (100, 69), (1000, None), (1000, 650)])
@pytest.mark.parametrize("far,q", [(-float("inf"), [1.0, 0.3, 7.0]), (-2.0 ** 127, [3.3e38, 1e38, 2.9e38])])
def test_latent_scores_of_minus_infinity(n, window, far, q):
    """Keys whose scores are minus infinity, by an infinite rotated element or by overflow, have no weight."""
    from synaptix_b200 import ops
    H, R, Dr, scale = 3, 32, 16, 0.25
    pages, table, rows, maxp = latent_cache([n], R + Dr, n)
    gone = torch.zeros(n, dtype=torch.bool)
    gone[n - (window or n):][:9], gone[::3] = True, True
    k, at = rows[0], torch.where(gone, far, 0.0)
    k[:, R + 5] = 0.0
    for p in range(maxp):
        pages[table[0, p], 0, :len(at[p * 64:(p + 1) * 64]), R + 5] = at[p * 64:(p + 1) * 64].to(torch.bfloat16).cuda()
    qa = torch.randn(1, H, R + Dr, generator=torch.Generator().manual_seed(2))
    z = qa[0].double()
    qa[0, :, R + 5] = torch.tensor(q)
    got = ops.latent_attention(qa.cuda(), pages, Step([n - 1], maxp), table, H, R, Dr, scale, window).merged().double().cpu()[0]
    k = k[n - (window or n):][~gone[n - (window or n):]]
    want = torch.softmax(z @ k.T * scale, -1) @ k[:, :R]
    off = (R + Dr + 8) * ULP * float(z.norm(dim=-1).max()) * float(k.norm(dim=-1).max()) * scale
    assert (got - want).abs().max() <= (2 * off + (n + 32) * ULP) * float(k.abs().max())


@pytest.mark.parametrize("T,H,D,Dr,R", [(1, 1, 1, 0, 2), (3, 2, 16, 8, 126), (8, 3, 65, 4, 128), (9, 2, 64, 16, 320), (8, 1, 130, 0, 130)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_latent_query(T, H, D, Dr, R, dtype):
    from synaptix_b200 import ops
    g = torch.Generator().manual_seed(T + D)
    q = torch.randn(T, H * (D + Dr), generator=g).to(dtype)
    w = torch.randn(H * D, R, generator=g).to(dtype)
    got = ops.latent_query(q.cuda(), w.cuda(), H, D, Dr, R, None, 0, False, Step(list(range(T)), 1)).double().cpu()
    qd, wd = q.double().view(T, H, D + Dr), w.double().view(H, D, R)
    want = torch.einsum("thd,hdr->thr", qd[..., :D], wd)
    bound = (D + 8) * ULP * torch.einsum("thd,hdr->thr", qd[..., :D].abs(), wd.abs())
    assert ((got[..., :R] - want).abs() <= bound).all()
    assert torch.equal(got[..., R:], qd[..., D:])


@pytest.mark.parametrize("T,H,Dv,R,parts", [(1, 1, 1, 4, 1), (7, 2, 33, 128, 3), (8, 3, 128, 320, 1), (9, 2, 40, 512, 40), (5, 1, 65, 516, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gate,sink", [(None, False), ("head", True), ("elements", False)])
def test_latent_output(T, H, Dv, R, parts, dtype, gate, sink):
    from synaptix_b200 import ops
    from synaptix_b200.ops.latent import WeightedLatents
    g = torch.Generator().manual_seed(T + Dv)
    ol = torch.randn(T, H, parts, R, generator=g)
    ml = torch.stack([torch.randn(T, H, parts, generator=g), torch.rand(T, H, parts, generator=g) + 0.5], -1)
    if parts > 1:
        ml[:, :, 0, 0], ml[:, :, 0, 1], ol[:, :, 0] = float("-inf"), 0.0, 0.0          # a part without a key
    w = torch.randn(H * Dv, R, generator=g).to(dtype)
    proj = torch.randn(T, 3 + H * Dv, generator=g).to(dtype)
    sinks = torch.randn(H, generator=g) if sink else None
    got = ops.latent_output(WeightedLatents(ol.cuda(), ml.cuda(), parts), w.cuda(), H, Dv, R, proj.cuda(), -1 if gate is None else 3, dtype,
                            sinks=None if sinks is None else sinks.cuda(), gate_elements=gate == "elements").double().cpu().view(T, H, Dv)
    m, l = ml[..., 0].double(), ml[..., 1].double()
    e = torch.exp(m)
    total = (e * l).sum(-1) + (0 if sinks is None else torch.exp(sinks.double())[None])
    o = (ol.double() * e[..., None]).sum(2) / total[..., None]
    mag = (ol.double().abs() * e[..., None]).sum(2) / total[..., None]
    wd = w.double().view(H, Dv, R)
    want, mag = torch.einsum("thr,hjr->thj", o, wd), torch.einsum("thr,hjr->thj", mag, wd.abs())
    if gate is not None:
        z = torch.sigmoid(proj.double()[:, 3:])
        f = z.view(T, H, Dv) if gate == "elements" else z[:, :H, None]
        want, mag = want * f, mag * f
    bound = (R + 3 * parts + 24) * ULP * mag + (BF16 if dtype == torch.bfloat16 else ULP) * want.abs()
    assert ((got - want).abs() <= bound).all()


@pytest.mark.parametrize("T,E,top", [(1, 1, 1), (1, 16, 4), (8, 5, 2), (9, 16, 4), (16, 3, 3)])
@pytest.mark.parametrize("ff,W", [(8, 32), (24, 96), (41, 1056), (130, 544)])
@pytest.mark.parametrize("same", [False, True])
def test_experts(T, E, top, ff, W, same):
    """Gated and ungated first products and the second one; ``same``: every choice of every token names the last expert."""
    from synaptix_b200 import ops
    g = torch.Generator().manual_seed(T * 100 + ff)
    x = torch.randn(T, W, generator=g).to(torch.bfloat16)
    gate_up = (torch.randn(E, 2 * ff, W, generator=g) * W ** -0.5).to(torch.bfloat16)
    ids = torch.full((T, top), E - 1) if same else torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)])
    plan = ops.moe_sort(ids.to(torch.int32).cuda(), E)
    order = plan.order.long().cpu()
    row, ex = order // top, ids.flatten()[order]
    xd, wd = x.double()[row], gate_up.double()[ex]                                # [pairs, W], [pairs, 2 ff, W]
    z, mag = torch.einsum("pw,pfw->pf", xd, wd), torch.einsum("pw,pfw->pf", xd.abs(), wd.abs())
    off = (W + 4) * ULP * mag
    a, u = z[:, :ff], z[:, ff:]
    got = ops.moe_gate_up(x.cuda(), gate_up.cuda(), plan, top).double().cpu()
    want = a * torch.sigmoid(a) * u
    # |d silu| <= 1.1
    bound = 1.1 * off[:, :ff] * u.abs() + a.abs() * off[:, ff:] + (BF16 + 1e-6) * want.abs() + 1e-9
    assert ((got - want).abs() <= bound).all()
    with ops.gate_activation(form="relu2"):
        got = ops.moe_up(x.cuda(), gate_up.cuda(), plan, top).double().cpu()
    want = z.clamp(min=0) ** 2
    assert ((got - want).abs() <= 2 * z.abs() * off + off ** 2 + (BF16 + 1e-6) * want + 1e-9).all()
    h = torch.randn(T * top, W, generator=g).to(torch.bfloat16)
    down = (torch.randn(E, ff, W, generator=g)).to(torch.bfloat16)
    got = ops.moe_down(h.cuda(), down.cuda(), plan).double().cpu()
    hd, dd = h.double(), down.double()[ex]
    want, mag = torch.einsum("pw,pfw->pf", hd, dd), torch.einsum("pw,pfw->pf", hd.abs(), dd.abs())
    assert ((got - want).abs() <= (W + 4) * ULP * mag).all()


@pytest.mark.parametrize("T,E,top", [(1, 128, 8), (3, 257, 3), (1, 512, 1), (9, 1024, 2)])
@pytest.mark.parametrize("same", [False, True])
def test_fewer_pairs_than_experts(T, E, top, same):
    """The blocks look for the experts that were chosen, 256 of them at a time."""
    test_experts(T, E, top, 24, 96, same)


@pytest.mark.parametrize("counts", [[512], [0, 1, 127, 128, 129, 0, 300, 2], [3] * 200, [0] * 37 + [600, 0, 0]])
@pytest.mark.parametrize("ff,W", [(8, 64), (130, 200), (384, 1048)])
def test_experts_of_a_prompt(counts, ff, W):
    """From 512 rows on: tiles of 128 rows of one expert, dealt out to the blocks that walk over all of them.  The tensor cores add
    in 32-bit without rounding to nearest, so a sum is off by at most (n + 4) 2^-23 times the magnitudes."""
    from synaptix_b200 import ops
    E, g = len(counts), torch.Generator().manual_seed(ff + len(counts))
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(sum(counts), generator=g)]
    T, top = len(ids), 1
    x = torch.randn(T, W, generator=g).to(torch.bfloat16)
    gate_up = (torch.randn(E, 2 * ff, W, generator=g) * W ** -0.5).to(torch.bfloat16)
    plan = ops.moe_sort(ids.to(torch.int32).view(T, top).cuda(), E)
    order, ex = plan.order.long().cpu(), ids[plan.order.long().cpu()]
    z = torch.empty(T, 2 * ff, dtype=torch.float64)
    mag = torch.empty_like(z)
    for e in range(E):
        r = (ex == e).nonzero()[:, 0]
        z[r], mag[r] = x.double()[order[r]] @ gate_up[e].double().T, x.double()[order[r]].abs() @ gate_up[e].double().abs().T
    off = (W + 4) * 2 * ULP * mag
    a, u = z[:, :ff], z[:, ff:]
    want = a * torch.sigmoid(a) * u
    got = ops.moe_gate_up(x.cuda(), gate_up.cuda(), plan, top).double().cpu()
    assert ((got - want).abs() <= 1.1 * off[:, :ff] * u.abs() + a.abs() * off[:, ff:] + (BF16 + 1e-5) * want.abs() + 1e-9).all()
    got = ops.moe_down(x.cuda()[plan.order.long()], gate_up.cuda(), plan).double().cpu()
    assert ((got - z).abs() <= off).all()


@pytest.mark.parametrize("T,W,top", [(1, 4, 1), (3, 1024, 4), (5, 1028, 3), (2, 6, 2), (300, 260, 5)])
@pytest.mark.parametrize("y_dtype,out_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
def test_weighted_sum_of_experts(T, W, top, y_dtype, out_dtype):
    from synaptix_b200.ops.moe import moe_combine_rows
    g = torch.Generator().manual_seed(T + W)
    y = torch.randn(T * top, W, generator=g).to(y_dtype)
    place = torch.randperm(T * top, generator=g).to(torch.int32)
    w = torch.rand(T, top, generator=g)
    got = moe_combine_rows(y.cuda(), place.cuda(), w.cuda(), out_dtype).double().cpu()
    rows = y.double()[place.long()].view(T, top, W)
    want = (rows * w.double()[..., None]).sum(1)
    bound = (top + 1) * ULP * (rows.abs() * w.double()[..., None]).sum(1) + (BF16 if out_dtype == torch.bfloat16 else 0) * want.abs() + 1e-30
    assert ((got - want).abs() <= bound).all()


@pytest.mark.parametrize("dim,rot,vdim", [(96, 32, 128), (48, 16, 64), (24, 8, 32)])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("lens", [[300], [1, 64, 65, 127, 129], [256]])
def test_prompts_whose_pages_held_anything(dim, rot, vdim, window, lens, monkeypatch):
    """Whole prompts through keys and values a head, whose pages are made for the step: what the memory held before (NaN, and every
    other tensor that is made begins so, too) makes no difference to what zeros give."""
    from synaptix_b200.cache.store import KVView
    from synaptix_b200.parts import LatentAttention, RotaryPairs, Runtime
    from test_gpu_vemedra import step_ctx
    g, bf = torch.Generator().manual_seed(dim), torch.bfloat16
    W, H, rq, rk, p = 64, 3, 32, 40, "m."
    sizes = {"dq": (rq, W), "uq": (H * (dim + rot), rq), "dkv": (rk + rot, W), "uk": (H * dim, rk), "uv": (H * vdim, rk), "o": (W, H * vdim)}
    w = {p + n: (torch.randn(*s, generator=g) * s[1] ** -0.5).to(bf) for n, s in sizes.items()}
    w[p + "dq.norm"], w[p + "dkv.norm"] = torch.ones(rq), torch.ones(rk)
    part = LatentAttention(p, W, H, dim, rot, vdim, rq, rk, scale=0.3, norm_eps=1e-5, window=window, position=RotaryPairs(rot, 800.0), gated=False)
    part.bind_all(w, Runtime(torch.device("cuda:0"), bf))
    x = torch.randn(sum(lens), W, generator=g).to(bf).cuda()
    maxp = max((n + 63) // 64 for n in lens)
    table = (torch.arange(len(lens) * maxp, dtype=torch.int32) + 1).view(len(lens), maxp).cuda()
    ctx = step_ctx([0] * len(lens), lens, list(range(len(lens))), [table], bf)
    assert part._whole_prompts(ctx)
    real, got = torch.empty, []
    for value in (0.0, float("nan")):
        def filled(*args, **kw):
            t = real(*args, **kw)
            return t.fill_(value) if t.is_floating_point() else t
        monkeypatch.setattr(torch, "empty", filled)
        ctx.scratch.clear()
        pages = torch.full((len(lens) * maxp + 1, 1, 64, rk + rot), value, dtype=bf, device="cuda")
        got.append(part.forward(x, ctx, KVView(pages, None, 0, window)))
        monkeypatch.setattr(torch, "empty", real)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])
