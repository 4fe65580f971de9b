"""Float32 attention of prompt portions (tiles of 32 rows on the tensor cores, operands in pieces) against 64-bit sums, at the edges of
tiles, pages and groups of keys.  A sum of n products of pieces is off by less than (n + 4) 2^-24 of the products' magnitudes from
n = 64 on (16 roundings of 2^-23 within a slice of 16, one of 2^-24 a slice, 2^-23 for the pieces left out), which is the
bound on a score; a weight is off by twice that and a few roundings, and the weighted mean by the weights' relative error and
(keys + 16) roundings times the largest value."""
import ctypes
import itertools
import math

import pytest
import torch

from test_gpu_float32 import attention
from test_gpu_kernels import dev, make_paged

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24


def setup(nh, nkv, hd, past, new, seed):
    g = torch.Generator().manual_seed(seed)
    ks = [torch.randn(p + n, nkv, hd, generator=g) for p, n in zip(past, new)]
    vs = [torch.randn(p + n, nkv, hd, generator=g) for p, n in zip(past, new)]
    q = torch.randn(sum(new), nh, hd, generator=g)
    pos = torch.cat([torch.arange(p, p + n) for p, n in zip(past, new)]).to(torch.int32)
    sot = torch.cat([torch.full((n,), i) for i, n in enumerate(new)]).to(torch.int32)
    return q, ks, vs, pos, sot


def portions(past, new):
    return (ctypes.c_int * (len(new) + 1))(*([0] + list(itertools.accumulate(new)))), (ctypes.c_int * len(past))(*past)


def run(q, ks, vs, pos, sot, past, new, nkv, hd, scale, window=None, out=None, **options):
    from synaptix_b200 import ops
    kp, vp, bt = make_paged(ks, vs, nkv, hd, torch.float32, seed=2)
    for s, (p, n) in enumerate(zip(past, new)):      # what lies behind the last key and ahead of the first is never read into a result
        if (p + n) % 64:
            page = int(bt[s, (p + n) // 64])
            kp[page, :, (p + n) % 64:], vp[page, :, (p + n) % 64:] = float("nan"), float("nan")
        gone = max(0, p - window + 1) if window else 0
        if gone % 64:
            page = int(bt[s, gone // 64])
            kp[page, :, :gone % 64], vp[page, :, :gone % 64] = float("nan"), float("nan")
    sinks = options.pop("sinks", None)
    return ops.attn_generic(dev(q.view(q.shape[0], -1)), kp, vp, dev(pos), dev(sot), bt, q.shape[1], nkv, hd, scale, window, out,
                            sinks=None if sinks is None else dev(sinks), **options)


@pytest.mark.parametrize("nh,nkv,hd", [(40, 8, 128), (37, 37, 64), (48, 4, 64)])
@pytest.mark.parametrize("past,new", [([0], [64]), ([0, 0], [150, 45]), ([63, 700], [67, 30]), ([1, 64, 30, 5], [96, 1, 33, 31])])
@pytest.mark.parametrize("options", [{}, {"window": 70}, {"softcap": 5.0, "sinks": True}, {"chunk": 50, "window": 33}])
def test_prompt_attention(nh, nkv, hd, past, new, options):
    T = sum(new)
    q, ks, vs, pos, sot = setup(nh, nkv, hd, past, new, nh + hd)
    scale = 1 / math.sqrt(hd)
    sinks = torch.randn(nh) if options.get("sinks") else None
    kw = dict(softcap=options.get("softcap"), chunk=options.get("chunk"))
    out = run(q, ks, vs, pos, sot, past, new, nkv, hd, scale, options.get("window"), torch.full((T, nh * hd + 7), 3.0, device="cuda"),
              sinks=sinks, out_col=3, out_scale=0.5, **kw)
    want = attention(q, ks, vs, pos, sot, scale, options.get("window"), kw["softcap"], sinks, kw["chunk"]).view(T, -1) * 0.5
    off = (hd + 4) * ULP * float(q.norm(dim=-1).max()) * max(float(k.norm(dim=-1).max()) for k in ks) * scale
    bound = (2 * off + (max(p + n for p, n in zip(past, new)) + 16) * ULP) * max(float(v.abs().max()) for v in vs)
    assert (out[:, 3:3 + nh * hd].double().cpu() - want).abs().max() <= bound
    assert (out[:, :3] == 3.0).all() and (out[:, 3 + nh * hd:] == 3.0).all()


def test_numbers_at_the_ends_of_the_range():
    """Scores of minus infinity have no weight; an infinite value, a NaN and a score of plus infinity reach exactly the rows that see
    them; tiny values keep their 24 bits."""
    nh, nkv, hd, n = 40, 8, 64, 130
    q, ks, vs, pos, sot = setup(nh, nkv, hd, [0], [n], 5)
    q[..., 3] = 1e20
    ks[0][:, :, 3] = 0.0
    gone = [j for j in range(n) if j % 3 == 1]
    ks[0][gone, :, 3] = -1e20                        # (the products overflow, and their pieces have both signs)
    vs[0] *= 2.0 ** -120
    vs[0][42, 2, 7] = float("inf")
    ks[0][72, 4, 9] = float("nan")
    scale = 1 / math.sqrt(hd)
    out = run(q, ks, vs, pos, sot, [0], [n], nkv, hd, scale).cpu().view(n, nkv, nh // nkv, hd)
    kept = [j for j in range(n) if j not in gone]
    q[..., 3] = 0.0
    want = torch.empty(n, nh, hd, dtype=torch.float64)
    for t in range(n):
        seen = [j for j in kept if j <= t]
        k, v = ks[0][seen].double(), vs[0][seen].double()
        for h in range(nh):
            want[t, h] = torch.softmax(k[:, h // 5] @ q[t, h].double() * scale, 0) @ v[:, h // 5]
    want = want.view(n, nkv, nh // nkv, hd)
    assert out[72:, 4].isnan().all() and out[:72, 4].isfinite().all()
    assert torch.isinf(out[42:, 2, :, 7]).all() and out[:42, 2].isfinite().all()
    clean = want.clone()
    clean[72:, 4], clean[42:, 2, :, 7] = 0.0, 0.0
    got = out.double()
    got[72:, 4], got[42:, 2, :, 7] = 0.0, 0.0
    off = (hd + 4) * ULP * float(q.norm(dim=-1).max()) * float(ks[0][kept].nan_to_num().norm(dim=-1).max()) * scale
    finite = vs[0][vs[0].isfinite()].abs().max()
    assert (got - clean).abs().max() <= (2 * off + (n + 16) * ULP) * float(finite)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("case", ["scores", "columns", "weights"])
def test_small_numbers_against_large_ones(hd, case):
    """Keys below the least numbers whose pieces are whole against large queries; columns of values of different sizes; a weight
    that small against large values.  Every result within the bound of its own magnitudes, a weight's own last bit (2^-149) among them."""
    nh, nkv, n = 40, 8, 140
    q, ks, vs, pos, sot = setup(nh, nkv, hd, [0], [n], 3)
    scale = 1 / math.sqrt(hd)
    if case == "scores":
        q, ks[0], scale = q * 2.0 ** 104, ks[0] * 2.0 ** -122, scale * 2.0 ** 18
    elif case == "columns":
        vs[0] *= torch.tensor([2.0 ** -(41 * (d % 4)) for d in range(hd)])
    else:                                            # of neighbouring keys one has the weight 2^-130 and values of 2^106
        q[..., 3], ks[0][:, :, 3] = 1.0, 0.0
        ks[0][1::2, :, 3] = -90 / scale
        vs[0][1::2] *= 2.0 ** 106
        vs[0][::2] *= 2.0 ** -40
    out = run(q, ks, vs, pos, sot, [0], [n], nkv, hd, scale).cpu().view(n, nh, hd).double()
    for h in range(nh):
        k, v = ks[0][:, h // 5].double(), vs[0][:, h // 5].double()
        z = (q[:, h].double() @ k.T) * scale
        w = torch.softmax(z.masked_fill(torch.ones(n, n, dtype=torch.bool).triu(1), -math.inf), -1)
        off = (hd + 4) * ULP * float((q[:, h].double().abs() @ k.abs().T).max()) * scale
        bound = (2 * off + (n + 16) * ULP) * (w @ v.abs()) + 2.0 ** -149 * v.abs().sum(0) + n * 2.0 ** -149
        assert ((out[:, h] - w @ v).abs() <= bound).all(), h


def test_time_of_rows_that_are_not_finite():
    """A key whose scores overflow, seen by all rows behind it: the rows once in pieces and once in 32 bits, 16 keys at a time."""
    from synaptix_b200 import ops
    nh, nkv, hd, n = 16, 8, 128, 1024
    q, ks, vs, pos, sot = setup(nh, nkv, hd, [0], [n], 7)
    ks[0][:, :, 0] = 0.0
    kp, vp, bt = make_paged(ks, vs, nkv, hd, torch.float32, seed=2)
    big = q.clone()
    big[..., 0] = 1e20
    far = kp.clone()
    far[int(bt[0, 0]), :, 7, 0] = -1e20

    def ms(q, k):
        q, p, s = dev(q.view(n, -1)), dev(pos), dev(sot)
        one = lambda: ops.attn_generic(q, k, vp, p, s, bt, nh, nkv, hd, hd ** -0.5)  # noqa: E731
        one()
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(5):
            y = one()
        end.record()
        end.synchronize()
        assert y.isfinite().all()
        return start.elapsed_time(end)
    assert ms(big, far) <= 10 * ms(q, kp)


# sequences of fewer than 6, 17 or 33 tokens (left to the other kernel) and of so many: ahead of others, behind them and between, next
# to a tile's edge and across it
@pytest.mark.parametrize("past,new", [([300, 0], [1, 70]), ([0, 90, 64], [62, 5, 6]), ([0, 9, 0, 70, 3], [30, 4, 90, 5, 1]), ([5, 0, 128, 0], [6, 57, 1, 65]),
                                      ([0, 100, 20, 0], [64, 6, 7, 90]), ([0, 1500, 0], [81, 16, 90]), ([0, 0, 2000], [60, 100, 32])])
@pytest.mark.parametrize("known", [False, True])
@pytest.mark.parametrize("nh,nkv,hd", [(40, 8, 128), (37, 37, 64)])
def test_steps_of_long_and_short_portions(nh, nkv, hd, known, past, new):
    q, ks, vs, pos, sot = setup(nh, nkv, hd, past, new, sum(new))
    out = run(q, ks, vs, pos, sot, past, new, nkv, hd, hd ** -0.5, out=torch.full((sum(new), nh * hd), 3.0, device="cuda"),
              portions=portions(past, new) if known else None)
    want = attention(q, ks, vs, pos, sot, hd ** -0.5, None, None, None, None).view(sum(new), -1)
    off = (hd + 4) * ULP * float(q.norm(dim=-1).max()) * max(float(k.norm(dim=-1).max()) for k in ks) * hd ** -0.5
    bound = (2 * off + (max(p + n for p, n in zip(past, new)) + 16) * ULP) * max(float(v.abs().max()) for v in vs)
    assert (out.double().cpu() - want).abs().max() <= bound


@pytest.mark.parametrize("past,new,kernels", [([0, 0], [70, 90], 1), ([0, 50], [90, 1], 2), ([9, 50], [1, 1], 1), ([0], [90], 1)])
def test_kernels_of_a_step_are_counted(past, new, kernels):
    from synaptix_b200 import ops

    class Counter:
        kernel_launches = 0
    q, ks, vs, pos, sot = setup(40, 8, 64, past, new, 2)
    run(q, ks, vs, pos, sot, past, new, 8, 64, 0.125, portions=portions(past, new))        # (loaded)
    ops.set_launch_counter(Counter)
    try:
        run(q, ks, vs, pos, sot, past, new, 8, 64, 0.125, portions=portions(past, new))
    finally:
        ops.set_launch_counter(None)
    assert Counter.kernel_launches == kernels


@pytest.mark.parametrize("known", [False, True])
def test_time_of_steps_of_long_and_short_portions(known):
    """A prompt of 500 tokens with twenty single tokens behind 1,000 others, or eight behind 6,000, costs about what either costs alone."""
    from synaptix_b200 import ops
    nh, nkv, hd = 16, 8, 128

    def ms(past, new):
        q, ks, vs, pos, sot = setup(nh, nkv, hd, past, new, 1)
        kp, vp, bt = make_paged(ks, vs, nkv, hd, torch.float32, seed=2)
        args = dev(q.view(sum(new), -1)), kp, vp, dev(pos), dev(sot), bt, nh, nkv, hd, hd ** -0.5
        more = {"portions": portions(past, new)} if known else {}
        ops.attn_generic(*args, **more)
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(20):
            ops.attn_generic(*args, **more)
        end.record()
        end.synchronize()
        return start.elapsed_time(end)
    assert ms([0] + [1000] * 20, [500] + [1] * 20) <= 2.5 * (ms([0], [500]) + ms([1000] * 20, [1] * 20))
    if known:
        assert ms([0, 6000], [500, 8]) <= 2.0 * (ms([0], [500]) + ms([6000], [8]))
