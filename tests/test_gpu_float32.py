"""The float32 kernels for aligned sizes (streamed rows, tiles shared by a cluster, attention with eight lanes a key) against
64-bit sums, at the sizes where they change form.  Bounds: a sum of n products in any order is off by at most
(n + 2) 2^-24 times the sum of the products' magnitudes."""
import math

import pytest
import torch

from test_gpu_kernels import dev, make_paged

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 263])
@pytest.mark.parametrize("N,K", [(1, 4), (130, 252), (127, 256), (389, 1020), (96, 1024), (1024, 3072), (4099, 260), (5, 2052)])
def test_product(M, N, K):
    from synaptix_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M * 1000003 + N * 1009 + K)
    a = torch.randn(M, K, generator=g, device="cuda")
    w = torch.randn(N, K, generator=g, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda")
    want = a.double() @ w.double().T
    bound = (K + 3) * ULP * (a.double().abs() @ w.double().abs().T + bias.double().abs() + want.abs())
    assert ((ops.gemm_generic(a, w).double() - want).abs() <= bound).all()
    assert ((ops.gemm_generic(a, w, bias=bias).double() - want - bias.double()).abs() <= bound).all()


def test_product_keeps_infinities_and_nans_where_they_are():
    from synaptix_b200 import ops
    for M in (3, 40):
        a, w = torch.ones(M, 1024, device="cuda"), torch.ones(200, 1024, device="cuda")
        a[1, 1000] = float("inf")
        w[7, 3] = float("nan")
        y = ops.gemm_generic(a, w)
        assert y[:, 7].isnan().all() and torch.isinf(y[1, :7]).all() and torch.isinf(y[1, 8:]).all()
        y[:, 7], y[1] = 0, 0
        assert y.isfinite().all()


def attention(q, ks, vs, pos, sot, scale, window, softcap, sinks, chunk):
    out = torch.empty(q.shape[0], q.shape[1], vs[0].shape[2], dtype=torch.float64)
    for t in range(q.shape[0]):
        s, p = int(sot[t]), int(pos[t])
        lo = max(0 if window is None else p - window + 1, 0 if chunk is None else p // chunk * chunk, 0)
        k, v = ks[s][lo:p + 1].double(), vs[s][lo:p + 1].double()
        for h in range(q.shape[1]):
            kh = h // (q.shape[1] // k.shape[1])
            z = (k[:, kh] @ q[t, h].double()) * scale
            if softcap is not None:
                z = softcap * torch.tanh(z / softcap)
            if sinks is not None:
                z = torch.cat([z, sinks[h].double()[None]])
            out[t, h] = torch.softmax(z, 0)[:k.shape[0]] @ v[:, kh]
    return out


@pytest.mark.parametrize("nh,nkv,hd", [(2, 2, 64), (4, 2, 128), (8, 2, 64), (9, 3, 128), (16, 2, 128)])
@pytest.mark.parametrize("past,new", [([0], [1]), ([63, 64, 700], [1, 1, 1]), ([0, 130, 31], [67, 1, 3])])
@pytest.mark.parametrize("options", [{}, {"window": 70}, {"softcap": 5.0, "sinks": True}, {"chunk": 50, "window": 33}])
def test_attention(nh, nkv, hd, past, new, options):
    from synaptix_b200 import ops
    torch.manual_seed(nh + hd + len(past))
    ks = [torch.randn(p + n, nkv, hd) for p, n in zip(past, new)]
    vs = [torch.randn(p + n, nkv, hd) for p, n in zip(past, new)]
    kp, vp, bt = make_paged(ks, vs, nkv, hd, torch.float32, seed=2)
    # what lies behind a sequence's last key must not be read into the result
    for s, (p, n) in enumerate(zip(past, new)):
        if (p + n) % 64:
            page = int(bt[s, (p + n) // 64])
            kp[page, :, (p + n) % 64:], vp[page, :, (p + n) % 64:] = float("nan"), float("nan")
    T = sum(new)
    q = torch.randn(T, nh, hd)
    pos = torch.cat([torch.arange(p, p + n) for p, n in zip(past, new)]).to(torch.int32)
    sot = torch.cat([torch.full((n,), i) for i, n in enumerate(new)]).to(torch.int32)
    scale = 1 / math.sqrt(hd)
    sinks = torch.randn(nh) if options.get("sinks") else None
    kw = dict(softcap=options.get("softcap"), chunk=options.get("chunk"))
    wide = torch.full((T, nh * hd + 8), 3.0, device="cuda")
    out = ops.attn_generic(dev(q.view(T, nh * hd)), kp, vp, dev(pos), dev(sot), bt, nh, nkv, hd, scale, options.get("window"), wide,
                           sinks=None if sinks is None else dev(sinks), out_col=4, out_scale=0.5, **kw)
    want = attention(q, ks, vs, pos, sot, scale, options.get("window"), kw["softcap"], sinks, kw["chunk"]).view(T, -1) * 0.5
    # a score is off by (hd + 4) 2^-24 |q| |k| scale (the cap only shrinks it), a weight by twice that and a few roundings, and the
    # weighted mean by the weights' relative error and (keys + 8) roundings times the largest value
    off = (hd + 4) * ULP * float(q.norm(dim=-1).max()) * max(float(k.norm(dim=-1).max()) for k in ks) * scale
    bound = (2 * off + (max(p + n for p, n in zip(past, new)) + 16) * ULP) * max(float(v.abs().max()) for v in vs)
    assert (out[:, 4:4 + nh * hd].double().cpu() - want).abs().max() <= bound
    assert (out[:, :4] == 3.0).all() and (out[:, 4 + nh * hd:] == 3.0).all()


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (8, 2, 128)])
@pytest.mark.parametrize("new", [[1], [1, 1], [200]])
@pytest.mark.parametrize("far", ["first", "most"])
def test_attention_with_scores_of_minus_infinity(nh, nkv, hd, new, far):
    """Keys whose scores overflow to minus infinity have no weight: what the others give is what there would be without them."""
    from synaptix_b200 import ops
    torch.manual_seed(nh)
    n = 300
    ks, vs = [torch.randn(n, nkv, hd) for _ in new], [torch.randn(n, nkv, hd) for _ in new]
    gone = [j for j in range(n) if (j < 40 if far == "first" else j % 33 != 0)]
    q = torch.randn(sum(new), nh, hd)
    q[..., 3] = 1e20
    for k in ks:
        k[:, :, 3] = 0.0
        k[gone, :, 3] = -1e20
    kp, vp, bt = make_paged(ks, vs, nkv, hd, torch.float32, seed=2)
    pos = torch.cat([torch.arange(n - m, n) for m in new]).to(torch.int32)
    sot = torch.cat([torch.full((m,), i) for i, m in enumerate(new)]).to(torch.int32)
    scale = 1 / math.sqrt(hd)
    out = torch.empty(sum(new), nh * hd, device="cuda")
    ops.attn_generic(dev(q.view(-1, nh * hd)), kp, vp, dev(pos), dev(sot), bt, nh, nkv, hd, scale, None, out)
    kept = [j for j in range(n) if j not in gone]
    q[..., 3] = 0.0                                  # (as the kept keys' element)
    want = torch.empty(sum(new), nh, hd, dtype=torch.float64)
    for t in range(sum(new)):
        seen = [j for j in kept if j <= int(pos[t])]
        k, v = ks[int(sot[t])][seen].double(), vs[int(sot[t])][seen].double()
        for h in range(nh):
            want[t, h] = torch.softmax(k[:, h // (nh // nkv)] @ q[t, h].double() * scale, 0) @ v[:, h // (nh // nkv)]
    off = (hd + 4) * ULP * float(q.norm(dim=-1).max()) * max(float(k[kept].norm(dim=-1).max()) for k in ks) * scale
    bound = (2 * off + (n + 16) * ULP) * max(float(v.abs().max()) for v in vs)
    assert (out.double().cpu() - want.view(-1, nh * hd)).abs().max() <= bound
