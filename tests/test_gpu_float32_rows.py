"""The float32 products of up to 16 rows that do what stands around them (the norm of their rows, the gated activation, the sum
into the residual stream) against 64-bit sums.  Bounds: a sum of n products in any order is off by at most (n + 2) 2^-24 times the
sum of the products' magnitudes; the gain, the factor (a sum of K squares, a root and a reciprocal of at most 4 ulp) and the sum
of a row's two parts add a few roundings of the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24
SIZES = [(2, 4), (6, 252), (130, 256), (30, 1020), (514, 1024), (1022, 2052), (96, 3072)]


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 1000003 + N * 1009 + K)
    x, w, bias, gain = (torch.randn(*s, generator=g, device="cuda") for s in ((M, K), (N, K), (N,), (K,)))
    return x * 3, w / K ** 0.5, bias, gain


def product(x, w, gain, eps):
    """The product in 64 bits and the bound on a 32-bit one."""
    K = x.shape[1]
    x64 = x.double()
    if gain is not None:
        x64 = x64 * (x64.pow(2).mean(1, keepdim=True) + eps).rsqrt() * gain.double()
    return x64 @ w.double().T, (K + 3 + (K / 2 + 8 if gain is not None else 0)) * ULP * (x64.abs() @ w.double().abs().T)


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", SIZES)
@pytest.mark.parametrize("normed", [False, True])
def test_rows(M, N, K, normed):
    from synaptix_b200 import ops
    x, w, bias, gain = operands(M, N, K)
    gain = gain if normed else None
    want, bound = product(x, w, gain, 1e-3)
    got = ops.gemm_rows_f32(x, w, gain=gain, eps=1e-3, bias=bias).double()
    assert ((got - want - bias.double()).abs() <= bound + 2 * ULP * (want.abs() + bias.double().abs())).all()
    h = torch.randn(M, N, device="cuda")
    before = h.double()
    assert ops.gemm_rows_f32(x, w, gain=gain, eps=1e-3, into=h) is h
    assert ((h.double() - before - want).abs() <= bound + 2 * ULP * (want.abs() + before.abs())).all()
    # silu(g) u: |silu'| < 1.1, |silu(g)| <= |g|; the exponential and the quotient a few ulp of the result
    g, u = want[:, :N // 2] + bias[:N // 2].double(), want[:, N // 2:] + bias[N // 2:].double()
    dg, du = (b + 2 * ULP * (z.abs() + c.double().abs()) for b, z, c in
              ((bound[:, :N // 2], g, bias[:N // 2]), (bound[:, N // 2:], u, bias[N // 2:])))
    y = ops.gemm_rows_f32(x, w, gain=gain, eps=1e-3, bias=bias, epilogue="silu_mul").double()
    z = torch.nn.functional.silu(g)
    assert ((y - z * u).abs() <= 1.1 * dg * (u.abs() + du) + z.abs() * du + 8 * ULP * (z * u).abs() + 1e-37).all()


@pytest.mark.parametrize("M", [1, 3, 12])
@pytest.mark.parametrize("N,K", [(30, 252), (30, 1020), (62, 2052)])
@pytest.mark.parametrize("eps", [1e-6, 1e-12, 0.5])
@pytest.mark.parametrize("size", [2.0 ** -140, 2.0 ** -132, 2.0 ** -100, 2.0 ** 50, 2.0 ** 125])
def test_norm_at_the_ends_of_the_range(M, N, K, eps, size):
    """Rows of next to nothing keep what a norm ahead of the product keeps of them (half of the least number, 2^-149, is lost of an
    element, of it times the gain, and of a sum, and the factor behind the sums is below 2); rows whose squares overflow are nothing, as they are there."""
    from synaptix_b200 import ops
    x, w, _, gain = operands(M, N, K)
    x, w = (x / 3).clamp(-4, 4) * size, w * K ** 0.5
    gain = gain * 4
    got = ops.gemm_rows_f32(x, w, gain=gain, eps=eps).double()
    if size == 2.0 ** 125:
        assert (got == 0).all() and (ops.gemm_generic(ops.add_rmsnorm(x, None, gain, eps, torch.float32), w) == 0).all()
        x[0, 1] = float("inf")
        got = ops.gemm_rows_f32(x, w, gain=gain, eps=eps)
        assert got[0].isnan().all() and (got[1:] == 0).all()
        return
    want, bound = product(x, w, gain, eps)
    assert ((got - want).abs() <= bound + 2.0 ** -149 * (w.double().abs() * (gain.double().abs() + 1) + 2).sum(1)).all()


def test_what_it_refuses():
    from synaptix_b200 import ops
    x, w, bias, gain = operands(4, 16, 64)
    for bad in (dict(x=x.bfloat16()), dict(w=w[:, :62].contiguous(), x=x[:, :62].contiguous()), dict(x=torch.randn(17, 64, device="cuda")),
                dict(x=x.reshape(-1)[1:193].view(3, 64)), dict(gain=gain[:63]), dict(into=torch.zeros(4, 15, device="cuda")),
                dict(into=torch.zeros(4, 16, device="cuda"), epilogue="silu_mul"), dict(epilogue="f32")):
        with pytest.raises(ops.KernelError):
            ops.gemm_rows_f32(**{"x": x, "w": w, **bad})


@pytest.mark.parametrize("M", [2, 16])
def test_dispatch_agrees_with_the_parts_one_by_one(M):
    """A norm, a stacked product and a sum through the functions that choose, against the kernels they replace."""
    from synaptix_b200 import ops
    from synaptix_b200.parts import PendingLinear, PendingNorm
    from synaptix_b200.parts.base import Runtime
    from synaptix_b200.parts.norm import RMSNorm
    x, w, _, gain = operands(M, 512, 256)
    h = torch.randn(M, 512, device="cuda")
    norm = RMSNorm("g", 512, 1e-6)
    norm.weight, norm._dtype = torch.rand(512, device="cuda") + 0.5, torch.float32
    wide = torch.randn(768, 512, device="cuda") / 20
    before = h.double()
    pn = norm.add_forward(h, PendingLinear(x, w), lazy=True)
    assert type(pn) is PendingNorm and pn.delta is None
    got = ops.linear_normed(pn, wide, epilogue="silu_mul")
    # the same in 64 bits, and how far 32-bit sums may be off: the stream, the normed rows (by the stream's error, and by the factor's,
    # which is its relative error in the norm), the products, the activation (as above)
    want_h = before + x.double() @ w.double().T
    dh = (256 + 3) * ULP * (before.abs() + x.double().abs() @ w.double().abs().T)
    assert pn.h_after() is h and ((h.double() - want_h).abs() <= dh).all()
    f = (want_h.pow(2).mean(1, keepdim=True) + 1e-6).rsqrt()
    scale, weights = f * norm.weight.double(), wide.double().abs().T
    dx = scale * (dh + want_h.abs() * (want_h.abs() * dh).sum(1, keepdim=True) / want_h.pow(2).sum(1, keepdim=True))
    z, dz = (want_h * scale) @ wide.double().T, dx @ weights + (512 * 3 / 2 + 11) * ULP * ((want_h * scale).abs() @ weights)
    g, u, dg, du = z[:, :384], z[:, 384:], dz[:, :384], dz[:, 384:]
    y = torch.nn.functional.silu(g)
    bound = 1.1 * dg * (u.abs() + du) + y.abs() * du + 8 * ULP * (y * u).abs()
    assert ((got.double() - y * u).abs() <= bound).all()
    # what 16 bits would give is outside
    low = (h * f.float() * norm.weight).bfloat16().double() @ wide.bfloat16().double().T
    assert ((torch.nn.functional.silu(low[:, :384]) * low[:, 384:] - y * u).abs() > bound).any()
