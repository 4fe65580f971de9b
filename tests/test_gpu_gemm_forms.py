"""The forms of the prompt steps' product: tiles 256 or 128 wide, of one block or of a pair of blocks, each with every epilogue
where its tiles, halves and pieces end."""
import math

import pytest
import torch

BF = torch.bfloat16
FORMS = ["one", "pair", "one_128", "pair_128"]


def operands(M, N, K, seed=0):
    g = torch.Generator().manual_seed(1000 * M + N + K + seed)
    x = torch.randn(M, K, generator=g).to(BF)
    w = (torch.randn(N, K, generator=g) * 2 / math.sqrt(K)).to(BF)
    b = torch.randn(N, generator=g)
    return x, w, b, x.double() @ w.double().T + b.double()


def error32(x, w, pieces=1):
    """What 32-bit sums of K products (and of the partial tiles) may be off by: half an ulp of the running sum per addition would
    be K 2^-24 sum |x w|; the tensor cores add 16 products at a time and truncate, 2^-22 a step."""
    return (x.shape[1] / 16 + pieces + 2) * 2.0 ** -22 * (x.abs().double() @ w.abs().double().T)


SIZES = [(1, 8, 8), (129, 264, 72), (255, 131, 200), (257, 520, 1032), (300, 2560, 640), (385, 1000, 3080),
         (1100, 2304, 2056), (2048, 2560, 4096)]


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("M,N,K", SIZES)
@pytest.mark.parametrize("cut", [False, True])
def test_products(form, M, N, K, cut):
    from synaptix_b200.ops.gemm_tc import gemm_tc, gemm_tc_status, plan_stream
    x, w, b, ref = operands(M, N, K)
    bound = error32(x, w, plan_stream(M, N, K, "f32", form)[2] if cut else 1)
    out = torch.full((M, N), float("nan"), device="cuda")
    xc, wc, bc = x.cuda(), w.cuda(), b.cuda()
    gemm_tc(xc, wc, epilogue="f32", out=out, bias=bc, form=form, cut=cut)
    assert ((out.cpu().double() - ref).abs() <= bound + 1e-6).all()
    assert torch.equal(out, gemm_tc(xc, wc, epilogue="f32", bias=bc, form=form, cut=cut))
    half = gemm_tc(xc, wc, bias=bc, form=form, cut=cut).cpu().double()
    assert ((half - ref).abs() <= bound + 2.0 ** -8 * ref.abs() + 1e-6).all()
    if N % 2 == 0:
        plan = plan_stream(M, N, K, "silu_mul", form)[2] if cut else 1
        e = error32(x, w, plan) + 1e-6
        gate, up = ref[:, :N // 2], ref[:, N // 2:]
        sig = 1 / (1 + torch.exp(-gate))
        want = gate * sig * up
        # d(silu) <= 1.1 |d gate|; the fast quotient and exponential: 2^-20; the rounding to bfloat16: 2^-8
        slack = 1.1 * e[:, :N // 2] * (up.abs() + e[:, N // 2:]) + (gate * sig).abs() * e[:, N // 2:] + (2.0 ** -8 + 2.0 ** -20) * want.abs()
        got = gemm_tc(xc, wc, epilogue="silu_mul", bias=bc, form=form, cut=cut).cpu().double()
        assert ((got - want).abs() <= 1.01 * slack + 1e-6).all()
    assert gemm_tc_status() == 0


# a last round of few tiles; several rows of tiles in equal pieces; one row of tiles whose shares end in one tile and begin in the
# next (of a row's tiles at least half as many as SMs, with ragged columns)
CUT = [("one", 2048, 2560, 4096), ("pair", 2048, 2560, 4096), ("one_128", 2048, 2560, 4096), ("pair_128", 2048, 2560, 4096),
       ("pair", 1300, 3484, 3656), ("one_128", 1024, 2560, 9728), ("pair", 8191, 520, 4096), ("one", 385, 1000, 3080), ("one_128", 385, 1000, 3080),
       ("one", 33, 30000, 264), ("one", 17, 25000, 200), ("one_128", 33, 15000, 264), ("one_128", 17, 12544, 200)]


@pytest.mark.gpu
@pytest.mark.parametrize("form,M,N,K", CUT)
def test_cut_products(form, M, N, K):
    """These sizes are cut over K in these forms, on a GPU of 148 SMs."""
    from synaptix_b200.ops.gemm_tc import plan_stream
    assert plan_stream(M, N, K, "f32", form)[1] > 0 and plan_stream(M, N, K, "silu_mul", form)[1] > 0
    test_products(form, M, N, K, True)


@pytest.mark.gpu
def test_plan_is_of_the_form_that_runs():
    """Asked for no form, the plan is that of the rule's."""
    from synaptix_b200.ops.gemm_tc import plan_stream
    for M, N, K in ((512, 2560, 4096), (2048, 2560, 4096), (385, 1000, 3080), (100, 30000, 264), (64, 19456, 2560)):
        for e in (None, "silu_mul"):
            assert plan_stream(M, N, K, e) == plan_stream(M, N, K, e, None) and plan_stream(M, N, K, e) in [plan_stream(M, N, K, e, f) for f in FORMS]
    assert plan_stream(512, 2560, 4096) == plan_stream(512, 2560, 4096, None, "pair_128") != plan_stream(512, 2560, 4096, None, "one")


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("M,N,K", [(130, 264, 72), (257, 520, 1032), (2048, 2560, 4096)])
def test_residual_norm_epilogue(form, M, N, K):
    from synaptix_b200.ops.gemm_tc import gemm_tc_resid_tanh, gemm_tc_status
    x, w, b, ref = operands(M, N, K, 1)
    g = torch.Generator().manual_seed(M)
    h, gain, shift = torch.randn(M, N, generator=g), 1 + 0.2 * torch.randn(N, generator=g), torch.randn(N, generator=g)
    hc = h.cuda()
    out = gemm_tc_resid_tanh(x.cuda(), w.cuda(), b.cuda(), hc, 0.7, gain.cuda(), shift.cuda(), form=form)
    e = error32(x, w, 16) + 1e-6
    want = ref + h.double()
    assert ((hc.cpu().double() - want).abs() <= e + 2.0 ** -23 * want.abs()).all()
    normed = torch.tanh(0.7 * want) * gain.double() + shift.double()
    assert ((out.cpu().double() - normed).abs() <= 0.7 * e * gain.abs().double() + 2.0 ** -8 * normed.abs() + 1e-5).all()
    assert gemm_tc_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("form", FORMS[1:])
@pytest.mark.parametrize("M,nh,nkv,K,bias", [(129, 4, 2, 264, False), (300, 6, 1, 1224, True), (600, 16, 8, 512, False)])
def test_head_preparation_epilogue(form, M, nh, nkv, K, bias):
    """The forms give what the 256-wide tiles of one block give (compared elsewhere with plain loops): each sums K in the same
    steps, so the results may differ by the rounding to bfloat16 alone."""
    from synaptix_b200 import ops
    from synaptix_b200.ops.gemm_tc import gemm_tc_qkv, gemm_tc_status
    x, w, b, _ = operands(M, (nh + 2 * nkv) * 128, K, 2)
    i32 = lambda t: t.to(torch.int32).cuda()
    g = torch.Generator().manual_seed(M)
    wq, wk, inv = (1 + 0.3 * torch.randn(128, generator=g)).cuda(), (1 + 0.3 * torch.randn(128, generator=g)).cuda(), (torch.rand(64, generator=g) * 0.3).cuda()
    positions, pages = torch.arange(M), (M + 63) // 64
    cos, sin = ops.rope_table(i32(positions), inv)
    table = torch.randperm(pages, generator=g).view(1, -1)
    got = []
    for f in ("one", form):
        k = torch.full((pages, nkv, 64, 128), float("nan"), dtype=BF, device="cuda")
        v, q = torch.full_like(k, float("nan")), torch.full((M, nh * 128), float("nan"), dtype=BF, device="cuda")
        gemm_tc_qkv(x.cuda(), w.cuda(), q, k, v, wq, wk, cos, sin, 1e-6, i32(positions), i32(torch.zeros(M)), i32(table), nh, nkv,
                    b.cuda() if bias else None, form=f)
        got.append((q, k, v))
    for a, c in zip(*got):
        assert torch.equal(torch.isnan(a), torch.isnan(c))
        a, c = torch.nan_to_num(a.float()), torch.nan_to_num(c.float())
        # two roundings to bfloat16 lie between the products and the results (the projection's and the heads')
        assert ((a - c).abs() <= 2.0 ** -6 * (a.abs() + 4)).all()
    assert gemm_tc_status() == 0


@pytest.mark.gpu
def test_rule():
    """The rule's choice is one of the forms, for every size; and each form is somebody's choice."""
    from synaptix_b200.ops.gemm_tc import plan_stream
    chosen = set()
    for M in (130, 180, 300, 611, 1024, 2048, 8191):
        for N, K in ((6144, 2560), (2560, 4096), (2560, 9728), (1024, 3072), (4096, 1024), (12288, 2048)):
            plan = plan_stream(M, N, K, None, None)
            chosen |= {f for f in FORMS if plan_stream(M, N, K, None, f) == plan}
            assert any(plan_stream(M, N, K, None, f) == plan for f in FORMS)
    assert chosen == set(FORMS)


@pytest.mark.gpu
@pytest.mark.parametrize("bias", [False, True])
def test_head_preparation_at_16_byte_places(bias):
    """Outputs that begin 16 bytes behind a 32-byte boundary are written in 16-byte pieces: the same bits, and nothing beside."""
    from synaptix_b200 import ops
    from synaptix_b200.ops.gemm_tc import gemm_tc_qkv, gemm_tc_status
    M, nh, nkv, K = 161, 4, 2, 264
    x, w, b, _ = operands(M, (nh + 2 * nkv) * 128, K, 3)
    i32 = lambda t: t.to(torch.int32).cuda()
    cos, sin = ops.rope_table(i32(torch.arange(M)), (torch.arange(64) / 100).cuda())
    got = []
    for off in (0, 8):
        bufs = [torch.full((n + 16,), float("nan"), dtype=BF, device="cuda") for n in (M * nh * 128, 3 * nkv * 64 * 128, 3 * nkv * 64 * 128)]
        q, k, v = (t[off:off + t.numel() - 16] for t in bufs)
        gemm_tc_qkv(x.cuda(), w.cuda(), q.view(M, nh * 128), k.view(3, nkv, 64, 128), v.view(3, nkv, 64, 128), None, None, cos, sin, 1e-6,
                    i32(torch.arange(M)), i32(torch.zeros(M)), i32(torch.tensor([[2, 0, 1]])), nh, nkv, b.cuda() if bias else None)
        got.append([t.clone() for t in (q, k, v)])
        assert all(torch.isnan(t[:off].float()).all() and torch.isnan(t[off + t.numel() - 16:].float()).all() for t in bufs)
    for a, c in zip(*got):
        assert torch.equal(torch.isnan(a), torch.isnan(c)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(c))
    assert not torch.isnan(got[0][0].float()).any() and gemm_tc_status() == 0
