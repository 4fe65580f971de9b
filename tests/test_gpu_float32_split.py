"""Float32 products of more than 16 rows, whose operands go to the tensor cores in pieces, over the range of 32-bit numbers against
64-bit sums: numbers near the least and near the largest, on either side and against each other.  Bounds: a product of pieces is off
by 2^-23 of the whole at most (three products of pieces are left out, each below 2^-24 / 2^8 of it, and two roundings), a sum of 16 in the tensor cores by 16 * 2^-23 of its magnitudes (whatever way they round),
and the K / 16 sums of slices by 2^-24 each: below (K + 3) 2^-24, what the same sum of whole products is given, from K = 64 on."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ULP = 2.0 ** -24


def operands(M, N, K, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + M * 1009 + N * 17 + K)
    return torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")


# tiles of 32 and of 64 rows with their remainders, one block a tile and clusters of all sizes, slices of 16 with remainders
@pytest.mark.parametrize("M,N,K", [(17, 389, 64), (32, 128, 1020), (33, 129, 84), (64, 4100, 260), (65, 7, 4096), (263, 1024, 3072),
                                   (700, 2600, 132)])
@pytest.mark.parametrize("up,down", [(0, 0), (-60, 0), (0, -118), (-70, -30), (60, 55), (100, -100), (60, -120), (110, -125), (100, -126), (100, -140),
                                     (-140, 100), (0, -140), (-70, -70)])
def test_products_over_the_range(M, N, K, up, down):
    from synaptix_b200 import ops
    a, w = operands(M, N, K)
    a, w = a * 2.0 ** up, w * 2.0 ** down
    a[:, ::5] *= 2.0 ** -20                          # numbers of different sizes in one sum
    got, want = ops.gemm_generic(a, w).double(), a.double() @ w.double().T
    bound = (K + 3) * ULP * (a.double().abs() @ w.double().abs().T) + K * 2.0 ** -149
    assert ((got - want).abs() <= bound).all()


def test_error_is_no_larger_than_a_chain_of_multiply_adds():
    """263 rows of 1,024 x 3,072: 2-norm of the error against 64 bits, and that of one 32-bit sum an output in the order of K."""
    from synaptix_b200 import ops
    a, w = operands(263, 1024, 3072, 5)
    want = a.double() @ w.double().T
    chain = torch.zeros(263, 1024, device="cuda")
    for k in range(3072):
        chain = torch.addcmul(chain, a[:, k, None], w[None, :, k])
    assert (ops.gemm_generic(a, w).double() - want).norm() <= (chain.double() - want).norm()


@pytest.mark.parametrize("M", [17, 40, 80])
def test_numbers_at_the_ends_of_the_range(M):
    from synaptix_b200 import ops
    a, w = torch.zeros(M, 1024, device="cuda"), torch.zeros(200, 1024, device="cuda")
    a[0, 5] = torch.finfo(torch.float32).max        # rounds up to an infinite bfloat16
    a[1, 6], a[2, 7], a[3, 8], a[4, 9] = float("-inf"), float("nan"), 2.0 ** -126 * 1.5, 2.0 ** 127
    w[:, 5:10] = 0.5
    w[9, 9], w[11, 6] = 4.0, 0.0
    y = ops.gemm_generic(a, w)
    assert (y[0] == torch.finfo(torch.float32).max / 2).all()
    assert torch.isinf(y[1, :11]).all() and (y[1, :11] < 0).all() and y[1, 11].isnan() and y[2].isnan().all()
    assert (y[4, :9] == 2.0 ** 126).all() and y[4, 9] == float("inf") and (y[5:] == 0).all()
    assert torch.allclose(y[3], torch.full_like(y[3], 2.0 ** -127 * 1.5), rtol=0, atol=2.0 ** -149)


@pytest.mark.parametrize("M,N,K", [(32, 260, 1024), (300, 1024, 3072), (2048, 2560, 260)])
def test_sums_that_are_not_finite(M, N, K):
    """Rows and columns with a NaN, an infinity or numbers too large for pieces, also where K is shared by a cluster: they are what
    the numbers give, and the other sums are what they are without them, bit by bit."""
    from synaptix_b200 import ops
    a, w = operands(M, N, K, 9)
    plain = ops.gemm_generic(a, w)
    a[3, K - 1], a[17, 5], w[130, 0] = float("nan"), float("inf"), float("-inf")
    a[M - 2] = a[M - 2].abs() * 2.0 ** 115
    w[N - 1] = w[N - 1].abs() * 2.0 ** 113           # (row M - 2 with column N - 1 overflows, in any order of the sum)
    got, want = ops.gemm_generic(a, w), a.double() @ w.double().T
    want = want.float().double()                     # (to infinity where it overflows)
    other = want.isfinite()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and (got[got.isinf()] == want[want.isinf()]).all()
    bound = (K + 3) * ULP * (a.double().abs() @ w.double().abs().T)
    assert ((got.double() - want).abs() <= bound)[other].all()
    kept = torch.ones(M, N, dtype=torch.bool, device="cuda")
    kept[[3, 17, M - 2]], kept[:, [130, N - 1]] = False, False
    assert torch.equal(got[kept], plain[kept])


def test_time_of_sums_that_are_not_finite():
    """Half of all sums NaN: the tiles once in pieces and once in whole numbers, not a multiple of that."""
    from synaptix_b200 import ops
    a, w = operands(1024, 2048, 2048)
    b = a.clone()
    b[::2, 7] = float("nan")

    def ms(x):
        ops.gemm_generic(x, w)
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(5):
            ops.gemm_generic(x, w)
        end.record()
        end.synchronize()
        return start.elapsed_time(end)
    assert ms(b) <= 8 * ms(a)
