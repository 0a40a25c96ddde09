"""GPU: FP64 products on the int8 tensor cores (stk_gemm_f64_i8) against long-double sums.

Tolerance.  A row is rounded to 2^-56 of its scale 2^e <= 2 max|x| at each value, and the digit
products i + j >= 8 are dropped, about sqrt(5 K) 73^2 256^4 of 2^110 (a scaled product of the largest
values): with normal values, max|x| < 5 rms, the whole is below 2^-55 |a||b|.  C's elements are
|a||b| / sqrt(K) on average, and the result is rounded to FP64 (2^-53 in all, with the two
conversions): relative L2 below 2^-53 (1 + sqrt(K) / 4)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch


def product(torch, A, B, C=None):
    """C (+)= A B^T through the C ABI; returns M x N."""
    from stkfmm_b200 import lib
    M, K = A.shape
    N = B.shape[0]
    a, b = torch.as_tensor(A, device="cuda"), torch.as_tensor(B, device="cuda")
    out = torch.as_tensor(np.zeros((N, M)) if C is None else np.ascontiguousarray(C.T), device="cuda")
    rc = lib().stk_gemm_f64_i8(M, N, K, a.data_ptr(), K, b.data_ptr(), K, out.data_ptr(), M, 0 if C is None else 1,
                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0, rc
    torch.cuda.synchronize()
    return out.cpu().numpy().T


# one block; ragged M, N, K; several K blocks; more tiles than one CTA's turn; two K segments
@pytest.mark.parametrize("M,N,K", [(128, 128, 32), (1, 1, 1), (129, 257, 33), (37, 5, 640), (300, 200, 100),
                                   (3000, 2000, 64), (130, 70, 16384), (130, 70, 16385), (64, 40, 33000)])
def test_matches_long_double(torch_cuda, M, N, K):
    rng = np.random.default_rng(M + 7 * N + 13 * K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(N, K))
    A *= np.exp2(rng.integers(-40, 40, size=(M, 1)))  # every row its own scale
    C0 = rng.normal(size=(M, N)) * np.abs(A).max(1, keepdims=True)
    got = product(torch_cuda, A, B)
    sub = slice(0, M, max(1, M // 150)), slice(0, N, max(1, N // 150))
    ref = A[sub[0]].astype(np.longdouble) @ B[sub[1]].astype(np.longdouble).T
    rows = np.abs(A[sub[0]]).max(1, keepdims=True)
    err = np.linalg.norm(((got[sub] - ref) / rows).astype(float)) / np.linalg.norm((ref / rows).astype(float))
    assert err < 2.0 ** -53 * (1 + np.sqrt(K) / 4), err
    # += adds the same product, rounded once more
    both = product(torch_cuda, A, B, C0)
    np.testing.assert_allclose(both, C0 + got, rtol=0, atol=float(2.0 ** -51 * np.abs(C0 + got).max()))
    np.testing.assert_array_equal(got, product(torch_cuda, A, B))  # integer sums: the same bits again


def test_digits_at_the_ends_of_their_range(torch_cuda):
    """Values whose digits are all extreme (the int32 sums' bound), powers of two, exact integers, and
    the smallest and largest magnitudes."""
    K = 16384
    for top in (np.nextafter(1.0, 0.0), 1.0, 127 / 128, np.nextafter(127 / 128, 0.0), 0.5):
        big = np.full((2, K), top)
        big[1] *= -1
        got = product(torch_cuda, big, big)
        assert np.allclose(got, K * top * top * np.array([[1, -1], [-1, 1]]), rtol=2.0 ** -50, atol=0), top
    rng = np.random.default_rng(3)
    ints = rng.integers(-2 ** 20, 2 ** 20, size=(140, 200)).astype(float)
    np.testing.assert_array_equal(product(torch_cuda, ints, ints), ints @ ints.T)
    for s in (2.0 ** -1000, 2.0 ** -1060, 2.0 ** 1000):
        x = ints[:5, :64] * s
        np.testing.assert_allclose(product(torch_cuda, x, ints[:5, :64] / 2 ** 20), (x / 2.0 ** 20) @ ints[:5, :64].T,
                                   rtol=1e-14, atol=0 if s > 1e-305 else 2.0 ** -1000)


def test_zero_and_non_finite_rows(torch_cuda):
    rng = np.random.default_rng(4)
    A, B = rng.normal(size=(6, 70)), rng.normal(size=(9, 70))
    A[1] = 0.0
    A[2, 3], A[3, 69], B[4, 0] = np.inf, np.nan, -np.inf
    got = product(torch_cuda, A, B)
    bad = np.zeros((6, 9), bool)
    bad[2:4] = bad[:, 4] = True
    assert not np.isfinite(got[bad]).any()
    np.testing.assert_allclose(got[~bad], (A @ B.T)[~bad], rtol=0, atol=1e-13)
    assert (got[1, ~bad[1]] == 0).all()


def test_rows_at_the_ends_of_the_double_range(torch_cuda):
    """Rows from 2^-1060 to 2^1000, every pair of them in one tile: whole numbers below 2^20, so that
    sums of 64 products are exact and the result is one rounding of them (none but where it is
    subnormal: one unit of the smallest there, for a rounding before the last)."""
    rng = np.random.default_rng(5)
    exps = np.array([-1060, -1022, -1000, -988, -700, -536, -465, -300, 0, 300, 465, 536, 700, 970, 1000])
    ia, ib = (rng.integers(-2 ** 20, 2 ** 20, size=(3 * len(exps), 64)).astype(float) for _ in range(2))
    ea, eb = np.repeat(exps, 3), np.tile(exps, 3)
    with np.errstate(over="ignore"):
        ref = np.ldexp(ia @ ib.T, ea[:, None] + eb[None, :])
    got = product(torch_cuda, np.ldexp(ia, ea[:, None]), np.ldexp(ib, eb[:, None]))
    normal = ~(np.abs(ref) < 2.0 ** -1022)
    np.testing.assert_array_equal(got[normal], ref[normal])
    assert np.abs(got[~normal] - ref[~normal]).max() <= 2.0 ** -1074


@pytest.mark.parametrize("beta", [0, 1])
def test_empty_sum(torch_cuda, beta):
    """K = 0: zeros (beta 0) or C as it was, and nothing beyond its M rows."""
    from stkfmm_b200 import lib
    C = np.arange(1.0, 36.0).reshape(5, 7)  # 5 columns of M = 4 within ldc = 7
    out = torch_cuda.as_tensor(C, device="cuda")
    a = torch_cuda.zeros(8, dtype=torch_cuda.float64, device="cuda")
    rc = lib().stk_gemm_f64_i8(4, 5, 0, a.data_ptr(), 0, a.data_ptr(), 0, out.data_ptr(), 7, beta,
                               torch_cuda.cuda.current_stream().cuda_stream)
    assert rc == 0
    want = C.copy()
    want[:, :4] *= beta
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("K", [1, 40, 3584])
def test_error_bound_holds_for_graded_rows(torch_cuda, K):
    """The stated bound, 4.2 K 2^-56 max|a| max|b| + 2^-52 |c|, where rows of A fall by nine decades and
    those of B rise by as many (each product as large as any other), where only A is graded and B misses
    its largest value, and on plain values."""
    rng = np.random.default_rng(K)
    g = np.logspace(0, -9, K)
    rows = lambda: rng.uniform(0.5, 1.0, size=(20, K)) * rng.choice([-1.0, 1.0], size=(20, K))
    A = np.concatenate([rows() * g, np.abs(rows()) * g, rows()])
    miss = rows()
    miss[:, 0] = 0.0
    B = np.concatenate([rows() / g, miss, np.abs(rows()) / g, rows()])
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    bound = 4.2 * K * 2.0 ** -56 * np.abs(A).max(1)[:, None] * np.abs(B).max(1) + 2.0 ** -52 * np.abs(ref)
    assert (np.abs(product(torch_cuda, A, B) - ref) <= bound).all()


def test_m2l_shape(torch_cuda):
    """A product of the triply periodic RPY case's M2L (rank 636, 32,768 nodes, 3,584 stacked ranks) on
    normal operands, 12 columns of it against long-double sums (also the profiled launch)."""
    from stkfmm_b200 import lib
    torch = torch_cuda
    M, N, K = 636, 32768, 3584
    gen = torch.Generator(device="cuda").manual_seed(11)
    A = torch.randn((M, K), dtype=torch.float64, device="cuda", generator=gen)
    B = torch.randn((N, K), dtype=torch.float64, device="cuda", generator=gen)
    C = torch.empty((N, M), dtype=torch.float64, device="cuda")
    rc = lib().stk_gemm_f64_i8(M, N, K, A.data_ptr(), K, B.data_ptr(), K, C.data_ptr(), M, 0,
                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    cols = np.linspace(0, N - 1, 12).astype(int)
    ref = B[cols].cpu().numpy().astype(np.longdouble) @ A.cpu().numpy().astype(np.longdouble).T
    err = np.linalg.norm((C[cols].cpu().numpy() - ref).astype(float)) / np.linalg.norm(ref.astype(float))
    assert err < 2.0 ** -53 * (1 + np.sqrt(K) / 4), err
