"""GPU: the split float64 GEMM (digit planes on the tensor cores) against the
product in extended precision, at the edges of its 128 x 64 tiles, 32-wide K
slices and 4-slice drains, through gpk_gemm_f64.

Tolerance: one rounding of the result, 2^-53 |c|, and for each of the K terms
the rounding of both elements at 2^-56 of a scale below twice the row's
largest element plus the digit products left out: together below
2^-53 max|a_i| max|b_j|."""
import numpy as np
import pytest
import torch

from gpjax_gb300 import _lib, linalg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,kind", [
    (129, 257, 1200, "normal"), (128, 512, 64, "normal"), (1000, 65, 97, "range"),
    (63, 2200, 33, "range"), (200, 190, 1025, "positive"), (256, 256, 385, "constant"),
    (300, 130, 128, "cubed"), (127, 255, 160, "zero_row"),
])
def test_split_product(cuda_lib, m, n, k, kind):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    if kind == "range":  # rows and columns of very different size
        a *= np.exp(rng.uniform(-200, 200, (m, 1)))
        b *= np.exp(rng.uniform(-9, 9, (n, k)))
    elif kind == "positive":
        a, b = np.abs(a), np.abs(b)
    elif kind == "constant":
        a[:], b[:] = 2.0 / 3.0, -1.0 / 3.0
    elif kind == "cubed":
        a, b = a ** 9, b ** 9
    elif kind == "zero_row":
        a[5], b[7] = 0.0, 0.0
    got = linalg.matmul(torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda"),
                        transb=True).cpu().numpy()
    ref = a.astype(np.longdouble) @ b.astype(np.longdouble).T
    tol = 2.0 ** -53 * (np.abs(ref) + k * np.abs(a).max(1)[:, None] * np.abs(b).max(1)[None, :])
    assert np.all(np.abs(got - ref) <= tol)


def test_split_product_non_finite(cuda_lib):
    rng = np.random.default_rng(0)
    a, b = rng.standard_normal((300, 200)), rng.standard_normal((170, 200))
    a[3, 5], a[140, 0], b[9, 199] = np.nan, np.inf, -np.inf
    c = linalg.matmul(torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda"),
                      transb=True)
    bad = torch.zeros(300, 170, dtype=torch.bool, device="cuda")
    bad[3], bad[140], bad[:, 9] = True, True, True
    assert torch.equal(torch.isfinite(c), ~bad)


# The product's error bound for any order of the sum, K u sum_k |a_ik| |b_jk|,
# plus the rounding of the result: it knows nothing of the range along K.
# Sizes on both sides of 8e6 multiply-adds.
@pytest.mark.parametrize("size", [180, 256])
@pytest.mark.parametrize("r", [1e6, 1e12, 1e16, 2.0 ** 60])
def test_product_range_along_k(cuda_lib, size, r):
    rng = np.random.default_rng(size)
    a, b = rng.standard_normal((size, size)), rng.standard_normal((size, size))
    if r == 2.0 ** 60:  # large entries against zeros
        a[:, 0], b[:, 0] = r, 0.0
    else:  # a column of A larger by r, the matching column of B smaller by r
        a[:, 0] *= r
        b[:, 0] /= r
    got = linalg.matmul(torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda"),
                        transb=True).cpu().numpy()
    ref = a.astype(np.longdouble) @ b.astype(np.longdouble).T
    tol = 2.0 ** -53 * (np.abs(ref) + size * (np.abs(a) @ np.abs(b).T))
    assert np.all(np.abs(got - ref) <= tol)


def test_product_infinity(cuda_lib):
    """An infinity in a row gives an infinity where the sum has one."""
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((260, 300)), np.abs(rng.standard_normal((250, 300))) + 0.1
    a[3, 5], a[7, 2] = np.inf, -np.inf
    c = linalg.matmul(torch.as_tensor(a, device="cuda"), torch.as_tensor(b, device="cuda"),
                      transb=True).cpu().numpy()
    assert np.all(c[3] == np.inf) and np.all(c[7] == -np.inf)
    assert np.isfinite(np.delete(c, [3, 7], 0)).all()


# X = M B through the inverse M of L: componentwise within a few n u |M| |L| |M| |B|
# (each product's error is n u of the products of the absolute values), which
# scaled rows or columns of L leave as it is.
@pytest.mark.parametrize("axis", ["rows", "columns"])
@pytest.mark.parametrize("spread", [0, 7, 14, 20])
def test_triangular_solve_graded(cuda_lib, axis, spread):
    n, rng = 512, np.random.default_rng(spread)
    g = rng.standard_normal((n, n + 8))
    low = np.linalg.cholesky(g @ g.T / n)
    s = np.exp(rng.uniform(-spread, spread, n))
    scaled = low * (s[:, None] if axis == "rows" else s[None, :])
    b = scaled @ rng.standard_normal((n, 300))
    x = linalg.solve_triangular(torch.as_tensor(scaled, device="cuda"),
                                torch.as_tensor(b, device="cuda")).cpu().numpy()
    m = np.linalg.inv(low)  # scaling L scales M exactly as well: sizes only
    m = np.abs(m / s[None, :] if axis == "rows" else m / s[:, None])
    res = scaled.astype(np.longdouble) @ x.astype(np.longdouble) - b
    bound = np.abs(scaled) @ (m @ (np.abs(scaled) @ (m @ np.abs(b))))
    assert np.all(np.abs(res) <= 4 * n * 2.0 ** -53 * bound)


def test_triangular_solve_range_of_right_side(cuda_lib):
    b = np.ones((256, 256))
    b[0] = 1e20
    x = linalg.solve_triangular(torch.eye(256, dtype=torch.float64, device="cuda"),
                                torch.as_tensor(b, device="cuda")).cpu().numpy()
    assert np.array_equal(x, b)


def test_split_product_wait_timeout_is_reported(cuda_lib):
    """A bounded wait that runs out (the self-test's MMA warp waits 20M cycles on
    a barrier nothing arrives on) gives info = -1 and a NaN result; the context
    stays usable."""
    dev = torch.device("cuda")
    info = torch.zeros(1, dtype=torch.int32, device=dev)
    c = torch.zeros(256, 256, dtype=torch.float64, device=dev)
    ws = _lib.workspace(cuda_lib.gpk_selftest_split_wait_timeout_workspace_bytes(), dev)
    _lib.call("gpk_selftest_split_wait_timeout", c.data_ptr(), info.data_ptr(), ws.data_ptr(),
              ws.numel(), _lib.stream_ptr())
    torch.cuda.synchronize()
    assert int(info.item()) == -1
    assert torch.isnan(c).all()
    a = torch.eye(300, dtype=torch.float64, device=dev)
    assert torch.equal(linalg.matmul(a, a), a)
