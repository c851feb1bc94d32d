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

from gpjax_gb300 import linalg

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
