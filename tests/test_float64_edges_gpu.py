"""GPU: the float64 form where its kernels and their dispatch change shape --
the 64-wide fixed-point Cholesky blocks and their panels, the tile edges of the
gradient reduction and of the cross-covariance cotangents, the column blocks
of the collapsed bound, and the range of the integer exp and sqrt."""
import numpy as np
import pytest
import torch

import gpjax_gb300 as gpx
from gpjax_gb300 import linalg
from oracle import gp_oracle as O
from tests._gpu_helpers import KINDS, grads_of, make_posterior, to_cuda_params
from tests.test_sgpr_gpu import _oracle as elbo_oracle, _run as elbo_run

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


# |A - L L^T| <= (n + 1) u |L| |L|^T <= (n + 1) u sqrt(a_ii a_jj) for any order
# of a float64 Cholesky's sums; the fixed-point block rounds an entry at 2^-60
# of a scale below 2 sqrt(a_ii), well inside u.  A factor of 4 covers the panel
# and update products' own scales (powers of two above a row's largest entry).
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 200, 513, 900])
@pytest.mark.parametrize("spread", [0.0, 40.0])
def test_cholesky_blocks(cuda_lib, n, spread):
    rng = np.random.default_rng(n)
    b = rng.standard_normal((n, n + 3))
    s = np.exp(rng.uniform(-spread, spread, n))
    a = (b @ b.T + 0.01 * np.eye(n)) * s[:, None] * s[None, :]
    a = np.tril(a) + np.tril(a, -1).T
    low = linalg.lower_cholesky(linalg.Dense(torch.as_tensor(a, device="cuda"))).to_dense()
    low = np.tril(low.cpu().numpy()).astype(np.longdouble)
    size = np.sqrt(np.diag(a))
    err = np.abs((low @ low.T - a) / (size[:, None] * size[None, :]).astype(np.longdouble))
    assert float(err.max()) <= 4 * (n + 1) * U, float(err.max()) / U


# Indefinite matrices whose last pivot, 1 - (n - 1) c^2, lies far below the range
# [-8, 8) of a fixed-point entry: in all of them the leading minors before the
# last are positive, so the order that fails is n.
@pytest.mark.parametrize("n", [64, 65, 200])
@pytest.mark.parametrize("c", [0.3, 0.5, 0.7, 0.75, 0.8, 0.85, 0.9, 0.95, 1.0])
def test_cholesky_indefinite_arrow(cuda_lib, n, c):
    a = np.eye(n)
    a[-1, :-1] = a[:-1, -1] = c
    low, info = linalg.cholesky_dense(torch.as_tensor(a, device="cuda"))
    assert int(info.item()) == n
    assert np.isnan(low[-1, -1].item())


# An entry of the factor is good relative to itself, however small beside its
# row's diagonal: here each one is a_ij / l_jj but for products below 1e-25 of it
# (two roundings, one of the reciprocal).
@pytest.mark.parametrize("n", [2, 64, 130, 200])
def test_cholesky_small_entries(cuda_lib, n):
    rng = np.random.default_rng(n)
    d = np.exp(rng.uniform(-3, 3, n))
    a = np.tril(rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-31, -30, (n, n)), -1)
    a = a + np.diag(d)
    low, info = linalg.cholesky_dense(torch.as_tensor(a + np.tril(a, -1).T, device="cuda"))
    ref = np.tril(a, -1) / np.sqrt(d)[None, :] + np.diag(np.sqrt(d))
    assert int(info.item()) == 0
    assert np.all(np.abs(np.tril(low.cpu().numpy()) - ref) <= 4 * U * np.abs(ref))


# The columns before the order that fails hold the factor, all entries of the
# lower triangle from there on are NaN.
@pytest.mark.parametrize("n,k", [(60, 7), (200, 70), (200, 128), (130, 129)])
def test_cholesky_failed_factor(cuda_lib, n, k):
    rng = np.random.default_rng(k)
    g = rng.standard_normal((n, n + 5))
    a = g @ g.T
    ref = np.linalg.cholesky(a)
    a[k, k] = -1.0
    low, info = linalg.cholesky_dense(torch.as_tensor(a, device="cuda"))
    low = np.tril(low.cpu().numpy())
    assert int(info.item()) == k + 1
    assert np.abs(low[:k, :k] - ref[:k, :k]).max() <= 1e-10 * np.abs(ref).max()
    assert np.isnan(low[k:, k:][np.tril_indices(n - k)]).all()


# The same through the marginal likelihood: 63 points at distance r from the
# last (kernel value c there), sqrt(2) r or 2 r from one another (c^2, c^4), and
# a negative jitter that leaves D on Sigma's diagonal.  The leading minors are
# positive (D > 2 c^2), the last pivot is far below -D.
@pytest.mark.parametrize("D", [0.035, 0.04, 0.05, 0.06])
@pytest.mark.parametrize("ratio", [17.0, 20.0, 25.0, 30.0])
def test_mll_indefinite_sigma(cuda_lib, D, ratio):
    r = np.sqrt(np.log(ratio / D))
    x = np.concatenate([r * np.eye(32), -r * np.eye(32)[:31], np.zeros((1, 32))])
    sigma = O.gram(0, x, np.ones(32), 1.0)
    sigma[np.diag_indices(64)] = D
    assert np.linalg.eigvalsh(sigma[:63, :63])[0] > 0.5 * D
    assert sigma[63, :63] @ np.linalg.solve(sigma[:63, :63], sigma[63, :63]) > 8 * D
    post = to_cuda_params(make_posterior(0, np.ones(32), 1.0, 1e-3, 0.0, jitter=D - 1.0 - 1e-6))
    val = gpx.objectives.conjugate_mll(
        post, gpx.Dataset(X=x, y=np.sin(np.arange(64.0))[:, None]), precision="fp64")
    assert np.isnan(val.item()) and int(val.grad_fn.info.item()) == 64


# Same bounds as the float64 parity test of the marginal likelihood, at the
# sizes on either side of each tile edge of the gradient reduction.
@pytest.mark.parametrize("kind,n,d", [(0, 128, 3), (1, 130, 5), (2, 384, 2), (0, 385, 9),
                                      (1, 1536, 4), (2, 1537, 3)])
def test_mll_tile_edges(cuda_lib, kind, n, d):
    rng = np.random.default_rng(n + d)
    x = rng.uniform(-2, 2, size=(n, d))
    y = np.sin(x).sum(1, keepdims=True) + 0.1 * rng.standard_normal((n, 1))
    ls = np.exp(rng.uniform(np.log(0.5), np.log(2.0), d))
    post = to_cuda_params(make_posterior(kind, ls, 1.2, 0.3, 0.1))
    val = gpx.objectives.conjugate_mll(post, gpx.Dataset(X=x, y=y), precision="fp64")
    val.backward()
    got = grads_of(post)
    ref = O.conjugate_mll(kind, x, y, ls, 1.2, 0.3, 0.1)
    _, g = O.conjugate_mll_torch(kind, x, y, ls, 1.2, 0.3, 0.1, lu=False)
    gref = np.concatenate([np.atleast_1d(g["lengthscale"]),
                           [g["variance"], g["obs_stddev"], g["constant"]]])
    assert abs(float(val) - ref) <= 1e-10 * max(1.0, abs(ref))
    assert np.allclose(got, gref, rtol=1e-7, atol=1e-8 * max(1.0, np.abs(gref).max()))


# Odd row counts below a panel that writes digit planes: the last warp of the
# last block then holds one row, whose exponent its lanes read before one of
# them replaces it.  Bounds and repeatability as above; equal bits each time.
@pytest.mark.parametrize("n", [129, 195, 323, 577])
def test_mll_odd_panels(cuda_lib, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-2, 2, size=(n, 2))
    y = np.sin(x).sum(1, keepdims=True) + 0.1 * rng.standard_normal((n, 1))
    ls = np.array([0.7, 1.3])
    runs = []
    for _ in range(4):
        post = to_cuda_params(make_posterior(1, ls, 1.2, 0.3, 0.1))
        val = gpx.objectives.conjugate_mll(post, gpx.Dataset(X=x, y=y), precision="fp64")
        val.backward()
        runs.append(np.concatenate([[val.item()], grads_of(post)]))
    assert all(np.array_equal(runs[0], r) for r in runs[1:])
    ref = O.conjugate_mll(1, x, y, ls, 1.2, 0.3, 0.1)
    assert abs(runs[0][0] - ref) <= 1e-10 * max(1.0, abs(ref))


# A noise whose square is infinite: Sigma's diagonal is infinite, its inverse
# zero, the predictive variance the prior's, and no order fails.
@pytest.mark.parametrize("n", [30, 100, 400])
def test_infinite_noise(cuda_lib, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-2, 2, size=(n, 2))
    post = to_cuda_params(make_posterior(0, np.ones(2), 1.0, 1e200, 0.1))
    dist = post.predict(torch.as_tensor(x[:5], device="cuda"),
                        gpx.Dataset(X=x, y=np.sin(x[:, :1])), precision="fp64")
    assert int(dist.info.item()) == 0
    assert np.allclose(dist.variance.cpu().numpy(), 1.0 + 1e-6, rtol=1e-15, atol=0)


# 16-, 32- and 64-wide tiles with ragged last tiles, and d on both sides of the
# 64-wide form's bound.  Sums of at most n terms of mixed sign, each with a few
# roundings and an exp whose argument is below 100: 1e-12 of the sum of the
# terms' sizes is 4e3 times u n at n = 2.
@pytest.mark.parametrize("kind,n,m,d", [(0, 15, 17, 3), (1, 1, 40, 1), (2, 385, 417, 5),
                                        (0, 1121, 1217, 16), (1, 1121, 1217, 17)])
def test_cross_covariance_cotangent_tiles(cuda_lib, kind, n, m, d):
    rng = np.random.default_rng(n + m + d)
    x, z = rng.uniform(-2, 2, (n, d)), rng.uniform(-2, 2, (m, d))
    G, ls = rng.standard_normal((n, m)), np.exp(rng.uniform(0.0, 1.0, d))
    k = KINDS[kind](lengthscale=ls, variance=1.3)
    for p in (k.lengthscale, k.variance):
        p.to("cuda").requires_grad_(True)
    xt, zt = (torch.as_tensor(v, device="cuda").requires_grad_(True) for v in (x, z))
    K = k.cross_covariance(xt, zt)
    got = torch.autograd.grad(K, [k.lengthscale.value, k.variance.value, xt, zt],
                              torch.as_tensor(G, device="cuda"))
    xr, zr, lr, vr = (torch.as_tensor(v, dtype=torch.float64).requires_grad_(True)
                      for v in (x, z, ls, 1.3))
    sq = (((xr[:, None] - zr[None]) / lr) ** 2).sum(-1)
    t = torch.sqrt(sq)
    Kr = vr * [torch.exp(-0.5 * sq), (1 + 3 ** 0.5 * t) * torch.exp(-3 ** 0.5 * t),
               (1 + 5 ** 0.5 * t + 5.0 / 3.0 * sq) * torch.exp(-5 ** 0.5 * t)][kind]
    ref = torch.autograd.grad(Kr, [lr, vr, xr, zr], torch.as_tensor(G))
    assert torch.allclose(K.detach().cpu(), Kr.detach(), rtol=1e-12, atol=0)
    # sizes of the terms: |G| times bounds of |dK/d.|, at most 4 K-sized factors
    for g, r, terms in zip(got, ref, (n * m, n * m, m, n)):
        assert float((g.cpu() - r).abs().max()) <= 1e-12 * 4 * 1.3 * 4 * terms


# 128 MB of partial row sums hold 69 of these 79 column tiles: two groups.  Against
# the same sums in torch; bounds as above.
def test_cross_covariance_cotangent_groups(cuda_lib):
    n, m, d = 30000, 5003, 8
    g = torch.Generator(device="cuda").manual_seed(1)
    x, z, G = (torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)
               for s in ((n, d), (m, d), (n, m)))
    ls = torch.linspace(0.7, 2.0, d, dtype=torch.float64)
    th = torch.cat([ls, torch.tensor([1.3, 0.0, 0.0], dtype=torch.float64)]).cuda()
    from gpjax_gb300.objectives import cross_covariance_vjp
    gth, gx, gz = cross_covariance_vjp(0, d, th, x, z, G, need_x=True, need_y=True)
    rx, rz, rl = torch.zeros_like(x), torch.zeros_like(z), torch.zeros(d + 1).to(x)
    xs, zs = x / ls.cuda(), z / ls.cuda()
    for lo in range(0, m, 500):
        k = torch.exp(-0.5 * sum((xs[:, None, q] - zs[None, lo:lo + 500, q]) ** 2
                                 for q in range(d)))
        c = G[:, lo:lo + 500] * k
        rl[d] += c.sum()
        for q in range(d):
            df = xs[:, None, q] - zs[None, lo:lo + 500, q]
            rx[:, q] -= 1.3 * (c * df).sum(1) / ls[q]
            rz[lo:lo + 500, q] = 1.3 * (c * df).sum(0) / ls[q]
            rl[q] += 1.3 * (c * df * df).sum() / ls[q]
    for got, ref, terms in ((gth[:d + 1], rl, n * m), (gx, rx, m), (gz, rz, n)):
        assert float((got - ref).abs().max()) <= 1e-12 * 4 * 1.3 * 4 * terms


# Columns on both sides of a 65536-wide block; the bounds of the parity test of
# the collapsed bound (the inducing points are spread: K is well conditioned).
@pytest.mark.parametrize("n,m", [(65536, 33), (65537, 150)])
def test_elbo_column_blocks(cuda_lib, n, m):
    rng = np.random.default_rng(n)
    x = rng.uniform(-2, 2, size=(n, 2))
    y = np.sin(x).sum(1, keepdims=True) + 0.1 * rng.standard_normal((n, 1))
    Z, ls = rng.uniform(-2, 2, (m, 2)), np.array([0.3, 0.4])
    val, g, gz = elbo_run(1, x, y, Z, ls, 1.2, 0.3, 0.1)
    ref, gref, gzref = elbo_oracle(1, x, y, Z, ls, 1.2, 0.3, 0.1)
    cond = np.linalg.cond(O.gram(1, Z, ls, 1.2) + 1e-6 * np.eye(m))
    tol = max(1e-9, 1e-12 * cond)
    assert abs(val - ref) <= tol * abs(ref)
    assert np.allclose(g, gref, rtol=max(1e-6, 10 * tol), atol=1e-7 * np.abs(gref).max())
    assert np.allclose(gz, gzref, rtol=max(1e-6, 10 * tol), atol=1e-7 * np.abs(gzref).max())


# Variances where 1 / variance is no number or Phi holds nothing: the bounds of
# the parity test for a well conditioned K.
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("var", [0.0, 1e-310, 1e-7, 30.0])
def test_elbo_small_variance(cuda_lib, kind, var):
    rng = np.random.default_rng(5)
    x = rng.uniform(-2, 2, size=(400, 2))
    y = np.sin(x).sum(1, keepdims=True) + 0.1 * rng.standard_normal((400, 1))
    Z, ls = x[:12], np.array([0.3, 0.4])
    val, g, gz = elbo_run(kind, x, y, Z, ls, var, 0.3, 0.1)
    ref, gref, gzref = elbo_oracle(kind, x, y, Z, ls, var, 0.3, 0.1)
    assert abs(val - ref) <= 1e-9 * abs(ref)
    assert np.allclose(g, gref, rtol=1e-6, atol=1e-7 * np.abs(gref).max())
    assert np.allclose(gz, gzref, rtol=1e-6, atol=1e-7 * np.abs(gzref).max())


# exp(-a) with a formed in float64 from t = sqrt(sq): a is off by at most 4 u a
# (square, sqrt, constant, product), so the value by (4 a + 6) u plus the
# functions' own last bit; past 708 the results are below 2^-1021, where one
# step of the subnormal range (2^-1074) is allowed as well.
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_kernel_values_over_range(cuda_lib, kind):
    r = np.concatenate([[0.0], np.exp(np.linspace(np.log(1e-9), np.log(400.0), 3000)),
                        np.linspace(30.0, 45.0, 500)])
    k = KINDS[kind](lengthscale=1.0, variance=1.0)
    k.lengthscale.to("cuda")
    k.variance.to("cuda")
    got = k.cross_covariance(torch.as_tensor(r[:, None], device="cuda"),
                             torch.zeros(1, 1, dtype=torch.float64, device="cuda"))
    got = got.detach().cpu().numpy()[:, 0]
    q = r.astype(np.longdouble)
    t = np.maximum(q, np.longdouble(1e-18))  # the kernels' floor of sq, 1e-36
    if kind == 0:
        a, f = q * q / 2, 1
    elif kind == 1:
        a = np.sqrt(np.longdouble(3)) * t
        f = 1 + a
    else:
        a = np.sqrt(np.longdouble(5)) * t
        f = 1 + a + a * a / 3
    ref = f * np.exp(-a)
    tol = (4 * a + 12) * U * ref + np.longdouble(2.0) ** -1074 * (1 + f)
    tol = np.where(ref < 2.0 ** -1021, np.maximum(tol, ref), tol)
    assert np.all(np.abs(got - ref) <= tol)


# d mll / d obs_stddev in 80-bit arithmetic (float64 and remainder): RBF of unit
# lengthscale and variance, noise 0.01, n = 1000, d = 4, inputs as below
NOISE_GRADIENTS = [
    (-531.36525574425, 1.0825e-14), (-739.6165996968416, 2.0428e-14),
    (-557.9018744831025, 1.1824e-14), (-482.77064718635705, -7.7161e-15),
    (-663.4948325301002, -2.2093e-14), (-634.2266094538219, -3.0476e-14),
    (-645.4184764004425, 1.9429e-15), (-505.19895390241936, -2.6701e-14),
    (-559.6680332924761, -1.2434e-14), (-559.0717053337254, 4.4797e-14),
    (-692.2731405473314, -1.6209e-14), (-496.50009117651143, -3.0531e-16),
    (-582.2574271196455, 2.9476e-14), (-646.1361506316309, 3.0809e-14),
    (-613.6955398755817, 1.5543e-14), (-557.0100501669929, 9.6589e-15)]


def test_noise_gradient_error(cuda_lib):
    """The factor's split products keep the accuracy of a native float64 factor,
    whose median error on these inputs is 7.6e-15 (a diagonal of 1.01 puts the
    digits' row scale, a power of two, at twice the row's bound)."""
    errors = []
    for seed, (hi, lo) in enumerate(NOISE_GRADIENTS):
        rng = np.random.default_rng(seed)
        x = rng.uniform(-3.0, 3.0, (1000, 4))
        y = x[:, 0] * x[:, 1] / 4 - x[:, 2] / 2 + 0.2 * rng.uniform(-1.0, 1.0, 1000)
        kern = gpx.kernels.RBF(lengthscale=1.0, variance=1.0)
        post = gpx.gps.Prior(kernel=kern) * gpx.likelihoods.Gaussian(1000, obs_stddev=0.1)
        for p in (kern.lengthscale, kern.variance, post.likelihood.obs_stddev):
            p.to("cuda")
        _, g = gpx.objectives.value_and_grad(gpx.objectives.conjugate_mll, post,
                                             gpx.Dataset(X=x, y=y[:, None]), precision="fp64")
        errors.append(abs((float(g["likelihood.obs_stddev"]) - hi) - lo) / abs(hi))
    assert np.median(errors) <= 7.6e-15, sorted(errors)


@pytest.mark.parametrize("n", [65, 129, 200, 321])
@pytest.mark.parametrize("diag", [1.01, 1.99, 2.01, 3.99, 7.9])
def test_mll_row_scales(cuda_lib, n, diag):
    """Equal inputs make Sigma c 1 1^T + s I, with everything known in closed
    form: diagonals around the powers of two and four at which the factor's digit
    planes change their scale, at the largest top digits."""
    s, y = 0.01, np.cos(np.arange(n))
    c = diag - s
    kern = gpx.kernels.RBF(lengthscale=1.0, variance=c)
    post = gpx.gps.Prior(kernel=kern, jitter=0.0) * gpx.likelihoods.Gaussian(n, obs_stddev=0.1)
    for p in (kern.lengthscale, kern.variance, post.likelihood.obs_stddev):
        p.to("cuda")
    val, g = gpx.objectives.value_and_grad(gpx.objectives.conjugate_mll, post,
                                           gpx.Dataset(X=np.zeros((n, 2)), y=y[:, None]),
                                           precision="fp64")
    t = s + n * c
    alpha = (y - c * y.sum() / t) / s
    ref = -0.5 * (y @ alpha + (n - 1) * np.log(s) + np.log(t) + n * np.log(2 * np.pi))
    total = y.sum() / t  # of alpha
    gv = 0.5 * (total ** 2 - n / t)
    gs = 0.1 * (alpha @ alpha - ((n - 1) / s + 1 / t))
    assert abs(float(val) - ref) <= 1e-10 * abs(ref)
    assert abs(float(g["prior.kernel.variance"]) - gv) <= 0.5e-7 * (total ** 2 + n / t)
    assert abs(float(g["likelihood.obs_stddev"]) - gs) <= 1e-7 * abs(gs)
