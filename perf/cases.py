"""The work that users of this library have it do, as timed cases.

Each case is one call of a public entry point on inputs of the kind that the
call meets in use: the marginal likelihood with its gradient (one step of a
hyperparameter fit) in the float64 and the mixed form, prediction, the SGPR
bound with its gradient, a batch of independent GPs, and a cross-covariance
with its cotangents.  ``draw`` gives further cases of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gpjax_gb300 as gpx
from gpjax_gb300.objectives import BatchPlan, collapsed_elbo, conjugate_mll, value_and_grad

KERNELS = ("RBF", "Matern32", "Matern52", "Matern12", "RationalQuadratic")
ALPHA = 1.0        # shape of the rational quadratic kernel (its default)
EXACT_MLL_N = 17000  # above this the float64 reference takes longer than 20 s


def listed():
    return [
        # the introductory regression problem: one optimiser step at n = 100
        # in the default precision; launches and host work are the whole cost
        dict(name="mll_f64_n100", what="mll", precision="fp64", kernel="RBF", n=100, d=1,
             ard=False, data="box", noise=1e-2),
        # the plain conjugate GP configuration (X ~ U[-3, 3]^4, RBF)
        dict(name="mll_f64_n2048", what="mll", precision="fp64", kernel="RBF", n=2048, d=4,
             ard=False, data="box", noise=1e-2),
        # the largest exact GP that is still fitted in the default precision
        dict(name="mll_f64_n9001", what="mll", precision="fp64", kernel="Matern52", n=9001, d=8,
             ard=True, data="normal", noise=1e-2),
        # an ordinary dataset of ragged size in the mixed form
        dict(name="mll_mixed_n1500", what="mll", precision="mixed", kernel="Matern32", n=1500, d=5,
             ard=True, data="normal", noise=1e-2),
        # the headline: n = 16384, d = 8, Matern-5/2 ARD
        dict(name="mll_mixed_n16384", what="mll", precision="mixed", kernel="Matern52", n=16384,
             d=8, ard=True, data="normal", noise=1e-2),
        # large, sixteen inputs, low noise (the precision-stress distribution)
        dict(name="mll_mixed_n32768", what="mll", precision="mixed", kernel="RBF", n=32768, d=16,
             ard=True, data="unit", noise=1e-3),
        # posterior at 512 points with its full covariance, the default call
        dict(name="predict_f64_n2048", what="predict", precision="fp64", kernel="RBF", n=2048, d=4,
             ard=False, data="box", noise=1e-2, t=512, cov=True),
        # mean and variance at many points (an acquisition sweep, a test set)
        dict(name="predict_mixed_n8192", what="predict", precision="mixed", kernel="RBF", n=8192,
             d=16, ard=True, data="unit", noise=1e-3, t=4096, cov=False),
        # a sparse GP of ordinary size in the default precision
        dict(name="elbo_f64_n20000", what="elbo", precision="fp64", kernel="Matern52", n=20000,
             d=8, ard=True, m=300, noise=1e-2),
        # the large sparse GP: a million points, 1024 inducing points
        dict(name="elbo_mixed_n1e6", what="elbo", precision="mixed", kernel="RBF", n=1_000_000,
             d=8, ard=True, m=1024, noise=1e-2),
        # 512 independent GPs of 64 to 2048 points (multi-start fits)
        dict(name="batch_512", what="batch", count=512, n_lo=64, n_hi=2048, sizes=0),
        # a kernel matrix between two point sets and its cotangents (user-built models)
        dict(name="cross_cov_n3000", what="cross", kernel="Matern52", n=3000, m=1100, d=5,
             ard=True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["mll_f64", "mll_f64", "mll_mixed", "mll_mixed", "predict", "elbo", "batch",
                       "cross"])
    kernel = rng.choice(KERNELS)
    d = rng.randint(1, 16)
    ard = d > 1 and rng.random() < 0.7
    data = rng.choice(["box", "normal", "unit"])
    if what == "mll_f64":
        return dict(what="mll", precision="fp64", kernel=kernel, n=_log_int(rng, 64, 9001), d=d,
                    ard=ard, data=data, noise=1e-2)
    if what == "mll_mixed":
        return dict(what="mll", precision="mixed", kernel=kernel, n=_log_int(rng, 512, 32768),
                    d=d, ard=ard, data=data, noise=1e-2)
    if what == "predict":
        mixed = rng.random() < 0.5
        return dict(what="predict", precision="mixed" if mixed else "fp64", kernel=kernel,
                    n=_log_int(rng, 100, 8192 if mixed else 4096), d=d, ard=ard, data=data,
                    noise=1e-2, t=_log_int(rng, 50, 4096 if mixed else 1024),
                    cov=(not mixed) and rng.random() < 0.7)
    if what == "elbo":
        mixed = rng.random() < 0.5
        return dict(what="elbo", precision="mixed" if mixed else "fp64",
                    kernel=rng.choice(["RBF", "Matern32", "Matern52"]),
                    n=_log_int(rng, 2000, 1_000_000 if mixed else 30000), d=rng.randint(4, 10),
                    ard=ard, m=_log_int(rng, 50, 1024 if mixed else 400), noise=1e-2)
    if what == "batch":
        lo = rng.choice([16, 64, 100])
        return dict(what="batch", count=_log_int(rng, 8, 512), n_lo=lo,
                    n_hi=_log_int(rng, 2 * lo, 2048), sizes=rng.randint(0, 1 << 30))
    return dict(what="cross", kernel=kernel, n=_log_int(rng, 50, 6000), m=_log_int(rng, 20, 2000),
                d=d, ard=ard)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64, device=_dev())


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device=_dev())


def _prior_sample(g, kernel, x, ls, var, freqs=128):
    """A draw from (a finite-feature approximation of) the GP prior at x."""
    z = _normal(g, freqs, x.shape[1])
    nu = {"Matern12": 1, "Matern32": 3, "Matern52": 5}.get(kernel)
    if nu is not None:  # spectral density of the Matern family: a multivariate t
        z = z / torch.sqrt(_normal(g, freqs, nu).square().sum(1, keepdim=True) / nu)
    proj = (x / ls) @ z.T
    w = _normal(g, 2, freqs) * math.sqrt(var / freqs)
    return torch.cos(proj) @ w[0] + torch.sin(proj) @ w[1]


def _points(g, data, n, d):
    if data == "box":
        return _uniform(g, -3.0, 3.0, n, d)
    if data == "unit":
        return _uniform(g, 0.0, 1.0, n, d)
    return _normal(g, n, d)


def _lengthscale(g, case):
    lo, hi = (0.1, 1.0) if case.get("data") == "unit" else (0.3, 3.0)
    if case["what"] == "elbo":
        lo, hi = 0.5, 2.0
    if not case["ard"]:
        return torch.ones((), dtype=torch.float64, device=_dev())
    return torch.exp(_uniform(g, math.log(lo), math.log(hi), case["d"]))


def _inputs(case, seed):
    """The arrays of one case (everything but the library's objects)."""
    g = _gen(seed)
    if case["what"] == "batch":
        return _batch_inputs(case, seed, g)
    d, n = case["d"], case["n"]
    ls, var = _lengthscale(g, case), 1.0
    if case["what"] == "cross":
        x, z = _normal(g, n, d), _normal(g, case["m"], d)
        return dict(x=x, z=z, ls=ls, var=var, G=_normal(g, n, case["m"]))
    sd = math.sqrt(case["noise"])
    if case["what"] == "elbo":
        means = _uniform(g, -5.0, 5.0, 16, d)
        comp = torch.randint(0, 16, (n,), generator=g, device=_dev())
        x = means[comp] + 0.5 * _normal(g, n, d)
        y = torch.sin(x).sum(1) + sd * _normal(g, n)
        z = x[torch.randperm(n, generator=g, device=_dev())[:case["m"]]].clone()
        return dict(x=x, y=y[:, None].contiguous(), z=z, ls=ls, var=var, sd=sd)
    x = _points(g, case["data"], n, d)
    y = _prior_sample(g, case["kernel"], x, ls, var) + sd * _normal(g, n)
    out = dict(x=x, y=y[:, None].contiguous(), ls=ls, var=var, sd=sd)
    if case["what"] == "predict":
        out["t"] = _points(g, case["data"], case["t"], d)
    return out


def _batch_inputs(case, seed, g):
    """n ~ U{n_lo..n_hi}, d ~ U{2..10}, X ~ U[-1, 1]^d, RBF or Matern-3/2 with
    probability one half, log-uniform hyperparameters.  The sizes belong to
    the case, everything else to the seed."""
    shapes, rng = np.random.default_rng(case["sizes"]), np.random.default_rng(int(seed))
    items = []
    for _ in range(case["count"]):
        n, d = int(shapes.integers(case["n_lo"], case["n_hi"] + 1)), int(shapes.integers(2, 11))
        kernel = "RBF" if rng.random() < 0.5 else "Matern32"
        ls = np.exp(rng.uniform(np.log(0.1), np.log(2.0), d))
        var = float(np.exp(rng.uniform(np.log(0.5), np.log(2.0))))
        noise = float(np.exp(rng.uniform(np.log(1e-3), np.log(1e-1))))
        theta = torch.tensor([*ls, var, math.sqrt(noise), 0.0], dtype=torch.float64, device=_dev())
        x = _uniform(g, -1.0, 1.0, n, d)
        y = _prior_sample(g, kernel, x, theta[:d], var, freqs=100) + 0.05 * _normal(g, n)
        items.append((kernel, x, y, theta))
    return items


# ---------------------------------------------------------------------------
# What a program keeps, and one pass
# ---------------------------------------------------------------------------
def _kernel(case, a):
    kw = dict(alpha=ALPHA) if case["kernel"] == "RationalQuadratic" else {}
    kern = getattr(gpx.kernels, case["kernel"])(lengthscale=a["ls"], variance=a["var"], **kw)
    kern.lengthscale.to(_dev())
    kern.variance.to(_dev())
    return kern


def _posterior(case, a):
    prior = gpx.gps.Prior(kernel=_kernel(case, a),
                          mean_function=gpx.mean_functions.Constant(gpx.parameters.Real(0.0)))
    post = prior * gpx.likelihoods.Gaussian(case["n"], obs_stddev=a["sd"])
    post.likelihood.obs_stddev.to(_dev())
    prior.mean_function.constant.to(_dev())
    return post


def prepare(case, seed):
    a = _inputs(case, seed)
    what = case["what"]
    if what == "batch":
        plan = BatchPlan([getattr(gpx.kernels, k).kind for k, _, _, _ in a], [i[1] for i in a],
                         [i[2] for i in a], [i[3] for i in a], [i[1].shape[1] for i in a])
        return dict(case=case, plan=plan)
    if what == "cross":
        kern = _kernel(case, a)
        for p in (kern.lengthscale, kern.variance):
            p.requires_grad_(True)
        return dict(case=case, kern=kern, x=a["x"].requires_grad_(True),
                    z=a["z"].requires_grad_(True), G=a["G"])
    post = _posterior(case, a)
    state = dict(case=case, post=post, data=gpx.Dataset(X=a["x"], y=a["y"]))
    if what == "elbo":
        state["q"] = gpx.variational_families.CollapsedVariationalGaussian(
            posterior=post, inducing_inputs=gpx.parameters.Real(a["z"]))
    if what == "predict":
        state["t"] = a["t"]
    return state


_GRADS = {"lengthscale": "prior.kernel.lengthscale", "variance": "prior.kernel.variance",
          "obs_stddev": "likelihood.obs_stddev", "constant": "prior.mean_function.constant"}


def run(state):
    case = state["case"]
    what = case["what"]
    if what == "batch":
        mll, grads, info = state["plan"].execute()
        return dict(mll=mll, grads=torch.cat(grads), info=info)
    if what == "cross":
        kern, x, z = state["kern"], state["x"], state["z"]
        K = kern.cross_covariance(x, z)
        g = torch.autograd.grad(K, [kern.lengthscale.value, kern.variance.value, x, z],
                                state["G"])
        return dict(K=K.detach(), lengthscale=g[0], variance=g[1], x=g[2], z=g[3])
    if what == "predict":
        dist = state["post"].predict(state["t"], state["data"], precision=case["precision"],
                                     full_covariance=case["cov"])
        out = dict(mean=dist.mean, variance=dist.variance)
        if case["cov"]:
            out["covariance"] = dist.covariance()
        return out
    if what == "elbo":
        val, g = value_and_grad(collapsed_elbo, state["q"], state["data"],
                                precision=case["precision"])
        out = {k: g["posterior." + name] for k, name in _GRADS.items()}
        return dict(value=val, z=g["inducing_inputs"], **out)
    val, g = value_and_grad(conjugate_mll, state["post"], state["data"],
                            precision=case["precision"])
    return dict(value=val, **{k: g[name] for k, name in _GRADS.items()})


def work(case):
    what = case["what"]
    if what == "batch":
        lo, hi = case["n_lo"], case["n_hi"]  # means of n^3 and n over the uniform sizes
        n3 = sum(float(n) ** 3 for n in range(lo, hi + 1)) / (hi - lo + 1)
        nm = 0.5 * (lo + hi)
        return {"bytes": case["count"] * 8.0 * (nm * 7 + 20), "flops": case["count"] * n3}
    n, d = float(case["n"]), float(case["d"])
    if what == "cross":
        m = float(case["m"])
        return {"bytes": 8 * (2 * n * m + 2 * (n + m) * d), "flops": n * m * (8 * d + 20)}
    if what == "predict":
        t = float(case["t"])
        flops = n ** 3 / 3 + n * n * t + (n * t * t if case["cov"] else 0.0)
        return {"bytes": 8 * (n * (d + 1) + t * (d + 2) + (t * t if case["cov"] else 0.0)),
                "flops": flops}
    if what == "elbo":
        m = float(case["m"])
        return {"bytes": 8 * (n * (d + 1) + 2 * m * d), "flops": 3 * m * m * n + 4 * m ** 3}
    return {"bytes": 8 * (n * (d + 1) + d + 4), "flops": n ** 3}


# ---------------------------------------------------------------------------
# The same results from plain torch in float64
# ---------------------------------------------------------------------------
def _unit_kernel(kernel, sq):
    """(k, c) for unit variance on scaled squared distances: the kernel value
    and c = -2 dk/dsq."""
    if kernel == "RBF":
        k = torch.exp(-0.5 * sq)
        return k, k
    if kernel == "RationalQuadratic":
        u = 1.0 + sq / (2.0 * ALPHA)
        k = u ** -ALPHA
        return k, k / u
    t = torch.sqrt(torch.clamp(sq, min=1e-36))
    if kernel == "Matern12":
        k = torch.exp(-t)
        return k, torch.where(sq > 1e-36, k / t, torch.zeros_like(k))
    if kernel == "Matern32":
        e = torch.exp(-math.sqrt(3.0) * t)
        return (1.0 + math.sqrt(3.0) * t) * e, 3.0 * e
    r = math.sqrt(5.0) * t
    e = torch.exp(-r)
    return (1.0 + r + 5.0 / 3.0 * t * t) * e, 5.0 / 3.0 * (1.0 + r) * e


def _sqdist(xs, zs):
    sq = torch.zeros(xs.shape[0], zs.shape[0], dtype=torch.float64, device=xs.device)
    for k in range(xs.shape[1]):
        sq += (xs[:, k, None] - zs[None, :, k]).square_()
    return sq


def _cotangents(kernel, x, z, ls, var, G):
    """sum_ij G_ij dK_ij/d(lengthscale, variance, x, z) for K = K(x, z)."""
    xs, zs = x / ls, z / ls
    k, c = _unit_kernel(kernel, _sqdist(xs, zs))
    gv = (G * k).sum()
    gc = var * G * c
    gl, gx, gz = torch.zeros(x.shape[1]).to(x), torch.zeros_like(x), torch.zeros_like(z)
    lv = ls.expand(x.shape[1])
    for q in range(x.shape[1]):
        df = xs[:, q, None] - zs[None, :, q]
        t = gc * df
        gx[:, q] = -t.sum(1) / lv[q]
        gz[:, q] = t.sum(0) / lv[q]
        gl[q] = (t * df).sum() / lv[q]
    return (gl if ls.ndim else gl.sum()), gv, gx, gz


def _exact_mll(kernel, x, y, ls, var, sd, const=0.0):
    n = x.shape[0]
    K = var * _unit_kernel(kernel, _sqdist(x / ls, x / ls))[0]
    K.diagonal().add_(1e-6 + sd * sd)
    L = torch.linalg.cholesky(K)
    diff = y.reshape(-1, 1) - const
    alpha = torch.cholesky_solve(diff, L)
    alpha += torch.cholesky_solve(diff - K @ alpha, L)
    logdet = 2.0 * torch.log(L.diagonal()).sum()
    val = -0.5 * (n * math.log(2.0 * math.pi) + logdet + (diff * alpha).sum())
    del K
    G = torch.cholesky_inverse(L)
    del L
    G.mul_(-0.5)
    G.addmm_(alpha, alpha.T, alpha=0.5)
    gl, gv, _, _ = _cotangents(kernel, x, x, ls, var, G)
    return val, gl, gv, 2.0 * sd * G.diagonal().sum(), alpha.sum()


def _exact_predict(case, a):
    x, ls = a["x"], a["ls"]
    K = _unit_kernel(case["kernel"], _sqdist(x / ls, x / ls))[0]
    K.diagonal().add_(1e-6 + a["sd"] ** 2)
    L = torch.linalg.cholesky(K)
    Kxt = _unit_kernel(case["kernel"], _sqdist(x / ls, a["t"] / ls))[0]
    alpha = torch.cholesky_solve(a["y"], L)
    alpha += torch.cholesky_solve(a["y"] - K @ alpha, L)
    Q = torch.linalg.solve_triangular(L, Kxt, upper=False)
    out = dict(mean=(Kxt.T @ alpha)[:, 0], variance=1.0 + 1e-6 - Q.square().sum(0))
    if case["cov"]:
        cov = _unit_kernel(case["kernel"], _sqdist(a["t"] / ls, a["t"] / ls))[0] - Q.T @ Q
        cov.diagonal().add_(1e-6)
        out["covariance"] = cov
    return out


def _exact_elbo(case, a):
    """The collapsed bound through P = Phi Phi^T and c = Phi d, differentiated
    by autograd down to (K, P, c) and by hand from there to the inputs."""
    kernel, x, z, ls, var, sd = (case["kernel"], *(a[k] for k in ("x", "z", "ls", "var", "sd")))
    n, m = x.shape[0], z.shape[0]
    diff = a["y"][:, 0]
    step = max(1, 40_000_000 // m)
    P, c = torch.zeros(m, m).to(x), torch.zeros(m).to(x)

    def phi(lo):
        return var * _unit_kernel(kernel, _sqdist(z / ls, x[lo:lo + step] / ls))[0]

    for lo in range(0, n, step):
        f = phi(lo)
        P += f @ f.T
        c += f @ diff[lo:lo + step]
    K = var * _unit_kernel(kernel, _sqdist(z / ls, z / ls))[0]
    K.diagonal().add_(1e-6)
    s, s2, dd = (torch.tensor(float(v), dtype=torch.float64, device=x.device)
                 for v in (sd * sd, var, diff @ diff))
    leaves = [t.requires_grad_(True) for t in (K, P, c, s, s2, dd)]
    Lk, Lu = torch.linalg.cholesky(K), torch.linalg.cholesky(K + P / s)
    g = torch.cholesky_solve(c[:, None], Lu)[:, 0]
    trace = torch.cholesky_solve(P, Lk).diagonal().sum()
    logdets = 2.0 * (torch.log(Lu.diagonal()).sum() - torch.log(Lk.diagonal()).sum())
    val = 0.5 * (-n * torch.log(2.0 * math.pi * s) - logdets - (dd / s - c @ g / s ** 2)
                 - (n * s2 / s - trace / s))
    dK, dP, dc, ds, dvar, ddd = torch.autograd.grad(val, leaves)
    with torch.no_grad():
        dK, dP = 0.5 * (dK + dK.T), 0.5 * (dP + dP.T)
        gl, gv, ga, gb = _cotangents(kernel, z, z, ls, var, dK)
        gz = ga + gb
        gv = gv + dvar
        gm = -2.0 * ddd * diff.sum()
        for lo in range(0, n, step):
            f, dl = phi(lo), diff[lo:lo + step]
            l1, v1, z1, _ = _cotangents(kernel, z, x[lo:lo + step], ls, var,
                                        2.0 * dP @ f + dc[:, None] * dl[None, :])
            gl, gv, gz = gl + l1, gv + v1, gz + z1
            gm = gm - (f.T @ dc).sum()
    return dict(value=val.detach(), z=gz, lengthscale=gl, variance=gv, obs_stddev=2.0 * sd * ds,
                constant=gm)


def exact(case, seed):
    what = case["what"]
    if what == "mll" and case["n"] > EXACT_MLL_N:
        return None
    a = _inputs(case, seed)
    if what == "batch":
        vals, grads = [], []
        for kernel, x, y, theta in a:
            d = x.shape[1]
            r = _exact_mll(kernel, x, y, theta[:d], theta[d], theta[d + 1])
            vals.append(r[0])
            grads.append(torch.cat([r[1], r[2].reshape(1), r[3].reshape(1), r[4].reshape(1)]))
        return dict(mll=torch.stack(vals), grads=torch.cat(grads), info=None)
    if what == "cross":
        K = _unit_kernel(case["kernel"], _sqdist(a["x"] / a["ls"], a["z"] / a["ls"]))[0]
        gl, gv, gx, gz = _cotangents(case["kernel"], a["x"], a["z"], a["ls"], 1.0, a["G"])
        return dict(K=K, lengthscale=gl, variance=gv, x=gx, z=gz)
    if what == "predict":
        return _exact_predict(case, a)
    if what == "elbo":
        return _exact_elbo(case, a)
    val, gl, gv, gs, gm = _exact_mll(case["kernel"], a["x"], a["y"], a["ls"], a["var"], a["sd"])
    return dict(value=val, lengthscale=gl, variance=gv, obs_stddev=gs, constant=gm)
