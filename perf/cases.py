"""The work that users of this library run on the GPU, as measurable cases.

Each case goes through a public entry point of ``libkriging_gb300`` the way a user's program calls it: host arrays in,
host arrays out, on a fitted model that the program keeps.  ``listed()`` holds the named cases, ``draw(rng)`` gives
further cases of the same ranges, ``prepare`` builds the model, ``run`` makes one call, ``work`` states what the call
cannot do without, and ``exact`` gives the same outputs from plain torch / numpy in 64 bits.

Kinds of calls:

* ``loglik``     concentrated log-likelihood and its theta-gradient at one theta: the step of every L-BFGS-B fit
* ``multistart`` the same for many thetas in one call: one optimiser round of a BFGS[k] fit
* ``loo``        leave-one-out objective and gradient: the step of a fit with objective "LOO"
* ``predict``    mean and stdev (and their derivatives) of a fitted model at new points
* ``nested``     log-likelihood and gradient of every submodel of a NestedKriging: the step of its fit
* ``vll``        Vecchia log-likelihood and gradient: the step of a fit with objective "LLVecchia(m)"
* ``sets``       the Vecchia order and conditioning sets: the start of such a fit
* ``vpredict``   predictVecchia: local kriging of each new point on its m nearest observations
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libkriging_gb300 as lk

EXACT_FLOPS = 8e12  # largest dense problem that exact() solves in 64 bits (a few seconds on the GPU)


def listed():
    return [
        # the plain interpolation model of the README's and the tests' scale: a fit is a hundred of these calls
        dict(name="loglik_n200", kind="loglik", n=200, d=3, kernel="matern5_2", trend="constant", nugget=False, slices=0),
        # an ordinary noisy design with a linear trend; odd size, so every tile has a ragged edge
        dict(name="loglik_n1003", kind="loglik", n=1003, d=4, kernel="matern3_2", trend="linear", nugget=True, slices=0),
        # a large design on the default (FP64) precision
        dict(name="loglik_n4096", kind="loglik", n=4096, d=8, kernel="matern5_2", trend="constant", nugget=True, slices=0),
        # the benchmark's design, with the precision that it uses
        dict(name="loglik_n16384_mixed", kind="loglik", n=16384, d=8, kernel="matern5_2", trend="constant", nugget=True,
             slices=7),
        # one optimiser round of a 64-start fit
        dict(name="multistart_64x2048", kind="multistart", n=2048, d=6, kernel="gauss", trend="constant", k=64),
        # one step of a leave-one-out fit
        dict(name="loo_n1000", kind="loo", n=1000, d=4, kernel="matern5_2", trend="constant"),
        # predicting a curve's or an image row's worth of points from a small model
        dict(name="predict_n200_q1000", kind="predict", n=200, d=3, kernel="matern5_2", trend="constant", q=1000,
             deriv=False, slices=0),
        # predicting a set of test points from a large model; odd sizes
        dict(name="predict_n4001_q5003", kind="predict", n=4001, d=6, kernel="matern5_2", trend="constant", q=5003,
             deriv=False, slices=0),
        # the submodels of a NestedKriging, sizes 150 .. 2500 as in its benchmark
        dict(name="nested_24", kind="nested", groups=24, lo=150, hi=2500, d=4, kernel="matern3_2"),
        # one step of a Vecchia fit
        dict(name="vll_n100003", kind="vll", n=100003, d=3, kernel="gauss", m=30),
        # the sets that such a fit builds first
        dict(name="sets_n32768", kind="sets", n=32768, d=3, m=30),
        # local predictions of many points
        dict(name="vpredict_n10007_q20000", kind="vpredict", n=10007, d=3, kernel="gauss", m=30, q=20000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loglik", "loglik", "loglik", "multistart", "loo", "predict", "predict", "nested", "vll", "sets",
                       "vpredict"])
    kernel = rng.choice(["gauss", "exp", "matern3_2", "matern5_2"])
    trend = rng.choice(["constant", "constant", "linear"])
    if kind == "loglik":
        slices = rng.choice([0, 0, 7])
        n = _log_int(rng, 512, 12000) if slices else _log_int(rng, 60, 5000)
        return dict(kind=kind, n=n, d=rng.randint(2, 10), kernel=kernel, trend=trend,
                    nugget=bool(slices) or rng.random() < 0.5, slices=slices)
    if kind == "multistart":
        n = _log_int(rng, 100, 2048)
        k = max(2, min(64, _log_int(rng, 2, 64)))
        return dict(kind=kind, n=n, d=rng.randint(3, 8), kernel=rng.choice(["gauss", "matern5_2"]), trend="constant", k=k)
    if kind == "loo":
        return dict(kind=kind, n=_log_int(rng, 100, 1600), d=rng.randint(2, 6), kernel=kernel, trend=trend)
    if kind == "predict":
        deriv = rng.random() < 0.3
        n = _log_int(rng, 60, 1500) if deriv else _log_int(rng, 60, 5000)
        q = _log_int(rng, 10, 500) if deriv else _log_int(rng, 10, 6000)
        return dict(kind=kind, n=n, d=rng.randint(2, 8), kernel="matern5_2" if deriv else kernel, trend="constant", q=q,
                    deriv=deriv, slices=rng.choice([0, 0, 7]))
    if kind == "nested":
        hi = _log_int(rng, 300, 2500)
        return dict(kind=kind, groups=rng.randint(4, 24), lo=max(100, hi // 12), hi=hi, d=rng.randint(3, 5),
                    kernel=rng.choice(["matern3_2", "matern5_2"]))
    d, m = rng.randint(2, 4), rng.randint(10, 30)
    kernel = "matern5_2" if d == 2 else rng.choice(["gauss", "matern5_2"])
    if kind == "vll":
        return dict(kind=kind, n=_log_int(rng, 3000, 100003), d=d, kernel=kernel, m=m)
    if kind == "sets":
        return dict(kind=kind, n=_log_int(rng, 2000, 32768), d=d, m=m)
    return dict(kind=kind, n=_log_int(rng, 500, 10007), d=d, kernel=kernel, m=m, q=_log_int(rng, 100, 20000))


# ------------------------------------------------------------------------------------------------------- inputs
NUGGET = 1e-6  # nugget / sigma2 of the noisy models
NUM_NUGGET = 1e-10  # the default jitter of the Vecchia conditional blocks


def _theta(rng, kernel, n, d, size=None):
    """Ranges of the size that fits of these designs end at: a few times the points' mean distance."""
    h = n ** (-1.0 / d)
    lo, hi = (0.8, 1.6 if d > 2 else 1.1) if kernel == "gauss" else (1.0, 3.0)
    return np.clip(rng.uniform(lo * h, hi * h, size=size if size is not None else d), 0.02, 1.5)


def _response(rng, X, noise=0.1):
    return np.sin(2 * np.pi * X).sum(axis=1) + noise * rng.standard_normal(X.shape[0])


def _inputs(c, seed):
    rng = np.random.default_rng([seed, 17])
    kind, d = c["kind"], c["d"]
    i = {}
    if kind == "nested":
        # group sizes spread over lo .. hi, the largest and the smallest among them; each group a slab of the first axis
        sizes = np.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]), size=c["groups"])).astype(int)
        sizes[0], sizes[-1] = c["hi"], c["lo"]
        n = int(sizes.sum())
        X = rng.uniform(size=(n, d))
        order = np.argsort(X[:, 0], kind="stable")
        labels = np.empty(n, dtype=np.int32)
        labels[order] = np.repeat(np.arange(c["groups"], dtype=np.int32), sizes)
        i["labels"] = labels
        i["theta"] = rng.uniform(0.1, 0.3, size=(c["groups"], d))
    else:
        n = c["n"]
        X = rng.uniform(size=(n, d))
        if kind == "multistart":
            i["theta"] = _theta(rng, c["kernel"], n, d, (c["k"], d))
        elif kind != "sets":
            i["theta"] = _theta(rng, c["kernel"], n, d)
        if "q" in c:
            i["Xq"] = rng.uniform(size=(c["q"], d))
    i["X"], i["y"] = np.asfortranarray(X), _response(rng, X)
    return i


def prepare(case, seed):
    c, i = case, _inputs(case, seed)
    kind, X, y = c["kind"], i["X"], i["y"]
    s = dict(kind=kind, case=c, **i)
    if kind == "sets":
        return s
    if kind == "nested":
        s["model"] = lk.NestedKriging(c["kernel"], aggregation="gPoE")
        s["model"].fit_groups(y, X, i["labels"], "constant", "none", "LL", {"theta": i["theta"][:1]})
        return s
    nugget = c.get("nugget", kind == "multistart")
    m = lk.Kriging(c["kernel"], "nugget") if nugget else lk.Kriging(c["kernel"])
    P = {"theta": i["theta"][:1] if i["theta"].ndim == 2 else i["theta"].reshape(1, -1)}
    if nugget:
        P.update(sigma2=1.0, nugget=NUGGET)
    if kind == "vll":
        m.set_vecchia_exact_commit(False)
        m.fit(y, X, "constant", False, "BFGS", "LLVecchia(%d)" % c["m"], P)
    else:
        m.fit(y, X, c.get("trend", "constant"), False, "none", "LL", P)
    if c.get("slices"):
        m.set_precision(c["slices"])
    alpha = 1.0 / (1.0 + NUGGET)
    if kind == "loglik":
        s["gamma"] = np.append(i["theta"], alpha) if nugget else i["theta"]
    elif kind == "multistart":
        s["gamma"] = np.hstack([i["theta"], np.full((c["k"], 1), alpha)])
    s["model"] = m
    return s


def run(state):
    kind, m, c = state["kind"], state.get("model"), state["case"]
    if kind == "loglik":
        ll, grad, _ = m.logLikelihoodFun(state["gamma"], True, False)
        return {"ll": np.float64(ll), "grad": grad}
    if kind == "multistart":
        ll, grad = m.logLikelihoodFunBatch(state["gamma"], True)
        return {"ll": ll, "grad": grad}
    if kind == "loo":
        loo, grad = m.leaveOneOutFun(state["theta"], True)
        return {"loo": np.float64(loo), "grad": grad}
    if kind == "predict":
        mean, sd, _, dmean, dsd = m.predict(state["Xq"], True, False, c["deriv"])
        return {"mean": mean, "sd": sd, "dmean": dmean, "dsd": dsd} if c["deriv"] else {"mean": mean, "sd": sd}
    if kind == "nested":
        ll, grad = m.logLikelihoodGroups(state["theta"], True)
        return {"ll": ll, "grad": grad}
    if kind == "vll":
        vll, grad = m.logLikelihoodVecchiaFun(state["theta"], True)
        return {"vll": np.float64(vll), "grad": grad}
    if kind == "sets":
        order, nbr = lk.vecchia_sets(state["X"], c["m"])
        return {"order": order, "nbr": nbr}
    mean, sd = m.predictVecchia(state["Xq"], True, c["m"])
    return {"mean": mean, "sd": sd}


# ------------------------------------------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; flops of the textbook algorithm (Cholesky and inverse from it)."""
    c, kind, d = case, case["kind"], case["d"]
    if kind == "nested":
        sizes = np.exp(np.linspace(math.log(c["lo"]), math.log(c["hi"]), c["groups"]))
        return {"bytes": float(8 * sizes.sum() * (d + 1) + 16 * c["groups"] * (d + 1)),
                "flops": float((sizes ** 3).sum() + (sizes ** 2).sum() * 3 * d)}
    n = float(c["n"])
    if kind in ("loglik", "multistart"):
        k = c.get("k", 1)
        return {"bytes": 8 * n * (d + 1) + 16.0 * k * (d + 2), "flops": k * (n ** 3 + 3 * d * n * n)}
    if kind == "loo":  # factor, inverse, and one n x n x n product per dimension
        return {"bytes": 8 * n * (d + 1) + 16.0 * (d + 1), "flops": n ** 3 * (1 + 2 * d) + 3 * d * n * n}
    if kind == "predict":  # the model holds its factor
        q = float(c["q"]) * (1 + d if c["deriv"] else 1)
        return {"bytes": 4 * n * n + 8 * n * (d + 2) + 8.0 * c["q"] * (d + 2), "flops": n * n * q + 2 * n * q * d}
    m = float(c.get("m", 0))
    if kind == "vll":
        return {"bytes": n * (8 * (d + 1) + 4 * (m + 1)), "flops": n * (m ** 3 / 3 + (d + 6) * m * m)}
    if kind == "sets":  # one distance for each neighbour, and the tree of the next point
        return {"bytes": n * (8 * d + 4 * (m + 1)), "flops": n * (3 * d * m + 2 * math.log2(n))}
    return {"bytes": n * 8 * (d + 1) + 8.0 * c["q"] * (d + 2), "flops": c["q"] * (3 * d * m + m ** 3 / 3 + 6 * m * m)}


# ------------------------------------------------------------------------------------------------------- exact
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_device())


def _corr(kernel, A, B, theta):
    """Correlations of the rows of A (... x a x d) and B (... x b x d)."""
    out = torch.ones(A.shape[:-1] + (B.shape[-2],), dtype=torch.float64, device=A.device)
    for k in range(A.shape[-1]):
        t = (A[..., :, None, k] - B[..., None, :, k]).abs() / theta[k]
        if kernel == "gauss":
            out *= torch.exp(-0.5 * t * t)
        elif kernel == "exp":
            out *= torch.exp(-t)
        elif kernel == "matern3_2":
            t = math.sqrt(3.0) * t
            out *= (1 + t) * torch.exp(-t)
        else:
            t = math.sqrt(5.0) * t
            out *= (1 + t + t * t / 3) * torch.exp(-t)
    return out


def _dln(kernel, dx, th):
    """d ln C / d theta of one dimension."""
    t = dx.abs() / th
    if kernel == "gauss":
        return t * t / th
    if kernel == "exp":
        return t / th
    if kernel == "matern3_2":
        t = math.sqrt(3.0) * t
        return t * t / (1 + t) / th
    t = math.sqrt(5.0) * t
    return (t * t / 3) * (1 + t) / (1 + t + t * t / 3) / th


def _trend(X, trend):
    one = torch.ones(X.shape[0], 1, dtype=X.dtype, device=X.device)
    return torch.cat([one, X], 1) if trend == "linear" else one


def _gls(L, F, y):
    """beta and L^-1 (y - F beta)."""
    Fs, ys = torch.linalg.solve_triangular(L, F, upper=False), torch.linalg.solve_triangular(L, y[:, None], upper=False)
    Q, R = torch.linalg.qr(Fs)
    beta = torch.linalg.solve_triangular(R, Q.T @ ys, upper=True)
    return beta[:, 0], (ys - Fs @ beta)[:, 0], Fs, R


def _exact_ll(c, X, y, theta, alpha):
    n, d = X.shape
    C = _corr(c["kernel"], X, X, theta)
    R = C * alpha
    R.fill_diagonal_(1.0)
    L = torch.linalg.cholesky(R)
    _, E, _, _ = _gls(L, _trend(X, c.get("trend", "constant")), y)
    s2 = (E @ E) / n
    ll = -0.5 * (n * torch.log(2 * math.pi * s2) + 2 * torch.log(torch.diagonal(L)).sum() + n)
    x = torch.linalg.solve_triangular(L.T, E[:, None], upper=True)[:, 0]
    W = torch.outer(x, x) / s2 - torch.cholesky_inverse(L)
    W.fill_diagonal_(0.0)
    grad = []
    WR = W * R
    for k in range(d):
        grad.append(0.5 * (WR * _dln(c["kernel"], X[:, None, k] - X[None, :, k], theta[k])).sum())
    if alpha != 1.0:  # d LL / d alpha of R = alpha C + (1 - alpha) I
        C.fill_diagonal_(0.0)
        grad.append(0.5 * (W * C).sum())
    return float(ll), torch.stack(grad).cpu().numpy()


def _exact_loo(c, X, y, theta):
    n, d = X.shape
    R = _corr(c["kernel"], X, X, theta)
    L = torch.linalg.cholesky(R)
    Ri = torch.cholesky_inverse(L)
    F = _trend(X, c["trend"])
    RiF = Ri @ F
    B = Ri - RiF @ torch.linalg.solve(F.T @ RiF, RiF.T)
    By, s2 = B @ y, 1 / torch.diagonal(B)
    e = s2 * By
    grad = []
    for k in range(d):
        G = R * _dln(c["kernel"], X[:, None, k] - X[None, :, k], theta[k])
        BG = B @ G
        de = s2 * s2 * (BG * B.T).sum(1) * By - s2 * (BG @ By)
        grad.append(2 * (e * de).sum() / n)
    return float((e @ e) / n), torch.stack(grad).cpu().numpy()


def _exact_predict(c, X, y, theta, Xq):
    n, d = X.shape
    L = torch.linalg.cholesky(_corr(c["kernel"], X, X, theta))
    beta, E, Fs, Rs = _gls(L, _trend(X, c["trend"]), y)
    s2 = (E @ E) / n
    r = _corr(c["kernel"], X, Xq, theta)
    rs = torch.linalg.solve_triangular(L, r, upper=False)
    f = _trend(Xq, c["trend"])
    mean = f @ beta + rs.T @ E
    u = torch.linalg.solve_triangular(Rs, f - rs.T @ Fs, upper=True, left=False)
    var = s2 * (1 - (rs * rs).sum(0) + (u * u).sum(1)).clamp_min(0.0)
    out = {"mean": mean.cpu().numpy(), "sd": var.sqrt().cpu().numpy()}
    if c["deriv"]:  # matern5_2, constant trend
        dm, ds = torch.empty(len(Xq), d, dtype=r.dtype, device=r.device), torch.empty(len(Xq), d, dtype=r.dtype, device=r.device)
        for k in range(d):
            dx = Xq[None, :, k] - X[:, None, k]
            t = math.sqrt(5.0) * dx.abs() / theta[k]
            dr = -r * torch.sign(dx) * math.sqrt(5.0) / theta[k] * (t / 3) * (1 + t) / (1 + t + t * t / 3)
            drs = torch.linalg.solve_triangular(L, dr, upper=False)
            du = torch.linalg.solve_triangular(Rs, -(drs.T @ Fs), upper=True, left=False)
            dm[:, k] = drs.T @ E
            ds[:, k] = s2 * (-2 * (rs * drs).sum(0) + 2 * (u * du).sum(1)) / (2 * var.sqrt())
        out.update(dmean=dm.cpu().numpy(), dsd=ds.cpu().numpy())
    return out


def _order_and_sets(X, m):
    """Maxmin order from the point nearest the centroid, and each point's m nearest earlier points."""
    n = X.shape[0]

    def dist2(i):
        s = torch.zeros(n, dtype=X.dtype, device=X.device)
        for k in range(X.shape[1]):
            t = X[:, k] - X[i, k]
            s += t * t
        return s

    order = torch.empty(n, dtype=torch.int64, device=X.device)
    c = ((X - X.mean(0)) ** 2).sum(1).argmin().reshape(1)
    order[0:1] = c
    near = dist2(c)
    near[c] = -math.inf
    for t in range(1, n):
        c = near.argmax().reshape(1)
        order[t:t + 1] = c
        torch.minimum(near, dist2(c), out=near)
        near[c] = -math.inf
    Z = X[order]
    nbr = torch.full((n, m), -1, dtype=torch.int64, device=X.device)
    for a in range(0, n, 2048):
        b = min(n, a + 2048)
        D = torch.zeros(b - a, b, dtype=X.dtype, device=X.device)
        for k in range(X.shape[1]):
            t = Z[a:b, k, None] - Z[None, :b, k]
            D += t * t
        at = torch.arange(b, device=X.device)
        D.masked_fill_(at[None, :] >= torch.arange(a, b, device=X.device)[:, None], math.inf)
        v, j = D.topk(min(m, b), dim=1, largest=False)
        nbr[a:b, :j.shape[1]] = torch.where(torch.isinf(v), -1, order[j])
    return order, nbr


def _exact_vll(c, X, y, theta):
    n, d = X.shape
    order, nbr = _order_and_sets(X, c["m"])
    U, V, W, dU, dV, dW = [], [], [], [], [], []
    for a in range(0, n, 8192):
        o, N = order[a:a + 8192], nbr[a:a + 8192]
        has = (N >= 0)
        Nc = N.clamp_min(0)
        XN, x, yN = X[Nc], X[o], y[Nc] * has
        pair = has[:, :, None] & has[:, None, :]
        RN = _corr(c["kernel"], XN, XN, theta) * pair
        RN.diagonal(dim1=1, dim2=2).copy_(1.0 + NUM_NUGGET * has.to(X.dtype))
        r = _corr(c["kernel"], XN, x[:, None, :], theta)[:, :, 0] * has
        L = torch.linalg.cholesky(RN)
        av = torch.cholesky_solve(r[:, :, None], L)[:, :, 0]
        U.append(y[o] - (av * yN).sum(1))
        V.append((1 - (r * av).sum(1)).clamp_min(1e-15))
        W.append(1 - (av * has).sum(1))
        du, dv, dw = [], [], []
        for k in range(d):
            M = RN * _dln(c["kernel"], XN[:, :, None, k] - XN[:, None, :, k], theta[k])
            M.diagonal(dim1=1, dim2=2).zero_()
            dr = r * _dln(c["kernel"], XN[:, :, k] - x[:, None, k], theta[k])
            da = torch.cholesky_solve((dr - (M @ av[:, :, None])[:, :, 0])[:, :, None], L)[:, :, 0]
            dv.append(-((dr * av).sum(1) + (r * da).sum(1)))
            du.append(-(da * yN).sum(1))
            dw.append(-(da * has).sum(1))
        dU.append(torch.stack(du, 1))
        dV.append(torch.stack(dv, 1))
        dW.append(torch.stack(dw, 1))
    U, V, W, dU, dV, dW = (torch.cat(v) for v in (U, V, W, dU, dV, dW))
    beta = (W * U / V).sum() / ((W * W / V).sum() + NUM_NUGGET)
    e = U - W * beta
    Q = (e * e / V).sum()
    vll = -0.5 * n * torch.log(2 * math.pi * Q / n) - 0.5 * torch.log(V).sum() - 0.5 * n
    de = dU - dW * beta
    dQ = (2 * e[:, None] * de / V[:, None] - (e * e / (V * V))[:, None] * dV).sum(0)
    grad = -0.5 * n * dQ / Q - 0.5 * (dV / V[:, None]).sum(0)
    return float(vll), grad.cpu().numpy()


def _exact_vpredict(c, X, y, theta, Xq):
    L = torch.linalg.cholesky(_corr(c["kernel"], X, X, theta))
    beta, E, _, _ = _gls(L, _trend(X, "constant"), y)
    beta, s2 = beta[0], (E @ E) / len(X)
    mean, sd = [], []
    for a in range(0, len(Xq), 2048):
        x = Xq[a:a + 2048]
        D = torch.zeros(len(x), len(X), dtype=X.dtype, device=X.device)
        for k in range(X.shape[1]):
            t = x[:, None, k] - X[None, :, k]
            D += t * t
        N = D.topk(c["m"], dim=1, largest=False)[1]
        RN = _corr(c["kernel"], X[N], X[N], theta)
        RN.diagonal(dim1=1, dim2=2).fill_(1.0 + NUM_NUGGET)
        r = _corr(c["kernel"], X[N], x[:, None, :], theta)
        av = torch.cholesky_solve(r, torch.linalg.cholesky(RN))
        mean.append(beta + (av[:, :, 0] * (y[N] - beta)).sum(1))
        sd.append((s2 * (1 - (r * av).sum((1, 2))).clamp_min(0.0)).sqrt())
    return {"mean": torch.cat(mean).cpu().numpy(), "sd": torch.cat(sd).cpu().numpy()}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "sets":
        return None  # whole numbers: equal or not
    if kind in ("loglik", "multistart", "loo", "nested") and work(c)["flops"] > EXACT_FLOPS:
        return None
    i = _inputs(c, seed)
    X, y = _t(i["X"]), _t(i["y"])
    alpha = 1.0 / (1.0 + NUGGET)
    if kind == "loglik":
        ll, grad = _exact_ll(c, X, y, _t(i["theta"]), alpha if c["nugget"] else 1.0)
        return {"ll": np.float64(ll), "grad": grad}
    if kind in ("multistart", "nested"):
        ll, grad = [], []
        for g, th in enumerate(i["theta"]):
            at = torch.as_tensor(np.flatnonzero(i["labels"] == g), device=X.device) if kind == "nested" else slice(None)
            v, dv = _exact_ll(c, X[at], y[at], _t(th), alpha if kind == "multistart" else 1.0)
            ll.append(v)
            grad.append(dv)
        return {"ll": np.array(ll), "grad": np.array(grad)}
    if kind == "loo":
        loo, grad = _exact_loo(c, X, y, _t(i["theta"]))
        return {"loo": np.float64(loo), "grad": grad}
    if kind == "predict":
        return _exact_predict(c, X, y, _t(i["theta"]), _t(i["Xq"]))
    if kind == "vll":
        vll, grad = _exact_vll(c, X, y, _t(i["theta"]))
        return {"vll": np.float64(vll), "grad": grad}
    return _exact_vpredict(c, X, y, _t(i["theta"]), _t(i["Xq"]))
