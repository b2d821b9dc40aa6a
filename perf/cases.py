"""Performance cases: the calls a user of the library makes, through its public entry points.

A case is a dict of plain values.  `kind` selects the call:

  loglik     Session.loglik(theta): one objective evaluation, what every optimiser iteration does
  grad       Session.loglik(theta, grad=True): one objective + gradient evaluation of a gradient fit
  synthetic  Session.zvg(theta, e) and Session.z(): observations drawn from the model
  batch      Batch.loglik(thetas[, grad=True]): many regional fields, each with its own theta
  predict    Session.predict(...): kriging of held-out points with its mean square error
  assess     Session.fisher(theta) and mloe_mmom_host(...): the assessment of a finished fit

Locations are jittered grids in Morton order (unit square, or latitude / longitude in degrees for the
great-circle metric), uniform in the unit square for batches; observations are a sum of random plane
waves with the Matern spectral density (their covariance is the model's), so E[z' Sigma^-1 z] = N as
for a field drawn from the model itself.  theta is the named model's, moved by a few percent per
seed, as along an optimiser's path.  The reduced-precision gradient (precision 3) is an approximation good
to 1e-4 .. 1e-6 whose further digits are rounding noise, and so is not among the cases.
"""
import math

import numpy as np
import torch

import exageostat_b200 as xg

EARTH_KM = 6371.0


def listed():
    return [
        # the smallest fits: a few hundred stations, general smoothness; latency decides
        dict(name="loglik_n400", kind="loglik", n=400, kernel=0, dm="ed", dts=0, precision=0, beta=0.1, nu=0.73),
        # the 40 x 40 grid of the reference driver, exponential kernel, tile 320 as its command line has it
        dict(name="loglik_n1600", kind="loglik", n=1600, kernel=0, dm="ed", dts=320, precision=0, beta=0.1, nu=0.5),
        # an ordinary station network on the sphere with measurement error, ragged size
        dict(name="loglik_n5987_gc_nugget", kind="loglik", n=5987, kernel=1, dm="gc", dts=0, precision=0, beta=60.0,
             nu=1.0),
        # two variables at 3001 locations (parsimonious bivariate kernel)
        dict(name="loglik_biv_n6002", kind="loglik", n=6002, kernel=2, dm="ed", dts=0, precision=0, beta=0.1, nu=0.5),
        # the 200 x 200 grid, nu = 1.5: the plain FP64 path at scale
        dict(name="loglik_n40000", kind="loglik", n=40000, kernel=0, dm="ed", dts=0, precision=0, beta=0.1, nu=1.5),
        # one step of a gradient fit of the 40 x 40 grid
        dict(name="grad_n1600", kind="grad", n=1600, kernel=0, dm="ed", dts=0, precision=0, beta=0.1, nu=0.5),
        # one step of a gradient fit with a nugget, N = 20000
        dict(name="grad_n20000_nugget", kind="grad", n=20000, kernel=1, dm="ed", dts=0, precision=0, beta=0.1, nu=1.0),
        # the reduced-precision objective at scale (FP64 tiles, INT8-sliced updates)
        dict(name="sliced_n70000", kind="loglik", n=70000, kernel=0, dm="ed", dts=0, precision=3, beta=0.05, nu=0.5),
        # a synthetic data set, z = L(theta) e, as the reference driver starts
        dict(name="synthetic_n10000", kind="synthetic", n=10000, kernel=0, dm="ed", dts=0, beta=0.1, nu=0.73),
        # regional fields of 500 to 6000 points with their own parameters, objective and gradient
        dict(name="batch_grad_48", kind="batch", fields=48, lo=500, hi=6000, kernel=0, grad=True),
        # kriging of 1000 held-out points from 19000
        dict(name="predict_19000_1000", kind="predict", n=19000, miss=1000, kernel=0, dm="ed", dts=0, beta=0.1,
             nu=0.5),
        # Fisher information, MLOE and MMOM after a fit of 4000 points
        dict(name="assess_n4000_400", kind="assess", n=4000, miss=400, kernel=0, dm="ed", dts=0, beta=0.1, nu=0.73),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loglik", "loglik", "loglik", "grad", "grad", "sliced", "synthetic", "batch", "predict", "assess"])
    if kind == "batch":
        lo = _log_int(rng, 500, 2000)
        return dict(kind="batch", fields=rng.randint(3, 44), lo=lo, hi=rng.randint(lo, 5900), kernel=rng.choice([0, 1]),
                    grad=rng.random() < 0.5)
    if kind == "sliced":
        return dict(kind="loglik", n=_log_int(rng, 4000, 66000), kernel=0, dm="ed", dts=0, precision=3,
                    beta=round(rng.uniform(0.03, 0.06), 4), nu=rng.choice([0.5, round(rng.uniform(0.3, 0.55), 3)]))
    dm = rng.choice(["ed", "ed", "ed", "gc"])
    # smooth fields come with a nugget, as in practice (without one Sigma is numerically singular)
    kernel = rng.choice([0, 0, 1, 2]) if kind == "loglik" else rng.choice([0, 1]) if kind == "grad" else 0
    nu = {0: rng.choice([0.5, 1.5, round(rng.uniform(0.3, 1.2), 3)]), 1: round(rng.uniform(0.4, 2.0), 3),
          2: round(rng.uniform(0.4, 0.9), 3)}[kernel]
    beta = round(rng.uniform(0.04, 0.15), 4) * (600.0 if dm == "gc" else 1.0)
    base = dict(kind=kind, kernel=kernel, dm=dm, dts=rng.choice([0, 0, 0, 320, 512]), beta=beta, nu=nu)
    if kind == "loglik":
        n = _log_int(rng, 400, 38000)
        return dict(base, n=n + (n & 1) if kernel == 2 else n, precision=0)
    if kind == "grad":
        return dict(base, n=_log_int(rng, 400, 19000), precision=0)
    if kind == "synthetic":
        return dict(base, n=_log_int(rng, 400, 18000))
    if kind == "predict":
        return dict(base, n=_log_int(rng, 900, 18500), miss=_log_int(rng, 30, 1000))
    return dict(base, n=_log_int(rng, 500, 3900), miss=_log_int(rng, 30, 400))


# ---- inputs -------------------------------------------------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _spread(v):
    """The low 16 bits of each value, spread to the even bit positions."""
    v = v.astype(np.uint64)
    for shift, mask in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << np.uint64(shift))) & np.uint64(mask)
    return v


def _morton(x, y):
    q = lambda a: np.clip((a * 65536.0).astype(np.int64), 0, 65535)  # noqa: E731
    o = np.argsort(_spread(q(x)) | (_spread(q(y)) << np.uint64(1)), kind="stable")
    return x[o], y[o]


def _grid(n, rng):
    """n points of a jittered grid of the unit square, Morton order."""
    m = math.isqrt(n - 1) + 1
    i = rng.permutation(m * m)[:n]
    x = (i // m + 0.5 + rng.uniform(-0.4, 0.4, n)) / m
    y = (i % m + 0.5 + rng.uniform(-0.4, 0.4, n)) / m
    return _morton(x, y)


def _density(w2, beta, nu):
    """Spectral density of the unit-variance Matern field in the plane."""
    return nu / math.pi * beta * beta * (1.0 + beta * beta * w2) ** -(nu + 1.0)


def _waves(x, y, theta, kernel, rng, count=2048):
    """Observations at the plane points (x, y): random plane waves with the model's spectral density."""
    if kernel == 2:
        s1, s2, beta, nu1, nu2, rho = theta
    else:
        s1, beta, nu1 = theta[:3]
        s2, nu2, rho = s1, nu1, 0.0
    nu = np.where(np.arange(count) % 2 == 0, nu1, nu2)
    w = rng.standard_normal((2, count)) / (beta * np.sqrt(2.0 * rng.gamma(nu)))
    w2, phase = (w * w).sum(axis=0), rng.uniform(0.0, 2.0 * math.pi, count)
    f1, f2 = _density(w2, beta, nu1), _density(w2, beta, nu2)
    g = 0.5 * (f1 + f2)
    a = rng.standard_normal((2, count))
    amp = math.sqrt(2.0 / count)
    dev = _device()
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    c = torch.cos(t(x)[:, None] * t(w[0]) + t(y)[:, None] * t(w[1]) + t(phase))
    z1 = c @ t(np.sqrt(s1 * f1 / g) * a[0] * amp)
    if kernel != 2:
        z = z1.cpu().numpy()
        return z + math.sqrt(theta[3]) * rng.standard_normal(x.size) if kernel == 1 else z
    # cross-spectrum rho sqrt(f1 f2): coherence below one, so its 2 x 2 factor exists at every frequency
    f12 = rho * math.sqrt(nu1 * nu2) / (0.5 * (nu1 + nu2)) * _density(w2, beta, 0.5 * (nu1 + nu2))
    l21 = f12 * math.sqrt(s1 * s2) / np.sqrt(s1 * f1 * g)
    l22 = np.sqrt(np.maximum(s2 * f2 / g - l21 * l21, 0.0))
    z2 = c @ t((l21 * a[0] + l22 * a[1]) * amp)
    return torch.stack([z1, z2], dim=1).reshape(-1).cpu().numpy()


def _theta(case, rng):
    move = lambda v: v * float(np.exp(rng.uniform(-0.04, 0.04)))  # noqa: E731
    # closed-form orders stay on their value, as in a fit with the smoothness held
    nu = case["nu"] if case["nu"] in (0.5, 1.5, 2.5) else move(case["nu"])
    if case["kernel"] == 2:
        return [move(1.0), move(2.0), move(case["beta"]), nu, nu + 0.6, 0.4]
    theta = [move(1.0), move(case["beta"]), nu]
    return theta + [move(0.01)] if case["kernel"] == 1 else theta


def _split(a, b, n, rng):
    i = rng.permutation(a.shape[0])
    m, o = np.sort(i[n:]), np.sort(i[:n])
    return a[m], b[m], a[o], b[o], m, o


def inputs(case, seed):
    """Host arrays of one case: what a user's program has read from its files."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        d = dict(x=[], y=[], z=[], theta=[])
        for _ in range(case["fields"]):
            n = int(rng.integers(case["lo"], case["hi"], endpoint=True))
            # the smooth fields have a nugget: without one Sigma would be numerically singular
            theta = [rng.uniform(0.5, 2.0), rng.uniform(0.02, 0.3), rng.uniform(0.3, 2.5 if case["kernel"] else 1.0)]
            if case["kernel"]:
                theta.append(rng.uniform(0.005, 0.05))
            x, y = _morton(rng.uniform(size=n), rng.uniform(size=n))
            d["x"].append(x)
            d["y"].append(y)
            d["z"].append(_waves(x, y, theta, case["kernel"], rng, 512))
            d["theta"].append(theta)
        d["theta"] = np.array(d["theta"])
        return d
    kernel = case["kernel"]
    miss = case.get("miss", 0)
    nloc = (case["n"] + miss) // (2 if kernel == 2 else 1)
    px, py = _grid(nloc, rng)
    theta = _theta(case, rng)
    if case["dm"] == "gc":  # a region of about 5.4 x 5.4 degrees around 40 N, 100 W
        x, y = 37.3 + 5.4 * px, -102.7 + 5.4 * py
        rad = math.pi / 180.0 * EARTH_KM
        px, py = (x - 40.0) * rad, (y + 100.0) * rad * math.cos(math.radians(40.0))
    else:
        x, y = px, py
    if case["kind"] == "synthetic":
        return dict(x=x, y=y, theta=theta, e=rng.standard_normal(nloc))
    d = dict(x=x, y=y, z=_waves(px, py, theta, kernel, rng), theta=theta)
    if miss:
        d["xm"], d["ym"], d["xo"], d["yo"], m, o = _split(x, y, case["n"], rng)
        d["zm"], d["zo"] = d["z"][m], d["z"][o]
        d["est"] = [theta[0] * 1.1, theta[1] * 0.9, theta[2] * 1.05]
    return d


class _State:
    """A case's inputs and the handle a program keeps; the handle is given back with the state."""

    def __init__(self, case, data):
        self.case, self.data, self.handle = case, data, None

    def __del__(self):
        if self.handle is not None:
            self.handle.close()


def prepare(case, seed):
    d = inputs(case, seed)
    s = _State(case, d)
    if _device() == "cuda":
        torch.cuda.empty_cache()  # the library allocates its own device memory
    if case["kind"] == "batch":
        s.handle = xg.Batch(d["x"], d["y"], d["z"], kernel=case["kernel"])
        return s
    x, y = (d["xo"], d["yo"]) if case["kind"] == "assess" else (d["x"], d["y"])
    s.handle = xg.Session(x, y, kernel=case["kernel"], dm=case["dm"], dts=case["dts"])
    if case["kind"] in ("loglik", "grad"):
        s.handle.set_data(z=d["z"])
        if case["precision"] == 3:
            s.handle.set_sliced()
            s.handle.data.precision = 3
    return s


def run(s):
    d, h, kind = s.data, s.handle, s.case["kind"]
    if kind == "loglik":
        return np.array([h.loglik(d["theta"])])
    if kind == "grad":
        ll, g = h.loglik(d["theta"], grad=True)
        return {"loglik": np.array([ll]), "grad": g}
    if kind == "batch":
        if s.case["grad"]:
            ll, g = h.loglik(d["theta"], grad=True)
            return {"loglik": ll, "grad": g}
        return {"loglik": h.loglik(d["theta"])}
    if kind == "synthetic":
        h.zvg(d["theta"], d["e"])
        return h.z()
    if kind == "predict":
        mse, zmiss = h.predict(d["theta"], d["xm"], d["ym"], d["xo"], d["yo"], d["zo"], d["zm"])
        return {"mse": np.array([mse]), "zmiss": zmiss}
    F, Finv = h.fisher(d["theta"])
    mloe, mmom, terms, _ = xg.mloe_mmom_host(d["xm"], d["ym"], d["xo"], d["yo"], d["theta"], d["est"],
                                             kernel=s.case["kernel"], metric=1 if s.case["dm"] == "gc" else 0)
    return {"fisher": F, "fisher_inv": Finv, "mloe": np.array([mloe]), "mmom": np.array([mmom]), "terms": terms}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        mean3 = (case["hi"] ** 4 - case["lo"] ** 4) / (4.0 * max(1, case["hi"] - case["lo"])) \
            if case["hi"] > case["lo"] else float(case["hi"]) ** 3
        points = case["fields"] * 0.5 * (case["lo"] + case["hi"])
        return {"bytes": 24.0 * points + 56.0 * case["fields"],
                "flops": case["fields"] * mean3 * (1.0 if case["grad"] else 1.0 / 3.0)}
    n = float(case["n"])
    if kind == "loglik":
        return {"bytes": 24.0 * n + 32.0, "flops": n ** 3 / 3.0}
    if kind == "synthetic":
        return {"bytes": 32.0 * n, "flops": n ** 3 / 3.0 + n * n}
    if kind == "grad":  # the factor, its inverse and the inverse's product with itself
        return {"bytes": 24.0 * n + 64.0, "flops": n ** 3}
    m = float(case["miss"])
    if kind == "predict":
        return {"bytes": 24.0 * n + 32.0 * m, "flops": n ** 3 / 3.0 + 2.0 * n * m}
    # Sigma^-1 and its products with two derivatives; two factors, two solves and a product for the errors
    return {"bytes": 16.0 * (n + m) + 48.0 * m, "flops": 5.0 * n ** 3 + 2.0 * n ** 3 / 3.0 + 5.0 * m * n * n}


# ---- the same in 64 bits, from torch alone ------------------------------------------------------------------------


def _distance(x1, y1, x2, y2, dm):
    if dm == "gc":
        r = math.pi / 180.0
        u, v = torch.sin((x2 - x1) * r / 2), torch.sin((y2 - y1) * r / 2)
        return 2.0 * EARTH_KM * torch.asin(torch.sqrt(u * u + torch.cos(x1 * r) * torch.cos(x2 * r) * v * v))
    return torch.sqrt((x2 - x1) ** 2 + (y2 - y1) ** 2)


def _bessel(nu, r, derivatives):
    """e^r K_nu(r) by the trapezoidal rule on its integral over cosh (and, with derivatives, e^r K_{nu-1}
    and the derivative with respect to the order)."""
    h = torch.clamp(0.5 / torch.sqrt(r), max=0.15)
    k0, k1, kd = (torch.full_like(r, 0.5), torch.full_like(r, 0.5), torch.zeros_like(r)) if derivatives else \
        (torch.full_like(r, 0.5), None, None)
    for k in range(1, 400):
        t = k * h
        w = torch.exp(-2.0 * r * torch.sinh(0.5 * t) ** 2)
        k0 += w * torch.cosh(nu * t)
        if derivatives:
            k1 += w * torch.cosh((nu - 1.0) * t)
            kd += w * t * torch.sinh(nu * t)
        if k % 16 == 0 and float((w * torch.cosh((nu + 1.0) * t) / k0).max()) < 1e-19:
            break
    return (h * k0, h * k1, h * kd) if derivatives else h * k0


def _matern(d, sigma2, beta, nu, derivatives=False):
    """Matern covariance (and its derivatives with respect to beta and nu) at the distances d."""
    r = d / beta
    if not derivatives and nu in (0.5, 1.5, 2.5):
        p = {0.5: 1.0, 1.5: 1.0 + r, 2.5: 1.0 + r + r * r / 3.0}[nu]
        return sigma2 * p * torch.exp(-r)
    zero = r == 0.0
    r = torch.where(zero, torch.ones_like(r), r)
    con = sigma2 * 2.0 ** (1.0 - nu) / math.gamma(nu)
    f = con * torch.exp(nu * torch.log(r) - r)
    if not derivatives:
        return torch.where(zero, torch.full_like(r, sigma2), f * _bessel(nu, r, False))
    k, km1, kd = _bessel(nu, r, True)
    psi = float(torch.digamma(torch.tensor(nu, dtype=torch.float64)))
    c = f * k
    nil = torch.zeros_like(r)
    return (torch.where(zero, torch.full_like(r, sigma2), c), torch.where(zero, nil, f * r * km1 / beta),
            torch.where(zero, nil, c * (torch.log(r) - math.log(2.0) - psi) + f * kd))


def _cross(xr, yr, xc, yc, theta, dm, derivatives=False):
    """Covariance of the row and the column locations, by row blocks; with derivatives also d/dbeta, d/dnu."""
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=_device())  # noqa: E731
    xr, yr, xc, yc = t(xr), t(yr), t(xc), t(yc)
    out = [torch.empty(xr.numel(), xc.numel(), dtype=torch.float64, device=xr.device)
           for _ in range(3 if derivatives else 1)]
    step = max(1, (1 << 27) // xc.numel())
    for a in range(0, xr.numel(), step):
        d = _distance(xr[a:a + step, None], yr[a:a + step, None], xc[None], yc[None], dm)
        got = _matern(d, theta[0], theta[1], theta[2], derivatives)
        for o, g in zip(out, got if derivatives else (got,)):
            o[a:a + step] = g
    return out if derivatives else out[0]


def _covariance(x, y, theta, kernel, dm):
    if kernel == 2:
        s1, s2, beta, nu1, nu2, rho = theta
        nu12 = 0.5 * (nu1 + nu2)
        c12 = rho * math.sqrt(nu1 * nu2) / nu12 * math.sqrt(s1 * s2)
        n = x.size
        S = torch.empty(2 * n, 2 * n, dtype=torch.float64, device=_device())
        S[0::2, 0::2] = _cross(x, y, x, y, (s1, beta, nu1), dm)
        S[1::2, 1::2] = _cross(x, y, x, y, (s2, beta, nu2), dm)
        S[0::2, 1::2] = _cross(x, y, x, y, (c12, beta, nu12), dm)
        S[1::2, 0::2] = S[0::2, 1::2].T.clone()
        return S
    S = _cross(x, y, x, y, theta, dm)
    if kernel == 1:
        S.diagonal().add_(theta[3])
    return S


def _loglik(L, z):
    w = torch.linalg.solve_triangular(L, z[:, None], upper=False)
    return float(-0.5 * (w * w).sum() - torch.log(L.diagonal()).sum() - 0.5 * z.numel() * math.log(2.0 * math.pi))


def _loglik_grad(x, y, z, theta, kernel, dm):
    """Log-likelihood and gradient (sigma^2, beta, nu[, nugget])."""
    S, db, dn = _cross(x, y, x, y, theta, dm, True)
    ds = S / theta[0]
    if kernel == 1:
        S.diagonal().add_(theta[3])
    L = torch.linalg.cholesky(S)
    del S
    z = torch.as_tensor(z, dtype=torch.float64, device=L.device)
    ll = _loglik(L, z)
    inv = torch.cholesky_inverse(L)
    a = torch.cholesky_solve(z[:, None], L)[:, 0]
    g = []
    for D in (ds, db, dn):
        g.append(0.5 * float(a @ (D @ a)) - 0.5 * float((inv * D).sum()))
    if kernel == 1:
        g.append(0.5 * float(a @ a) - 0.5 * float(inv.diagonal().sum()))
    return ll, g


def _fisher(x, y, theta, dm):
    S, db, dn = _cross(x, y, x, y, theta, dm, True)
    L = torch.linalg.cholesky(S)
    M = [torch.cholesky_solve(D, L) for D in (S / theta[0], db, dn)]
    F = np.empty((3, 3))
    for j in range(3):
        for k in range(3):
            F[j, k] = 0.5 * float((M[j] * M[k].T).sum())
    return F


def _mloe_mmom(d, dm):
    t, a = d["theta"], d["est"]
    Lt, La = (torch.linalg.cholesky(_cross(d["xo"], d["yo"], d["xo"], d["yo"], p, dm)) for p in (t, a))
    kt, ka = (_cross(d["xo"], d["yo"], d["xm"], d["ym"], p, dm) for p in (t, a))
    wt, wa = torch.cholesky_solve(kt, Lt), torch.cholesky_solve(ka, La)
    e1 = (kt * wa).sum(0)
    x2 = t[0] - 2.0 * e1 + ((Lt.T @ wa) ** 2).sum(0)
    x3, x4 = t[0] - (kt * wt).sum(0), a[0] - (ka * wa).sum(0)
    terms = torch.stack([e1, x2, x3, x4, x2 / x3 - 1.0, x4 / x2 - 1.0], dim=1).cpu().numpy()
    return terms[:, 4].mean(), terms[:, 5].mean(), terms


def exact(case, seed):
    kind = case["kind"]
    if kind != "batch" and (case["n"] > 42000 or (kind == "grad" and case["n"] > 31000)):
        return None  # several dense copies of Sigma would no longer be quick
    d = inputs(case, seed)
    if kind == "batch":
        ll, g = [], []
        for x, y, z, theta in zip(d["x"], d["y"], d["z"], d["theta"]):
            a, b = _loglik_grad(x, y, z, list(theta), case["kernel"], "ed")
            ll.append(a)
            g.append(b)
        return {"loglik": np.array(ll), "grad": np.array(g)} if case["grad"] else {"loglik": np.array(ll)}
    dm, kernel = case["dm"], case["kernel"]
    if kind == "synthetic":
        L = torch.linalg.cholesky(_covariance(d["x"], d["y"], d["theta"], kernel, dm))
        return (L @ torch.as_tensor(d["e"], dtype=torch.float64, device=L.device)).cpu().numpy()
    if kind == "loglik":
        L = torch.linalg.cholesky(_covariance(d["x"], d["y"], d["theta"], kernel, dm))
        return np.array([_loglik(L, torch.as_tensor(d["z"], dtype=torch.float64, device=L.device))])
    if kind == "grad":
        ll, g = _loglik_grad(d["x"], d["y"], d["z"], d["theta"], kernel, dm)
        return {"loglik": np.array([ll]), "grad": np.array(g)}
    if kind == "predict":
        L = torch.linalg.cholesky(_cross(d["xo"], d["yo"], d["xo"], d["yo"], d["theta"], dm))
        a = torch.cholesky_solve(torch.as_tensor(d["zo"], dtype=torch.float64, device=L.device)[:, None], L)
        zmiss = (_cross(d["xm"], d["ym"], d["xo"], d["yo"], d["theta"], dm) @ a)[:, 0].cpu().numpy()
        return {"mse": np.array([np.mean((zmiss - d["zm"]) ** 2)]), "zmiss": zmiss}
    F = _fisher(d["xo"], d["yo"], d["theta"], dm)
    mloe, mmom, terms = _mloe_mmom(d, dm)
    return {"fisher": F, "fisher_inv": np.linalg.inv(F), "mloe": np.array([mloe]), "mmom": np.array([mmom]),
            "terms": terms}
