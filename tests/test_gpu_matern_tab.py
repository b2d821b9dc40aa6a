"""Covariance elements from the piecewise polynomial tables (fields of 64
locations and more, general order) against the direct evaluation of the same
elements, over the whole table and both of its ends.

Bar, per element: the direct form rounds (nu - 1/2) log r - r before its
exponential, |.| 2^-53, and both forms carry about 1e-14 of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [0.01, 0.3, 1.0, 2.2, 5.0])
@pytest.mark.parametrize("beta", [0.0015, 0.1, 40.0])
def test_table_elements_match_the_direct_form(gpu, nu, beta):
    rng = np.random.default_rng(11)
    n = 1030
    x, y = rng.uniform(size=n), rng.uniform(size=n)
    # neighbours at 1e-9 .. 1e-3 of the unit square, below the table's first interval for beta = 40
    x[1:200] = x[0] + 10.0 ** rng.uniform(-9, -3, 199)
    y[1:200] = y[0]
    theta = [1.3, beta, nu]
    C = gpu.covariance_dense(x, y, theta, ts=256)
    i, j = np.tril_indices(n, -1)
    direct = gpu.matern_pairs(x[i], y[i], x[j], y[j], theta)
    r = np.hypot(x[i] - x[j], y[i] - y[j]) / beta
    tol = 2e-14 + 2.3e-16 * (r + (nu + 0.5) * np.abs(np.log(np.maximum(r, 1e-300))))
    big = direct > 1e-290
    err = np.abs(C[i, j][big] - direct[big]) / direct[big]
    assert np.all(err <= tol[big]), (err.max(), r[big][np.argmax(err / tol[big])])
    assert np.all(np.abs(C[i, j][~big]) <= 1.1e-290)
    assert np.array_equal(np.diag(C), np.full(n, 1.3))


@pytest.mark.parametrize("e", [-960, -900, -700, 700, 900, 1000])
def test_variances_at_the_ends_of_the_double_range(gpu, e):
    """Powers of two as variances scale the covariance exactly: elements as
    the direct form gives them, near neighbours included, and the gradient of
    sigma^2 = 1 with the observations scaled, to 1e-9 of its largest entry."""
    rng = np.random.default_rng(13)
    n, s2 = 300, 2.0 ** e
    x, y, z = rng.uniform(size=n), rng.uniform(size=n), rng.standard_normal(n)
    x[1:100] = x[0] + 10.0 ** rng.uniform(-7, -3, 99)
    y[1:100] = y[0]
    i, j = np.tril_indices(n, -1)
    r = np.hypot(x[i] - x[j], y[i] - y[j]) / 0.1
    for nu in (0.3, 1.0, 2.2):
        C = gpu.covariance_dense(x, y, [s2, 0.1, nu], ts=256)[i, j]
        direct = gpu.matern_pairs(x[i], y[i], x[j], y[j], [s2, 0.1, nu])
        tol = 2e-14 + 2.3e-16 * (r + (nu + 0.5) * np.abs(np.log(np.maximum(r, 1e-300))))
        big = direct > 1e-290
        assert np.all(np.isfinite(C)) and np.all(np.abs(C - direct)[big] <= (tol * direct)[big])
        g = []
        for s in (1.0, s2):
            theta = [s, 0.1, nu, 0.25 * s]
            with gpu.Session(x, y, kernel=1) as h:
                h.set_data(z=z * np.sqrt(s))
                g.append(h.loglik(theta, grad=True)[1] * [s, 1.0, 1.0, s])
            with gpu.Batch([x], [y], [z * np.sqrt(s)], kernel=1) as b:
                g.append(b.loglik([theta], grad=True)[1][0] * [s, 1.0, 1.0, s])
        for v in g[1:]:
            assert np.abs(v - g[0]).max() <= 1e-9 * np.abs(g[0]).max(), (nu, g)


@pytest.mark.parametrize("beta", [0.0015, 0.1, 40.0])
@pytest.mark.parametrize("kernel", [2, 3])
def test_bivariate_table_elements(gpu, kernel, beta):
    """The three tables of a bivariate field, each block of the covariance
    against the direct elements of its own constants; bar as above."""
    from math import gamma, sqrt

    rng = np.random.default_rng(17)
    n = 520
    x, y = rng.uniform(size=n), rng.uniform(size=n)
    x[1:150] = x[0] + 10.0 ** rng.uniform(-9, -3, 149)
    y[1:150] = y[0]
    nu1, nu2 = 0.6, 1.7
    nu12 = 0.5 * (nu1 + nu2)
    if kernel == 2:
        theta = [1.3, 0.7, beta, nu1, nu2, -0.4]
        c12 = -0.4 * sqrt(gamma(nu1 + 1) * gamma(nu2 + 1) / (gamma(nu1) * gamma(nu2))) * gamma(nu12) / gamma(nu12 + 1)
        blocks = {(0, 0): [1.3, beta, nu1], (1, 1): [0.7, beta, nu2], (0, 1): [c12 * sqrt(1.3 * 0.7), beta, nu12]}
    else:  # scales a_1, a_2; theta_4 = 0: nu_12 is the mean order; theta_7 = 0
        a1, a2 = beta, 1.5 * beta
        theta = [a1, a2, 0.3, 0.2, nu1, nu2, 0.0, 0.0, 1.2, 0.8, 0.5]
        a12 = (0.5 * (a1 ** -2 + a2 ** -2) + 0.3 * (1 - 0.2)) ** -0.5
        rho = 1.2 * 0.8 * 0.5 * a12 ** (nu1 + nu2) * gamma(nu12 + 1) * gamma(nu12) / gamma(nu12 + 1)
        blocks = {(0, 0): [1.2 ** 2 * a1 ** (2 * nu1) * gamma(nu1), a1, nu1],
                  (1, 1): [0.8 ** 2 * a2 ** (2 * nu2) * gamma(nu2), a2, nu2], (0, 1): [rho, a12, nu12]}
    C = gpu.covariance_dense(x, y, theta, kernel=kernel, ts=256)
    C = np.tril(C) + np.tril(C, -1).T
    i, j = np.tril_indices(n, -1)
    for (a, b), (s2, scale, nu) in blocks.items():
        direct = np.sign(s2) * gpu.matern_pairs(x[i], y[i], x[j], y[j], [abs(s2), scale, nu])
        got = C[a::2, b::2][i, j]
        r = np.hypot(x[i] - x[j], y[i] - y[j]) / scale
        tol = 2e-14 + 2.3e-16 * (r + (nu + 0.5) * np.abs(np.log(np.maximum(r, 1e-300))))
        big = np.abs(direct) > 1e-290
        err = np.abs(got - direct)[big] / np.abs(direct)[big]
        assert np.all(err <= tol[big]), (a, b, err.max(), r[big][np.argmax(err / tol[big])])
        assert np.all(np.abs(got[~big]) <= 1.1e-290)
