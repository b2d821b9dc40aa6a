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
