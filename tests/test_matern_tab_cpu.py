"""The piecewise polynomial tables (xg_matern_tab.cuh, host/device code
compiled with g++) of the covariance and of its three derivatives against the
direct forms, at both ends of the table, at interval edges and inside, and the
index outside the table.

Bar as in the GPU test of the covariance: the direct form rounds
(nu - 1/2) log r - r before its exponential, |.| 2^-53, and both forms carry
about 1e-14 of their own; for the order's derivative relative to the sum of its
terms' magnitudes."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "xg_matern_tab.cuh"
int main(int argc, char **argv)
{
    const double nu = atof(argv[1]), con = 1.3 / (pow(2, nu - 1) * tgamma(nu)), sigma2 = 1.3, beta = 0.1, dl = -1.1;
    const XgTemme tm = xg_temme_consts(nu);
    std::vector<double> T[4];
    for (auto &t : T) t.resize(XG_TAB_SIZE);
    for (int i = 0; i < XG_TAB_NINT; ++i) {
        double c, hw, f[4][XG_TAB_NC], g[3];
        xg_tab_interval(i, &c, &hw);
        for (int j = 0; j < XG_TAB_NC; ++j) {
            const double r = xg_tab_node(c, hw, j);
            f[0][j] = xg_tab_matern(r, nu, con, tm);
            xg_tab_matern_grad(r, nu, con, sigma2, beta, dl, g);
            for (int p = 0; p < 3; ++p) f[1 + p][j] = g[p];
        }
        for (int p = 0; p < 4; ++p) xg_tab_coefficients(f[p], hw, &T[p][i * XG_TAB_NC]);
    }
    double r;
    while (scanf("%lf", &r) == 1) {
        const unsigned i = xg_tab_index(r);
        double m, d[4], t[4] = {0, 0, 0, 0};
        d[0] = xg_matern_general(r, nu, con);
        xg_matern_grad(r, nu, con, sigma2, beta, dl, &m, d + 1, d + 2, d + 3);
        if (i < XG_TAB_NINT)
            for (int p = 0; p < 4; ++p) t[p] = xg_tab_poly(T[p].data(), i, r - xg_tab_centre(r)) * exp(-r);
        printf("%u", i);
        for (int p = 0; p < 4; ++p) printf(" %.17g %.17g", d[p], t[p]);
        printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    d = tmp_path_factory.mktemp("tab")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-I", os.path.join(ROOT, "exageostat_b200", "csrc"), str(d / "t.cpp"), "-o",
                    str(d / "t")], check=True)

    def run(nu, r):
        out = subprocess.run([str(d / "t"), repr(nu)], input="\n".join(float(v).hex() for v in r), text=True, check=True,
                             capture_output=True).stdout
        a = np.array([line.split() for line in out.splitlines()], dtype=float)
        return a[:, 0].astype(np.int64), a[:, 1::2], a[:, 2::2]

    return run


@pytest.mark.parametrize("nu", [0.01, 0.5, 0.73, 1.0, 2.2, 3.7, 5.0])
def test_tables_match_the_direct_forms(tables, nu):
    rng = np.random.default_rng(3)
    edges = 2.0 ** rng.integers(-16, 9, 60) * (1 + rng.integers(0, 16, 60) / 16)
    r = np.concatenate([[2.0 ** -16, np.nextafter(2.0 ** -16, 1), np.nextafter(512.0, 0), 511.0, 2.0, np.nextafter(2.0, 3)],
                        edges, np.nextafter(edges[edges > 2.0 ** -16], 0), np.exp(rng.uniform(np.log(2.0 ** -16), np.log(512), 400))])
    i, direct, table = tables(nu, r)
    assert i.min() >= 0 and i.max() < 400
    tol = 2e-14 + 2.3e-16 * (r + (nu + 0.5) * np.abs(np.log(r)))
    for p in range(3):
        assert np.all(np.abs(table[:, p] - direct[:, p]) <= tol * np.abs(direct[:, p])), p
    scale = 2.0 * direct[:, 0] * (np.abs(np.log(r)) + 1.1) + np.abs(direct[:, 3])
    assert np.all(np.abs(table[:, 3] - direct[:, 3]) <= tol * scale)


def test_outside_the_table(tables):
    i, _, _ = tables(1.0, [np.nextafter(2.0 ** -16, 0), 1e-300, 512.0, 1e300, np.inf])
    assert np.all((i < 0) | (i >= 400))
    assert i.size == 5
