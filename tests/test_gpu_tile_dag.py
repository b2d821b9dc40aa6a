"""The one-launch tile factorisation against the oracle at the edges of its
128-blocks: a single partial block, exact blocks, one row past a block, a
stored tile of several blocks with whole blocks of padding, and the first
failing pivot.

Bars: l and kriging as in the parity tests (1e-10 and 1e-9 relative); z = L e
to 1e-11 of its norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THETA = [1.0, 0.1, 0.5]


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 127, 128, 129, 255, 257, 385, 513, 1153])
@pytest.mark.parametrize("ts", [128, 384, 512])
def test_loglik_and_zvg_at_block_edges(gpu, ora, n, ts):
    x, y = ora.generate_xy_loc(n, 2)
    e = ora.dlarnv(3, n)
    with gpu.Session(x, y, dts=ts) as s:
        s.zvg(THETA, e)
        z = s.z()
        zr = ora.dzvg(x, y, THETA, e)
        assert np.linalg.norm(z - zr) <= 1e-11 * np.linalg.norm(zr)
        for _ in range(2):  # a second evaluation starts from clean flags
            assert s.loglik(THETA) == pytest.approx(ora.dmle(x, y, z, THETA)[0], rel=1e-10)


@pytest.mark.parametrize("dup", [3, 130, 300])
def test_failing_pivot(gpu, ora, dup):
    """A NaN location fails at its own pivot; put right, the same handle
    evaluates as before."""
    n = 301
    x, y = ora.generate_xy_loc(n, 4)
    e = ora.dlarnv(5, n)
    z = ora.dzvg(x, y, THETA, e)
    xd, yd = x.copy(), y.copy()
    xd[dup], yd[dup] = np.nan, np.nan
    with gpu.Session(x, y, dts=128) as s:
        s.set_data(z=z)
        ll = s.loglik(THETA)
        s.set_data(x=xd, y=yd)
        with pytest.raises(gpu.XgError) as err:
            s.loglik(THETA)
        assert err.value.code == gpu.XG_ERR_NOT_SPD and "pivot %d)" % (dup + 1) in str(err.value)
        s.set_data(x=x, y=y)
        assert s.loglik(THETA) == ll


def test_wide_pivot_range(gpu, ora):
    """Variances far from one: pivots outside the fast reciprocal root's range
    take the general form."""
    n = 200
    x, y = ora.generate_xy_loc(n, 6)
    for s2 in (1e-295, 1e-200, 1e200, 1e295):
        theta = [s2, 0.1, 0.5]
        z = ora.dzvg(x, y, theta, ora.dlarnv(7, n))
        assert gpu.dmle_host(x, y, z, theta, ts=128)[1] == pytest.approx(ora.dmle(x, y, z, theta)[1], rel=1e-10)


@pytest.mark.parametrize("n", [2, 127, 129, 257, 513])
@pytest.mark.parametrize("ts", [128, 384])
def test_gradient_at_block_edges(gpu, ora, n, ts):
    """The inverse and product launch and the backward solve through the
    gradient, against the dense adjoint on the oracle's derivative tiles (1e-9
    of its largest entry, the bar of the batched gradients); batched likewise."""
    x, y = ora.generate_xy_loc(n, 8)
    z = ora.dzvg(x, y, THETA, ora.dlarnv(9, n))
    S = ora.covariance_full(x, y, THETA)
    inv = np.linalg.inv(S)
    a = inv @ z
    ref = []
    for p in range(3):
        D = ora.dcmg_deriv(n, n, 0, 0, x, y, x, y, THETA, p, 0)
        ref.append(0.5 * a @ D @ a - 0.5 * np.sum(inv * D))
    with gpu.Session(x, y, dts=ts) as s:
        s.set_data(z=z)
        _, g = s.loglik(THETA, grad=True)
    assert np.abs(g - ref).max() <= 1e-9 * max(1.0, np.abs(ref).max())
    with gpu.Batch([x, x[:1], x], [y, y[:1], y], [z, z[:1], z], ts=ts) as b:
        _, gb = b.loglik([THETA] * 3, grad=True)
    for f in (0, 2):
        assert np.abs(gb[f] - ref).max() <= 1e-9 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("ts", [128, 256])
def test_failing_pivot_of_every_panel(gpu, ora, ts):
    """A NaN location in each 16-wide panel of the first and of a later block:
    the pivot that fails, from the tile DAG, the per-step launches and a
    batch; all three evaluate again afterwards."""
    n = 301
    x, y = ora.generate_xy_loc(n, 4)
    z = ora.dzvg(x, y, THETA, ora.dlarnv(5, n))
    with gpu.Session(x, y, dts=ts) as s:
        s.set_data(z=z)
        ref = s.loglik(THETA)
        for bad in [16 * p + (3 * p) % 16 for p in range(8)] + [128 + 16 * p + 15 for p in range(8)]:
            xb = x.copy()
            xb[bad] = np.nan
            s.set_data(x=xb)
            for profiled in (False, True):
                s.set_profiling(profiled)
                with pytest.raises(gpu.XgError) as err:
                    s.loglik(THETA)
                assert err.value.code == gpu.XG_ERR_NOT_SPD and "pivot %d)" % (bad + 1) in str(err.value)
            s.set_profiling(False)
            with gpu.Batch([x, xb, x], [y, y, y], [z, z, z], ts=ts) as b:
                ll = b.loglik([THETA] * 3)
                assert ll[1] == -np.inf and ll[0] == ll[2] == pytest.approx(ref, rel=1e-12)
        s.set_data(x=x)
        assert s.loglik(THETA) == ref


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("n,ts", [(1, 128), (127, 128), (129, 128), (385, 128), (257, 256), (513, 256), (700, 384),
                                  (1153, 384), (513, 512), (1300, 512)])
def test_per_step_factorisation(gpu, ora, n, ts, kernel):
    """The per-step launches (a profiled evaluation runs them at any size) and
    what reads their factor and inverted diagonal blocks afterwards: l against
    the oracle to 1e-10, l and the gradient against the one-launch
    factorisation to 1e-10 and 1e-9 of its largest entry."""
    theta = [1.0, 0.1, 0.73] + [0.05] * kernel
    x, y = ora.generate_xy_loc(n, 8)
    z = ora.dzvg(x, y, theta, ora.dlarnv(9, n), kernel)
    ref = ora.dmle(x, y, z, theta, kernel)[0]
    with gpu.Session(x, y, kernel=kernel, dts=ts) as s:
        s.set_data(z=z)
        l0, g0 = s.loglik(theta, grad=True)
        s.set_profiling(True)
        assert s.loglik(theta) == pytest.approx(ref, rel=1e-10)
        l1, g1 = s.loglik(theta, grad=True)
        s.set_profiling(False)
        assert l1 == pytest.approx(l0, rel=1e-10)
        assert np.abs(g1 - g0).max() <= 1e-9 * np.abs(g0).max()
        assert s.loglik(theta) == l0


def test_per_step_factorisation_past_the_dataflow_sizes(gpu, ora):
    """N = 22145 at tiles of 128 takes the per-step launches without a profile:
    l and gradient against the seven-digit path, the bars of its own test."""
    n, theta = 22145, [1.0, 0.1, 0.5]
    x, y = ora.generate_xy_loc(n, 3)
    z = np.random.default_rng(1).standard_normal(n)
    got = []
    for ts in (512, 128):
        with gpu.Session(x, y, dts=ts) as s:
            s.set_data(z=z)
            got.append(s.loglik(theta, grad=True))
    assert got[1][0] == pytest.approx(got[0][0], rel=2e-12)
    assert np.abs(got[1][1] - got[0][1]).max() <= 1e-9 * np.abs(got[0][1]).max()
