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
