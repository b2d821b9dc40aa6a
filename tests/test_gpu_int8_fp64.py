"""Large FP64 evaluations, whose updates run as seven-digit integer products,
against the DMMA path (tile 128, which keeps it) on the same data: tiles
filled exactly, one row past, a nearly empty last tile.

Bars: l 2e-12 relative, ten times what a CPU model of the tiled factorisation
gives for the product as it should be (n = 2048, order 1.5, condition 2e6:
2e-13 from FP64).  One digit pair of level 5 counted twice or lost moves l by
9e-10 there, but by 6e-13 only at order 0.5 and condition 2e3: it is the
smoother orders that hold the pairs (at order 1.5 and N = 8065 the digits are
1e-13 from an extended-precision refinement, the DMMA path 1.3e-12).  The gradient 1e-9 of its largest entry;
kriging 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ts,theta,kernel", [
    (6656, 512, [1.0, 0.1, 0.5], 0),
    (6657, 512, [1.3, 0.07, 0.73], 0),
    (7041, 512, [1.0, 0.1, 1.0, 0.01], 1),
    (8065, 384, [0.8, 0.06, 1.5], 0),
    (11265, 256, [1.0, 0.1, 0.5], 0),
    (6500, 256, [1.3, 0.07, 0.73], 0),
    (6913, 384, [0.8, 0.06, 1.0], 0),
    (8192, 256, [1.0, 0.1, 1.0, 0.01], 1),
])
def test_matches_the_dmma_path(gpu, ora, n, ts, theta, kernel):
    x, y = ora.generate_xy_loc(n, 3)
    z = np.random.default_rng(1).standard_normal(n)
    got = {}
    for t in (ts, 128):
        with gpu.Session(x, y, kernel=kernel, dts=t) as s:
            s.set_data(z=z)
            ll = s.loglik(theta)
            ll2, g = s.loglik(theta, grad=True)
            assert ll2 == ll
            got[t] = (ll, g)
    assert got[ts][0] == pytest.approx(got[128][0], rel=2e-12)
    assert np.abs(got[ts][1] - got[128][1]).max() <= 1e-9 * np.abs(got[128][1]).max()


def test_kriging_and_synthetic_data(gpu, ora):
    n, m, theta = 6700, 50, [1.0, 0.1, 0.5]
    x, y = ora.generate_xy_loc(n + m, 5)
    e = ora.dlarnv(6, n + m)
    out = {}
    for t in (512, 128):
        with gpu.Session(x, y, dts=t) as s:
            s.zvg(theta, e)
            z = s.z()
            out[t] = (z, s.predict(theta, x[:m], y[:m], x[m:], y[m:], out[512][0][m:] if t == 128 else z[m:])[1])
    assert np.linalg.norm(out[512][0] - out[128][0]) <= 1e-11 * np.linalg.norm(out[128][0])
    assert np.linalg.norm(out[512][1] - out[128][1]) <= 1e-11 * np.linalg.norm(out[128][1])


def test_a_failing_pivot_is_reported(gpu, ora):
    n = 6657
    x, y = ora.generate_xy_loc(n, 3)
    bad = x.copy()
    bad[5000] = np.nan
    with gpu.Session(x, y, dts=512) as s:
        s.set_data(z=np.ones(n))
        ll = s.loglik([1.0, 0.1, 0.5])
        s.set_data(x=bad)
        with pytest.raises(gpu.XgError) as err:
            s.loglik([1.0, 0.1, 0.5])
        assert err.value.code == gpu.XG_ERR_NOT_SPD and "pivot 5001)" in str(err.value)
        s.set_data(x=x)
        assert s.loglik([1.0, 0.1, 0.5]) == ll


def test_the_digit_planes_are_given_back(gpu, ora):
    """Closed sessions and finished kriging calls leave the device's free
    memory where it was; the planes of one N = 7000 factor are 0.2 GB."""
    import torch

    n, m, theta = 7000, 50, [1.0, 0.1, 0.5]
    x, y = ora.generate_xy_loc(n + m, 3)
    z = np.random.default_rng(1).standard_normal(n + m)
    free = []
    for _ in range(3):
        with gpu.Session(x[m:], y[m:], dts=512) as s:
            s.set_data(z=z[m:])
            s.loglik(theta, grad=True)
            s.predict(theta, x[:m], y[:m], x[m:], y[m:], z[m:])
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[2] < 64 << 20, free


class _Full:
    """The device's memory but for `leave` bytes, held by another library."""

    def __init__(self, leave):
        import torch

        torch.cuda.empty_cache()
        self.t = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        import torch

        del self.t
        torch.cuda.empty_cache()


def test_the_path_does_not_depend_on_the_order_of_calls(gpu, ora):
    """Objective, gradient, objective, or the gradient first: the same values;
    and a session that found no memory for the planes takes them, with the
    same values again, once there is some."""
    import torch

    n, theta = 6657, [1.3, 0.07, 0.73]
    x, y = ora.generate_xy_loc(n, 3)
    z = np.random.default_rng(1).standard_normal(n)
    with gpu.Session(x, y, dts=512) as s:
        s.set_data(z=z)
        ref = s.loglik(theta)
        ll, gref = s.loglik(theta, grad=True)
        assert ll == ref == s.loglik(theta)
    with gpu.Session(x, y, dts=512) as s:
        s.set_data(z=z)
        ll, g = s.loglik(theta, grad=True)
        assert ll == ref and np.array_equal(g, gref) and s.loglik(theta) == ref
    with _Full(600 << 20):  # 0.22 GB of tiles, 0.19 of planes
        s = gpu.Session(x, y, dts=512)
        s.set_data(z=z)
        free = torch.cuda.mem_get_info()[0]
        assert s.loglik(theta) == pytest.approx(ref, rel=2e-12)
        assert free - torch.cuda.mem_get_info()[0] < 16 << 20
    ll, g = s.loglik(theta, grad=True)
    s.close()
    assert ll == ref and np.array_equal(g, gref)


@pytest.mark.parametrize("what", ["session", "batch", "kriging", "assessment", "mixed"])
def test_idle_planes_make_room_for_others(gpu, ora, what):
    """An allocation that the device refuses while an idle session holds its
    planes (0.31 GB) gets their memory; the session evaluates without them,
    and with them again when there is room."""
    n, m, theta = 9000, 50, [1.0, 0.1, 0.5]
    x, y = ora.generate_xy_loc(n + m, 3)
    z = np.random.default_rng(1).standard_normal(n + m)
    k = 6000

    def other(s):
        if what == "session":
            with gpu.Session(x[:k], y[:k], dts=256) as t:
                t.set_data(z=z[:k])
                return t.loglik(theta)
        if what == "batch":
            with gpu.Batch([x[:4000], x[4000:8000]], [y[:4000], y[4000:8000]], [z[:4000], z[4000:8000]]) as b:
                return b.loglik([theta] * 2)
        if what == "kriging":
            return s.predict(theta, x[n:], y[n:], x[:k], y[:k], z[:k])[1]
        if what == "mixed":
            with gpu.Session(x[:4096], y[:4096], dts=256) as t:
                t.set_data(z=z[:4096])
                t.set_mixed(band=12)
                return t.loglik(theta)
        return gpu.mloe_mmom_host(x[n:], y[n:], x[:4000], y[:4000], theta, [1.1, 0.09, 0.52])[2]

    with gpu.Session(x[:n], y[:n], dts=512) as s:
        s.set_data(z=z[:n])
        ref = s.loglik(theta)
        want = other(s)
        assert s.loglik(theta) == ref
        with _Full(100 << 20):
            assert np.array_equal(other(s), want)
            assert s.loglik(theta) == pytest.approx(ref, rel=2e-12)
        assert s.loglik(theta) == ref


@pytest.mark.parametrize("e", [-1000, -700, 700, 1000])
def test_variances_at_the_ends_of_the_double_range(gpu, ora, e):
    """Powers of two as variances: l and the gradient of sigma^2 = 1 with the
    observations scaled, within the file's bars."""
    n, s2 = 6657, 2.0 ** e
    x, y = ora.generate_xy_loc(n, 3)
    z = np.random.default_rng(1).standard_normal(n)
    got = []
    for s in (1.0, s2):
        with gpu.Session(x, y, dts=512) as h:
            h.set_data(z=z * np.sqrt(s))
            ll, g = h.loglik([s, 0.1, 0.5], grad=True)
        got.append((ll + 0.5 * n * np.log(s), g * [s, 1.0, 1.0]))
    assert got[1][0] == pytest.approx(got[0][0], rel=2e-12)
    assert np.abs(got[1][1] - got[0][1]).max() <= 1e-9 * np.abs(got[0][1]).max()


@pytest.mark.parametrize("kernel,theta,ts", [
    (2, [1.0, 2.0, 0.03, 0.5, 1.1, 0.4], 512),
    (2, [1e-6, 3.0, 0.03, 0.5, 0.7, -0.3], 256),
    (3, [0.08, 0.12, 1.0, 0.2, 0.5, 1.0, 0.2, 0.8, 1.24479, 4.41137, -0.4], 512),
])
def test_bivariate_fields(gpu, ora, kernel, theta, ts):
    """Interleaved rows of two variances and orders, against the DMMA path
    (kernel 3, whose ranges are three times longer, to the 1e-10 of its own
    test)."""
    n = 6658
    x, y = ora.generate_xy_loc(n // 2, 3)
    z = np.random.default_rng(1).standard_normal(n)
    z[0::2] *= np.sqrt(theta[0]) if kernel == 2 else 1.0
    got = []
    for t in (ts, 128):
        with gpu.Session(x, y, kernel=kernel, dts=t) as s:
            s.set_data(z=z)
            got.append(s.loglik(theta))
    assert got[0] == pytest.approx(got[1], rel=2e-12 if kernel == 2 else 1e-10)


@pytest.mark.parametrize("kernel", [0, 1])
def test_assessment(gpu, ora, kernel):
    """Fisher matrix and MLOE / MMOM from seven-digit factors against tiles of
    128, the bars of their own tests."""
    n, m = 6657, 130
    x, y = ora.generate_xy_loc(n + m, 3)
    truth, est = [1.3, 0.07, 0.73] + [0.05] * kernel, [1.1, 0.08, 0.7] + [0.04] * kernel
    F = [gpu.fisher_host(x[m:], y[m:], truth, kernel=kernel, ts=t) for t in (512, 128)]
    scale = np.sqrt(np.outer(np.diag(F[1]), np.diag(F[1])))
    assert (np.abs(F[0] - F[1]) / scale).max() < 1e-8
    a, b = [gpu.mloe_mmom_host(x[:m], y[:m], x[m:], y[m:], truth, est, kernel=kernel, ts=t) for t in (512, 128)]
    assert np.abs(a[2][:, :4] - b[2][:, :4]).max() < 1e-9 * truth[0]
    assert abs(a[0] - b[0]) < 1e-8 and abs(a[1] - b[1]) < 1e-8


def test_planes_in_use_by_other_threads_make_room_too(gpu, ora):
    """Two threads evaluate without a pause while a third opens sessions that
    the device has no memory for: it gets the planes when a call ends, and the
    evaluations stay right throughout (the file's bars: some run without)."""
    import threading

    theta, k = [1.0, 0.1, 0.5], 6000
    x, y = ora.generate_xy_loc(9000, 3)
    z = np.random.default_rng(1).standard_normal(9000)
    sessions, ref = [], []
    for n in (9000, 8000):
        s = gpu.Session(x[:n], y[:n], dts=512)
        s.set_data(z=z[:n])
        sessions.append(s)
        ref.append(s.loglik(theta))
    with gpu.Session(x[:k], y[:k], dts=256) as t:
        t.set_data(z=z[:k])
        want = t.loglik(theta)
    got, stop = [[], []], threading.Event()

    def evaluate(i):
        while not stop.is_set():
            got[i].append(sessions[i].loglik(theta))

    with _Full(100 << 20):
        threads = [threading.Thread(target=evaluate, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        try:
            for _ in range(5):
                with gpu.Session(x[:k], y[:k], dts=256) as t:
                    t.set_data(z=z[:k])
                    assert t.loglik(theta) == want
        finally:
            stop.set()
            for t in threads:
                t.join()
    for i in range(2):
        assert len(got[i]) > 0
        assert np.abs(np.array(got[i]) / ref[i] - 1).max() < 2e-12
        assert sessions[i].loglik(theta) == ref[i]
        sessions[i].close()
