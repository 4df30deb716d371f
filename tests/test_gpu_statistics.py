"""Histogram, grain statistics and gradient seed where their kernels split
the work: fewer grains than a block, ragged counts, every number of threads
with private bins (256 down to 16), areas beyond the last bin, dL/dh that is
not finite; against plain numpy over the polygons.

Tolerance: sums of n binary64 terms of one sign in any order differ by less
than n * 2^-53 relative (n < 4096: 5e-13)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-12


def engine(gpu, n, seed=5):
    m = gpu.voronoi(n, seed)
    o = gpu.default_options(n_grains=n, dt=1e-4, dtau=1.0, domain_bound=float(np.sqrt(n)), GB_eps=0.0, GB_scaling=1.0,
                            SE_eps=1.0, SE_min=999.0, SE_max=999.0, do_nucleation=0, nmax=10 ** 8, tmax=-1,
                            snap_gap=10 ** 8, n_blocks=32, n_threads=256)
    o.min_grains = -1
    return gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"])


def areas(st, D):
    out = []
    for g in np.nonzero(st["gen"] > 0)[0]:
        L = st["glist"][100 * g:100 * g + st["gvlen"][g]]
        x, y = st["px"][L], st["py"][L]
        x = x[0] + np.concatenate([[0], np.cumsum((np.diff(x) + D / 2) % D - D / 2)])
        y = y[0] + np.concatenate([[0], np.cumsum((np.diff(y) + D / 2) % D - D / 2)])
        x, y = x - x[0], y - y[0]
        out.append(0.5 * abs(np.sum(x * np.roll(y, -1) - y * np.roll(x, -1))))
    return np.array(out)


def b2(s):
    a = np.abs(s)
    return np.where(a <= 0.5, 0.75 - s * s, np.where(a <= 1.5, 0.5 * (1.5 - a) ** 2, 0.0))


@pytest.mark.parametrize("n", [64, 257, 3001])
def test_histogram_and_statistics(gpu, n):
    e = engine(gpu, n)
    for _ in range(3):
        e.step()
    D = e.opt.domain_bound
    a = areas(e.get_state(), D)
    for nbins, amax in [(1, 1.0), (7, 0.5), (64, 4.0), (200, 3.0), (500, 2.0), (1024, 6.0)]:
        t = a * len(a) / (D * D) / (amax / nbins)
        want = np.array([b2(t - k - 0.5).sum() for k in range(nbins)]) / len(a)
        got = e.area_histogram(nbins, amax)
        # a spline next to its knots moves by up to 1 per unit of t (relative error of an area ~1e-15)
        assert np.all(np.abs(got - want) <= TOL * (want + 1e-3 * nbins)), (n, nbins)
    s = e.grain_stats()
    assert s["n_grains"] == len(a)
    for key, val in (("mean_area", a.mean()), ("std_area", a.std()), ("min_area", a.min()), ("max_area", a.max())):
        assert abs(s[key] - val) <= 1e-11 * abs(val), key
    assert e.check_data() == e.check_data_host() == 0
    e.close()


def test_gradient_seed_with_non_finite_weights(gpu):
    """One NaN in dL/dh reaches every stored energy's gradient, as in the sum
    over all bins it stands for."""
    e = engine(gpu, 300)
    e.tape_start(4)
    e.step()
    w = np.zeros(20)
    w[19] = np.nan
    g, ggb, gmu = e.adjoint_histogram(20, 0.1, w)
    assert np.isnan(g).all() and np.isnan(ggb) and np.isnan(gmu)
    e.close()
