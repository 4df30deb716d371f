"""Profiling: times of the step's phases on meshes of every size, small ones
included (whose sparse phases are one launch otherwise), and the same results
as without."""
import pytest

pytestmark = pytest.mark.gpu

PHASES = {"boundary_geometry", "grain_fd", "two_three_count", "vertex_fd", "grain_dadt", "text_label", "removals", "flips",
          "update", "counts"}


@pytest.mark.parametrize("n,dt,steps", [(300, 0.1, 20), (4000, 0.3, 12), (32768, 0.1, 8), (33001, 0.1, 8)])
def test_phases_and_results(gpu, n, dt, steps):
    m = gpu.voronoi(n, 114 if n == 4000 else n)
    o = gpu.default_options(n_grains=n, dt=dt, dtau=1.0, domain_bound=float(n) ** 0.5, GB_eps=0.0, GB_scaling=1.0,
                            SE_eps=1.0, SE_min=0.0, SE_max=0.5, do_nucleation=0, nmax=10 ** 6, snap_gap=10 ** 6)
    a, b = (gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"]) for _ in range(2))
    a.set_profiling(True)
    events = 0
    for k in range(steps):
        x, y = a.step(), b.step()
        events += x.n_flips + x.n_removals
        assert (x.n_flips, x.n_removals, x.n_two_three, x.polling_iters, x.curr_n_grains) == \
            (y.n_flips, y.n_removals, y.n_two_three, y.polling_iters, y.curr_n_grains), k
        assert a.state_digest() == b.state_digest(), k
    assert events > 10
    prof = a.profile()
    assert PHASES <= set(prof), prof
    assert all(ms > 0 and count == steps for ms, count in (prof[p] for p in PHASES)), prof
    a.close()
    b.close()
