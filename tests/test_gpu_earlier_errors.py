"""A call that fails (here: a record larger than the GPU's memory) leaves the
CUDA runtime's last-error state of the thread set.  Steps, runs, read-backs and
statistics after it judge their own launches only: they succeed, with the
results of a thread that saw no error."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fail_once(gpu):
    """70 TB of draws: the allocation is refused"""
    buf = np.zeros(8)
    assert gpu.lib().sevc_rng_record(8192, 1 << 30, C.c_void_p(buf.ctypes.data)) != 0


def make(gpu, n):
    m = gpu.voronoi(n, n)
    o = gpu.default_options(n_grains=n, dt=1e-4, dtau=1.0, domain_bound=float(n) ** 0.5, GB_eps=0.0, GB_scaling=1.0,
                            SE_eps=1.0, SE_min=0.0, SE_max=0.5, do_nucleation=0, nmax=10 ** 8, tmax=-1, snap_gap=10 ** 8)
    o.min_grains = -1
    return gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"])


def calls(e):
    return [lambda: e.step().n, lambda: [i.n for i in e.run(3)], lambda: e.get_state()["px"].tobytes(),
            lambda: e.area_histogram(16, 4.0).tobytes(), lambda: e.grain_stats(), e.check_data, e.state_digest]


@pytest.mark.parametrize("n,graphs", [(300, 1), (300, 0), (40001, 1), (40001, 0)])
def test_calls_after_a_refused_allocation(gpu, n, graphs):
    a, b = make(gpu, n), make(gpu, n)
    a.set_graphs(graphs)
    for k, (f, g) in enumerate(zip(calls(a), calls(b))):
        want = g()
        fail_once(gpu)
        assert f() == want, k
    a.close()
    b.close()
