"""Histograms of different sizes from several threads at once, each with its
own handle: every call returns what it returns alone, whatever shared memory
the other threads' launches ask for."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_histograms_of_different_sizes_side_by_side(gpu):
    n = 1000
    m = gpu.voronoi(n, n)
    engines, want, amax = [], [], (4.0, 3.0)       # alternating: a call that left the last result would show
    bins = [1024, 1, 16, 700, 1024, 64]
    for nbins in bins:
        o = gpu.default_options(n_grains=n, dt=1e-4, dtau=1.0, domain_bound=float(n) ** 0.5, do_nucleation=0,
                                nmax=10 ** 8, tmax=-1, snap_gap=10 ** 8)
        engines.append(gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"]))
        want.append([engines[-1].area_histogram(nbins, a).tobytes() for a in amax])
    wrong, start = [], threading.Barrier(len(bins))

    def work(i):
        start.wait()
        for k in range(2000):
            try:
                if engines[i].area_histogram(bins[i], amax[k % 2]).tobytes() != want[i][k % 2]:
                    wrong.append((bins[i], k))
            except gpu.SevcError as e:
                wrong.append((bins[i], k, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(bins))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[:5])
    assert np.all([e.check_data() == 0 for e in engines])
    for e in engines:
        e.close()
