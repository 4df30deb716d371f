"""Steps of thousands of events: their dense form (the events applied over the
whole GPU, from the step after one of more than 1,024 events on) against the
oracle, and an ensemble whose dense steps must equal its members' own, which
are small enough for the one-launch form."""
import os

import numpy as np
import pytest

from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def options(n, dt, domain):
    return dict(n_grains=n, dt=dt, dtau=1.0, domain_bound=domain, GB_eps=0.0, GB_scaling=1.0, SE_eps=1.0, SE_min=0.0,
                SE_max=0.5, do_nucleation=0, nmax=10 ** 6, min_grains=10, snap_gap=10 ** 6)


@pytest.mark.parametrize("n,seed", [(33001, 11), (60000, 12)])
def test_dense_steps_bit_exact(gpu, oracle_mod, n, seed):
    mesh = gpu.voronoi(n, seed)
    kw = options(n, 0.12, float(n) ** 0.5)
    args = mesh["xy"], mesh["ridges"], mesh["oris"], mesh["se"]
    eng = gpu.Engine.from_arrays(gpu.default_options(**kw), *args)
    orc = oracle_mod.Oracle.from_arrays(oracle_mod.finish_options(oracle_mod.default_options(**kw)), *args)
    orc.set_threads(os.cpu_count() or 1)
    launches, events = [], []
    for k in range(14):
        rc = orc.step()
        if rc:                      # the mesh tore: both sides say so
            with pytest.raises(gpu.SevcError) as e:
                eng.step()
            assert e.value.code == rc
            break
        info, s = eng.step(), orc.s
        launches.append(info.kernel_launches)
        events.append(info.n_flips + info.n_removals)
        compare(eng.get_state(), orc, True, str((n, k)), complete=bool(info.outputs_complete))
        assert (info.n_flips, info.n_removals, info.n_two_three, info.n_conflicts, info.polling_iters) == \
            (s.ev_flips, s.ev_removals, s.ev_two_three, s.ev_conflicts, s.polling_iters), (n, k)
        orc.finish_step()
    assert max(events[:-1]) > 1024 and min(events) <= 1024
    for k in range(1, len(launches)):
        assert launches[k] == launches[0] + (4 if events[k - 1] > 1024 else 0), (k, launches, events)
    eng.close()


def test_dense_ensemble_equals_its_members(gpu):
    sizes = (14001, 9000, 7003, 4500)
    meshes = [gpu.voronoi(n, 20 + i) for i, n in enumerate(sizes)]
    domain = float(np.mean(sizes)) ** 0.5
    batch = gpu.Engine.from_batch(gpu.default_options(**options(sizes[0], 0.15, domain)), meshes)
    plain = [gpu.Engine.from_arrays(gpu.default_options(**options(n, 0.15, domain)), m["xy"], m["ridges"], m["oris"],
                                    m["se"]) for n, m in zip(sizes, meshes)]
    events = []
    for _ in range(10):
        info = batch.step()
        events.append(info.n_flips + info.n_removals)
        for p in plain:
            p.step()
    st = batch.get_state()
    assert sum(e > 1024 for e in events[:-1]) >= 2, events
    for i, p in enumerate(plain):
        part, own = batch.instance_state(st, i), p.get_state()
        for f in part:
            if f not in ("btext", "gdadt"):
                assert np.array_equal(part[f], own[f]), (i, f)
    for e in [batch] + plain:
        e.close()
