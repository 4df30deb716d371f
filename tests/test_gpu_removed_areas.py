"""The area that a removed grain keeps (snapshots print it) is the one of the
start of its last step, also when a 2x3 pass edited it before the step's
removals, or a later pass of the loop, took it: every field of every grain,
removed ones included, against the oracle, in the one-launch, the split and the
dense form of a step, and with nucleation."""
import os

import numpy as np
import pytest

from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed,dt,steps,se", [(4000, 114, 0.3, 12, None), (2000, 5, 0.3, 40, None),
                                               (20000, 6, 0.2, 25, None), (33001, 3, 0.2, 20, None),
                                               (60000, 12, 0.15, 14, None), (700, 700, 0.1, 50, 3.0),
                                               (33001, 33001, 0.1, 45, 3.0)])
def test_areas_of_removed_grains(gpu, oracle_mod, n, seed, dt, steps, se):
    mesh = gpu.voronoi(n, seed)
    kw = dict(n_grains=n, dt=dt, dtau=dt if se else 1.0, domain_bound=float(n) ** 0.5, GB_eps=0.0, GB_scaling=1.0,
              SE_eps=1.0, SE_min=0.0, SE_max=se or 0.5, do_nucleation=1 if se else 0, MC_k=0.5, nmax=10 ** 6,
              min_grains=10, snap_gap=10 ** 6)
    if se:
        kw["nucleation_gap"] = 1
    args = mesh["xy"], mesh["ridges"], mesh["oris"], np.full(n, se) if se else mesh["se"]
    eng = gpu.Engine.from_arrays(gpu.default_options(**kw), *args)
    orc = oracle_mod.Oracle.from_arrays(oracle_mod.finish_options(oracle_mod.default_options(**kw)), *args)
    if se:
        orc.rng_table(gpu.rng_record(8192, (2 * (2 * n // 8192 + 1) + 4) * steps))
    orc.set_threads(os.cpu_count() or 1)
    for k in range(steps):
        rc = orc.step()
        if rc:                      # the mesh tore: both sides say so
            with pytest.raises(gpu.SevcError) as e:
                eng.step()
            assert e.value.code == rc
            break
        info = eng.step()
        compare(eng.get_state(), orc, True, str((n, seed, k)), complete=bool(info.outputs_complete))
        orc.finish_step()
    eng.close()
