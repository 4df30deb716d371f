"""Nucleation attempts against the oracle, on meshes whose vertices give each
random stream none or one, up to one and more than one batch of eight, and
with free slots anywhere: an attempt every step past the 5/6 gate."""
import os

import numpy as np
import pytest

from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dt,steps", [(700, 0.1, 50), (4097, 0.1, 30), (33001, 0.1, 45)])
def test_attempts_bit_exact(gpu, oracle_mod, n, dt, steps):
    mesh = gpu.voronoi(n, n)
    kw = dict(n_grains=n, dt=dt, dtau=dt, domain_bound=float(n) ** 0.5, GB_eps=0.0, GB_scaling=1.0, SE_eps=1.0,
              SE_min=0.0, SE_max=3.0, do_nucleation=1, nucleation_gap=1, MC_k=0.5, nmax=10 ** 6, min_grains=10,
              snap_gap=10 ** 6)
    args = mesh["xy"], mesh["ridges"], mesh["oris"], np.full(n, 3.0)
    eng = gpu.Engine.from_arrays(gpu.default_options(**kw), *args)
    orc = oracle_mod.Oracle.from_arrays(oracle_mod.finish_options(oracle_mod.default_options(**kw)), *args)
    orc.rng_table(gpu.rng_record(8192, (2 * (2 * n // 8192 + 1) + 4) * steps))
    orc.set_threads(os.cpu_count() or 1)
    attempts = 0
    for k in range(steps):
        rc = orc.step()
        if rc:                      # the mesh tore: both sides say so
            with pytest.raises(gpu.SevcError) as e:
                eng.step()
            assert e.value.code == rc
            break
        info, s = eng.step(), orc.s
        where = str((n, k))
        st = eng.get_state()
        gone = st["gen"] == 0       # see test_gpu_tail
        st["garea"][gone] = orc.field("garea")[gone]
        compare(st, orc, True, where, complete=bool(info.outputs_complete))
        assert info.n_nucleations == s.ev_nucleations, where
        if info.nucleation_attempted:
            assert info.nucleation_candidate == s.vrt_id_candidate, where
            attempts += 1
        orc.finish_step()
    assert attempts > 3
    eng.close()
