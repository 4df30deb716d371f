"""The vertex and grain passes' forms for small meshes against the oracle, bit
for bit, on both sides of the sizes where they take over,
partial warps and blocks included; GB_scaling 1 and other than 1 are different
instantiations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXACT = ("px", "py", "vx", "vy", "venergy", "garea", "blen", "benergy", "gvlen", "glist", "vg", "vb")


@pytest.mark.parametrize("scaling", [1.0, 0.7])
@pytest.mark.parametrize("n", [64, 65, 301, 6143, 6144, 6145])
def test_small_mesh_bit_exact(gpu, oracle_mod, n, scaling):
    m = gpu.voronoi(n, n)
    kw = dict(n_grains=n, dt=1e-3, dtau=1.0, domain_bound=float(n) ** 0.5, GB_eps=0.0, GB_scaling=scaling, SE_eps=1.0,
              SE_min=0.0, SE_max=0.5, do_nucleation=0, nmax=10 ** 6, tmax=-1, snap_gap=10 ** 8, min_grains=1)
    args = m["xy"], m["ridges"], m["oris"], m["se"]
    eng = gpu.Engine.from_arrays(gpu.default_options(**kw), *args)
    orc = oracle_mod.Oracle.from_arrays(oracle_mod.finish_options(oracle_mod.default_options(**kw)), *args)
    eng.set_mobility(1.0)
    for k in range(6):
        assert orc.step() == 0
        eng.step()
        st = eng.get_state()
        for f in EXACT:
            assert np.array_equal(st[f], orc.field(f)), (n, scaling, k, f)
        orc.finish_step()
    eng.close()
