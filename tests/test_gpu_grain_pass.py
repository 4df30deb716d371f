"""The grain pass against the oracle, bit for bit, where its paths meet:
partial blocks and chunks, domains whose coordinates lie in, above and
below the binades the exactness certificate takes (grains at the axes and
across the wrap are always outside it), and a grain of more sides than the
ordered path holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXACT = ("px", "py", "vx", "vy", "venergy", "garea", "blen", "gvlen", "glist", "vg", "vb")


def pair(gpu, oracle_mod, xy, ridges, oris, se, domain):
    n = len(oris)
    kw = dict(n_grains=n, dt=1e-6 * domain * domain, dtau=1.0, domain_bound=domain, GB_eps=0.0, GB_scaling=1.0,
              SE_eps=1.0, SE_min=0.0, SE_max=0.5, do_nucleation=0, nmax=100, tmax=-1, snap_gap=10 ** 8, min_grains=10)
    eng = gpu.Engine.from_arrays(gpu.default_options(**kw), xy, ridges, oris, se)
    oopt = oracle_mod.finish_options(oracle_mod.default_options(**kw))
    return eng, oracle_mod.Oracle.from_arrays(oopt, xy, ridges, oris, se)


def lockstep(sevc_error, eng, orc, steps, where):
    for k in range(steps):
        rc = orc.step()
        if rc:              # time steps of domain^2 tear the largest meshes apart: both sides say so
            with pytest.raises(sevc_error) as e:
                eng.step()
            assert e.value.code == rc, (where, k)
            break
        eng.step()
        st = eng.get_state()
        for f in EXACT:
            assert np.array_equal(st[f], orc.field(f)), (where, k, f)
        orc.finish_step()
    eng.close()


@pytest.mark.parametrize("n,domain", [(64, 1.0), (65, 8.0), (95, 9.75), (129, 1e-7), (257, 1e-3), (1000, 37.5),
                                      (3001, 1e3), (999, 5e5), (1500, 3e6)])
def test_grain_pass_bit_exact(gpu, oracle_mod, n, domain):
    m = gpu.voronoi(n, n)
    lockstep(gpu.SevcError, *pair(gpu, oracle_mod, m["xy"], m["ridges"], m["oris"], m["se"], domain), 8, (n, domain))


@pytest.mark.parametrize("seed", [4, 6])
def test_launch_shapes_give_the_same_bits(gpu, oracle_mod, seed):
    """the shapes the autotuner may pick: it reports them, the steps after it
    equal the oracle's"""
    m = gpu.voronoi(40001, seed)
    eng, orc = pair(gpu, oracle_mod, m["xy"], m["ridges"], m["oris"], m["se"], 200.0)
    chosen = eng.autotune(steps=1)
    assert chosen[2] in (9, 10, 11, 12) and chosen[3] in (4, 5, 6, 8)
    lockstep(gpu.SevcError, eng, orc, 2, seed)


def test_hundred_sided_grain(gpu, oracle_mod):
    from test_gpu_failures import hundred_sided_mesh
    lockstep(gpu.SevcError, *pair(gpu, oracle_mod, *hundred_sided_mesh(), 1.0), 8, "100-gon")
