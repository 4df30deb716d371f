"""Every launch shape the autotuner may pick, against the oracle bit for bit:
each grains-per-block form with each side count from which grains get a warp
each (the 64-grain form works on nearly all its blocks in several chunks), and
each block size of the vertex and boundary passes."""
import ctypes as C
import itertools

import numpy as np
import pytest

from test_gpu_grain_chunks import ladder_mesh
from test_gpu_grain_pass import EXACT, pair

pytestmark = pytest.mark.gpu

SHAPES = list(itertools.product((128,), (128,), (9, 10, 11, 12), (4, 6))) + [(256, 512, 12, 6), (512, 256, 12, 6)]


def set_shape(gpu, eng, shape):
    return gpu.lib().sevc_set_launch_shape(eng._h, (C.c_int * 4)(*shape))


def mesh(gpu, name):
    if name == "ladder":
        return ladder_mesh(14, 3), 1.0
    m = gpu.voronoi(name, name)
    return (m["xy"], m["ridges"], m["oris"], m["se"]), float(name) ** 0.5


@pytest.mark.parametrize("name", [64, 129, 1001, 40001, "ladder"])
def test_each_shape_bit_exact(gpu, oracle_mod, name):
    arrays, domain = mesh(gpu, name)
    for k in range(2):
        engines = []
        for shape in SHAPES:
            eng, orc = pair(gpu, oracle_mod, *arrays, domain) if not engines else \
                (gpu.Engine.from_arrays(engines[0].opt, *arrays), orc)
            assert set_shape(gpu, eng, shape) == 0
            engines.append(eng)
        for _ in range(k + 1):
            assert orc.step() == 0
            orc.finish_step()
        for shape, eng in zip(SHAPES, engines):
            for _ in range(k + 1):
                eng.step()
            st = eng.get_state()
            for f in EXACT:
                assert np.array_equal(st[f], orc.field(f)), (name, shape, k, f)
            eng.close()


def test_other_shapes_are_refused(gpu):
    m = gpu.voronoi(64, 1)
    eng = gpu.Engine.from_arrays(gpu.default_options(n_grains=64, dt=1e-4, do_nucleation=0), m["xy"], m["ridges"],
                                 m["oris"], m["se"])
    for bad in ((64, 128, 12, 6), (128, 0, 12, 6), (128, 128, 8, 6), (128, 128, 13, 6), (128, 128, 12, 7),
                (128, 128, 12, 3)):
        assert set_shape(gpu, eng, bad) == 7, bad
    # a mesh without a block size of the vertex pass to choose keeps the one it has
    assert set_shape(gpu, eng, (512, 128, 12, 6)) == 0
    chosen = eng.autotune(steps=1)
    assert chosen[0] == 512 and chosen[3] in (4, 6)
    eng.close()
