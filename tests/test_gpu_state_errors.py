"""sevc_get_state with a missing array: refused, with nothing written to the
others."""
import ctypes as C

import numpy as np
import pytest

import sevc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])        # both ways out of the device
@pytest.mark.parametrize("field", [f for f, _, _ in sevc._MESH_FIELDS])
def test_missing_array_is_refused(gpu, field, shift):
    n = 64
    m = gpu.voronoi(n, n)
    o = gpu.default_options(n_grains=n, dt=1e-4, dtau=1.0, domain_bound=8.0, do_nucleation=0)
    e = gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"])
    size = {"v": e.nv, "v3": 3 * e.nv, "b": e.nb, "g": e.ng, "g100": 100 * e.ng}
    bufs = {f: np.full(size[k] * np.dtype(t).itemsize + 64, 0xA5, np.uint8) for f, k, t in sevc._MESH_FIELDS}
    mh = sevc.MeshHost(e.nv, e.nb, e.ng, *[None if f == field else bufs[f].ctypes.data + shift
                                           for f, _, _ in sevc._MESH_FIELDS])
    assert gpu.lib().sevc_get_state(e._h, C.byref(mh)) == 6
    assert b"array" in gpu.lib().sevc_last_error()
    assert all((b == 0xA5).all() for b in bufs.values())
    assert e.step().n == 0
    assert len(e.get_state()) == len(bufs)
    e.close()
