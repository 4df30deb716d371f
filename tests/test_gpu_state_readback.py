"""sevc_get_state's two ways out: the device storing to the caller's arrays,
and (arrays at odd addresses) through device memory; the same bytes, on
sizes around the kernel's vector and page granularity."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,shift", [(64, 1), (65, 4), (1001, 12), (50001, 8)])
def test_readback_into_shifted_arrays(gpu, n, shift):
    import sevc
    m = gpu.voronoi(n, n)
    o = gpu.default_options(n_grains=n, dt=1e-4, dtau=1.0, domain_bound=float(np.sqrt(n)), GB_eps=0.0, GB_scaling=1.0,
                            SE_eps=1.0, SE_min=0.0, SE_max=0.5, do_nucleation=0, nmax=10 ** 8, tmax=-1, snap_gap=1)
    o.min_grains = -1
    e = gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"])
    e.step()
    want = e.get_state()
    size = {"v": e.nv, "v3": 3 * e.nv, "b": e.nb, "g": e.ng, "g100": 100 * e.ng}
    bufs = {f: np.full(size[k] * np.dtype(t).itemsize + 64, 0xA5, np.uint8) for f, k, t in sevc._MESH_FIELDS}
    mh = sevc.MeshHost(e.nv, e.nb, e.ng, *[bufs[f].ctypes.data + shift for f, _, _ in sevc._MESH_FIELDS])
    assert gpu.lib().sevc_get_state(e._h, C.byref(mh)) == 0
    for f, k, t in sevc._MESH_FIELDS:
        nb = size[k] * np.dtype(t).itemsize
        assert bufs[f][shift:shift + nb].tobytes() == want[f].tobytes(), f
        assert (bufs[f][:shift] == 0xA5).all() and (bufs[f][shift + nb:] == 0xA5).all(), f
    s = e.state_digest()
    import digest
    assert s == digest.digest(want.__getitem__)
    e.close()
