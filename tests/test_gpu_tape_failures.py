"""Failures while a tape records in a pipelined run: a step that fails keeps
no checkpoint alive, and a checkpoint that finds no memory leaves the handle at
the step it reports."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def free_memory():
    rt = C.CDLL("libcudart.so.13")
    a, b = C.c_size_t(), C.c_size_t()
    assert rt.cudaMemGetInfo(C.byref(a), C.byref(b)) == 0
    return a.value


def make(gpu, n, dt):
    m = gpu.voronoi(n, n)
    o = gpu.default_options(n_grains=n, dt=dt, dtau=1.0, domain_bound=float(n) ** 0.5, GB_eps=0.0, GB_scaling=1.0,
                            SE_eps=1.0, SE_min=0.0, SE_max=0.5, do_nucleation=0, nmax=10 ** 8, tmax=-1, snap_gap=10 ** 8, n_blocks=1,
                            n_threads=1)
    o.min_grains = -1
    return gpu.Engine.from_arrays(o, m["xy"], m["ridges"], m["oris"], m["se"])


@pytest.mark.parametrize("every", [1, 2])
def test_failed_steps_keep_no_checkpoint(gpu, every):
    def fail():
        e = make(gpu, 20001, 0.1)
        before = free_memory()
        e.tape_start(every)
        e.set_limits(polling_cap=1)              # one grid thread: any candidate needs a second iteration
        with pytest.raises(gpu.SevcError) as err:
            e.run(8)
        assert err.value.code == 4, err.value
        e.tape_stop()
        after = free_memory()
        e.close()
        return before - after
    fail()                                       # what the first use of the kernels takes
    assert sum(fail() for _ in range(5)) < 20 << 20


@pytest.mark.parametrize("single", [False, True])
def test_no_memory_for_a_checkpoint(gpu, single):
    rt = C.CDLL("libcudart.so.13")
    rt.cudaMalloc.argtypes = [C.c_void_p, C.c_size_t]
    rt.cudaFree.argtypes = [C.c_void_p]
    n = 100003                                   # a checkpoint is some 150 MB
    e, plain, other = (make(gpu, n, 1e-4) for _ in range(3))
    e.tape_start(2)                              # the first use of the kernels, with memory
    e.run(5)
    e.tape_stop()
    plain.run(5)
    e.tape_start(2)
    plain.tape_start(2)
    hog = []
    try:
        size = 1 << 40
        while size >= 1 << 20 and free_memory() > 80 << 20:
            p = C.c_void_p()
            if size < free_memory() - (40 << 20) and rt.cudaMalloc(C.byref(p), size) == 0:
                hog.append(p)
            else:
                size //= 2
        assert 0 < free_memory() < 120 << 20
        with pytest.raises(gpu.SevcError) as err:
            if single:
                for _ in range(6):
                    e.step()
            else:
                e.run(6)
        assert err.value.code == 6, err.value
        with pytest.raises(gpu.SevcError):       # a tape that cannot start is none
            other.tape_start(3)
    finally:
        for p in hog:
            rt.cudaFree(p)
    with pytest.raises(gpu.SevcError) as err:
        other.adjoint_histogram(4, 4.0, [1.0] * 4)
    assert err.value.code == 7, err.value
    other.close()
    info = e.step()                              # and the tape goes on where it stands
    taken = info.n + 1 - 5
    assert 1 <= taken <= 6
    plain.run(taken)
    assert e.state_digest() == plain.state_digest()
    e.run(3)
    plain.run(3)
    d = [1.0, -1.0] * 8
    got, want = ([np.asarray(g).tobytes() for g in x.adjoint_histogram(16, 4.0, d)] for x in (e, plain))
    assert got == want
    assert e.state_digest() == plain.state_digest()
    e.close()
    plain.close()
