"""A tape recorded by run, which keeps two steps in flight and copies its
checkpoints between them, equals the one recorded step by step: the same
state and the same gradients, bit for bit; and the taped handle continues
from a saved file as one that never taped."""
import numpy as np
import pytest

from test_gpu_adjoint import AMAX, NB, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dt,steps,every", [(300, 1e-3, 7, 3), (300, 2e-3, 20, 5), (3000, 1e-4, 9, 20)])
def test_run_and_step_tapes_agree(gpu, n, dt, steps, every, tmp_path):
    mesh = gpu.voronoi(n, n + 1)
    out = []
    for whole in (True, False):
        e = make(gpu, mesh, dt)
        e.tape_start(every)
        if whole:
            e.run(steps)
        else:
            for _ in range(steps):
                e.step()
        d = np.linspace(1.0, -1.0, NB) / NB
        out.append((e.state_digest(), e.area_histogram(NB, AMAX).tobytes(),
                    [np.asarray(g).tobytes() for g in e.adjoint_histogram(NB, AMAX, d)], e.state_digest()))
        if whole:
            path = str(tmp_path / "c")
            e.checkpoint_save(path)
            e.tape_stop()
            plain = make(gpu, mesh, dt)
            plain.run(3)                     # another point of the run, its lists and counters in use
            plain.checkpoint_load(path)
            for a, b in zip(e.run(3), plain.run(3)):
                assert (a.n_flips, a.n_removals, a.polling_iters) == (b.n_flips, b.n_removals, b.polling_iters)
            assert e.state_digest() == plain.state_digest()
            plain.close()
        e.close()
    assert out[0] == out[1]
    assert out[0][0] == out[0][3]
