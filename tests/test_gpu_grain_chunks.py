"""The grain pass where a block's grains need more list slots than it holds
at once, so that it works on them in several chunks, at each block shape:
every block of the first hundreds to thousands of grains, all of 30 sides,
takes three chunks or more.  Bit for bit against the oracle."""
import numpy as np
import pytest

from test_gpu_grain_pass import lockstep, pair

pytestmark = pytest.mark.gpu


def ladder_mesh(nx, seed):
    """nx * nx hexagons (nx even) on a staggered grid, every edge between two
    of them split by a ladder of three small cells (triangle, quadrilateral,
    triangle): 30-sided grains, numbered first because their common corners
    are the first vertices, then nine small ones for each.  Triple junctions
    only; positions shaken by a few percent of an edge."""
    rng = np.random.default_rng(seed)
    up = np.array([0.5, 0.375])                 # corners above a seed: right and centre
    top = np.array([0.0, 0.625])
    corner = {}
    pts = []
    for j in range(nx):
        for i in range(nx):
            s = np.array([i + 0.5 * (j % 2), float(j)])
            corner[i, j, 0] = len(pts)
            pts.append(s + up)
            corner[i, j, 1] = len(pts)
            pts.append(s + top)
    ridges = []

    def ladder(a, b):
        p0, d = pts[a], pts[b] - pts[a]
        d = d - nx * np.round(d / nx)
        t = np.array([-d[1], d[0]])
        at = lambda x, y: p0 + x * d + y * t
        k = len(pts)
        pts.extend([at(0.2, 0), at(0.4, 0.1), at(0.4, -0.1), at(0.6, 0.1), at(0.6, -0.1), at(0.8, 0)])
        ridges.extend([(a, k), (k, k + 1), (k, k + 2), (k + 1, k + 2), (k + 1, k + 3), (k + 2, k + 4), (k + 3, k + 4),
                       (k + 3, k + 5), (k + 4, k + 5), (k + 5, b)])

    for j in range(nx):
        for i in range(nx):
            odd = j % 2
            below = (j - 1) % nx
            # below a seed: the top corners of the row below lie at its lower right and left
            lower = corner[i if not odd else (i + 1) % nx, below, 1]
            ladder(corner[i, j, 0], lower)                           # towards the seed at the right
            ladder(corner[i, j, 0], corner[i, j, 1])                 # upper right
            ladder(corner[i, j, 1], corner[(i - 1) % nx, j, 0])      # upper left
    xy = np.array(pts) + 0.02 * rng.random((len(pts), 2))
    n = 10 * nx * nx
    return (xy / nx) % 1.0, np.array(ridges, np.int32), rng.random(n), rng.random(n)


# grains: 8 a block up to 6,144, 16 up to 32,768, 32 above
@pytest.mark.parametrize("nx", [4, 14, 32, 58])
def test_blocks_of_several_chunks(gpu, oracle_mod, nx):
    xy, ridges, oris, se = ladder_mesh(nx, nx)
    eng, orc = pair(gpu, oracle_mod, xy, ridges, oris, se, 1.0)
    sides = eng.get_state()["gvlen"]
    assert (sides[:nx * nx] == 30).all() and len(sides) == 10 * nx * nx
    lockstep(gpu.SevcError, eng, orc, 2, nx)
