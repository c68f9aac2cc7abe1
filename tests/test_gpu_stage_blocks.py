"""The plain 2D Euler stage kernel at the edges of its 64-element blocks:
bit for bit the oracle's step on meshes just below, at and above whole blocks,
with neighbours spread over the blocks in every way (elements and their
vertices shuffled), and with non-finite coefficients."""
import numpy as np
import pytest

import golden_cases as gc
import wasl_b200
from golden.make_golden import seeded_state
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


def shuffled(arrays, seed):
    tags, xy, tris = arrays
    rng = np.random.Generator(np.random.PCG64(seed))
    tris = tris[rng.permutation(len(tris))]
    turn = rng.integers(0, 3, len(tris))
    return tags, xy, np.stack([tris[np.arange(len(tris)), (turn + k) % 3] for k in range(3)], 1)


@pytest.mark.parametrize("p", [0, 1, 2, 3])
@pytest.mark.parametrize("nx,ny,boundary,shuffle", [
    (1, 1, "transmissive", False), (31, 1, "transmissive", False), (8, 4, "periodic", False),
    (33, 1, "transmissive", True), (8, 8, "periodic", True), (5, 13, "periodic", True),
    (7, 23, "transmissive", True)])
def test_block_edges(oracle, p, nx, ny, boundary, shuffle):
    arrays = meshgen.jittered_box(nx, jitter=0.1, seed=nx + ny, ny=ny)
    if shuffle:
        arrays = shuffled(arrays, 5)
    om = oracle.tri_mesh(*arrays)
    c = seeded_state(om.ne, p, 40 + p)
    kw = {"boundary": boundary}
    if boundary == "periodic":
        kw["donors"], kw["basis"] = om.periodic_trace(p)
    with wasl_b200.Solver(*arrays, polynomial_order=p, boundary=boundary) as g:
        g.set_state(c)
        dt = g.stable_dt(0.2)
        for _ in range(2):
            g.step(dt)
            om.euler_step(gc.GAMMA, p, dt, c, **kw)
        assert np.array_equal(g.get_state(), c, equal_nan=True)


@pytest.mark.parametrize("p", [0, 1, 2, 3])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 0.0])
def test_not_finite(oracle, p, value):
    """A NaN, infinite or vacuum coefficient spreads as in the oracle."""
    arrays = shuffled(meshgen.jittered_box(9, jitter=0.1, seed=3), 6)
    om = oracle.tri_mesh(*arrays)
    c = seeded_state(om.ne, p, 60 + p).reshape(4, -1, om.ne)
    c[0, -1, 70] = value
    c[3, 0, 11] = value
    c = c.ravel().copy()
    with wasl_b200.Solver(*arrays, polynomial_order=p, boundary="transmissive") as g:
        g.set_state(c)
        g.step(1e-3)
        om.euler_step(gc.GAMMA, p, 1e-3, c, boundary="transmissive")
        assert np.array_equal(g.get_state(), c, equal_nan=True)
