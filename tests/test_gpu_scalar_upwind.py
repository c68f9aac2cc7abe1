"""The 2D scalar stage kernel's one upwind trace per face: bit for bit the
oracle's steps for every flow direction (none among them), at the edges of its
128-element blocks, with elements and vertices shuffled, and with non-finite
coefficients."""
import numpy as np
import pytest

import wasl_b200
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


def shuffled(arrays, seed):
    tags, xy, tris = arrays
    rng = np.random.Generator(np.random.PCG64(seed))
    tris = tris[rng.permutation(len(tris))]
    turn = rng.integers(0, 3, len(tris))
    return tags, xy, np.stack([tris[np.arange(len(tris)), (turn + k) % 3] for k in range(3)], 1)


@pytest.mark.parametrize("p", [0, 1, 2, 3])
@pytest.mark.parametrize("velocity", [(1.0, 0.5), (-0.7, 1.1), (-1.0, -0.2), (0.0, -1.0), (0.0, 0.0)])
@pytest.mark.parametrize("nx,ny,value", [(8, 8, None), (9, 7, None), (5, 13, None), (9, 7, np.nan),
                                         (9, 7, np.inf)])
def test_upwind_steps(oracle, p, velocity, nx, ny, value):
    arrays = shuffled(meshgen.jittered_box(nx, jitter=0.1, seed=nx, ny=ny), 3)
    om = oracle.tri_mesh(*arrays)
    M = (p + 1) * (p + 2) // 2
    c = np.random.Generator(np.random.PCG64(p)).standard_normal((M, om.ne))
    if value is not None:
        c[-1, 70] = value
    donors, basis = om.periodic_trace(p)
    with wasl_b200.Solver(*arrays, equation="scalar", polynomial_order=p, velocity=velocity) as g:
        g.set_state(c)
        ref = c.T.ravel().copy()  # the oracle's scalar layout: [element][mode]
        for _ in range(2):
            g.step(1e-3)
            om.scalar_step(*velocity, p, 1e-3, ref, donors, basis)
        got = g.get_state().reshape(M, om.ne)
    assert np.array_equal(got, ref.reshape(om.ne, M).T, equal_nan=True)
