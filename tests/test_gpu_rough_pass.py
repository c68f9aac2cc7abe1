"""The mixed form's second pass (elements with a face across a jump of the cell
means, 16 lanes each): lists of every length, from all of a two-element mesh
to more elements than the pass has lanes for at once, against the FP64 oracle."""
import numpy as np
import pytest

import golden_cases as gc
import wasl_b200
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


def jumping_state(ne, p, seed):
    """Cell means that differ by far more than 5% across most faces."""
    rng = np.random.Generator(np.random.PCG64(seed))
    M = (p + 1) * (p + 2) // 2
    c = 0.01 * rng.standard_normal((4, M, ne))
    c[0, 0] = np.sqrt(2.0) * rng.uniform(0.5, 1.5, ne)
    c[1:3, 0] = 0.1 * rng.standard_normal((2, ne))
    c[3, 0] = np.sqrt(2.0) * rng.uniform(1.5, 3.5, ne)
    return c.ravel()


@pytest.mark.parametrize("kernel", [2, 5, 8, 10, 12])  # tile 128 and 64, shared-face 128, patch 128 and 64
@pytest.mark.parametrize("p,nx,ny,boundary", [
    (1, 1, 1, "transmissive"), (2, 3, 3, "periodic"), (3, 3, 3, "transmissive"),
    (1, 13, 5, "periodic"), (2, 13, 5, "transmissive"), (3, 13, 5, "periodic"),
    (1, 80, 80, "transmissive"), (3, 25, 25, "transmissive")])
def test_rough_elements_against_fp64(oracle, kernel, p, nx, ny, boundary):
    """Tolerance: one step moves the state by about CFL x |u|; the perturbations
    are FP32 sums of at most 256 rounded terms of that size, the rest is FP64."""
    cfl = 0.2
    arrays = meshgen.jittered_box(nx, jitter=0.1, seed=nx + p, ny=ny)
    om = oracle.tri_mesh(*arrays)
    c = jumping_state(om.ne, p, 10 * p + nx)
    kw = {"boundary": boundary}
    if boundary == "periodic":
        kw["donors"], kw["basis"] = om.periodic_trace(p)
    with wasl_b200.Solver(*arrays, polynomial_order=p, boundary=boundary, precision="mixed",
                          limiting=True, sensor_threshold=1e30, mixed_kernel=kernel) as g:
        g.set_state(c)
        dt = g.stable_dt(cfl)
        g.step(dt)
        got = g.get_state()
    om.euler_step(gc.GAMMA, p, dt, c, **kw)
    assert np.max(np.abs(got - c)) <= 256 * 2.0 ** -24 * cfl * np.max(np.abs(c))
