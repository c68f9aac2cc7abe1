"""Always-on positivity through the suspects the stage kernels list: after a
step every check point of every element has positive density and pressure,
whether none, a few or all elements are listed, in each kernel family that lists
them; with none the pass changes nothing."""
import numpy as np
import pytest

import wasl_b200
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


def state(ne, p, share, seed):
    """A `share` of the elements with density and energy swinging to about zero,
    in a gas at rest (momentum over a density at its floor would be a velocity
    that no time step follows)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    M = (p + 1) * (p + 2) // 2
    c = 1e-3 * rng.standard_normal((4, M, ne))
    c[1:3] = 0.0
    c[0, 0], c[3, 0] = np.sqrt(2.0), np.sqrt(2.0) * 2.5
    wild = rng.uniform(size=ne) < share
    swing = 0.9 * rng.choice([-1.0, 1.0], ne)
    c[0, 1:] += np.where(wild, swing, 0.0)
    c[3, 1:] += np.where(wild, 2.4 * swing, 0.0)
    return c


def check_points(oracle, p):
    xi, eta, _ = oracle.tri_volume_rule(p)[:3]
    edges = oracle.tri_edge_rules(p)
    return np.array([oracle.dubiner(x, y, p) for x, y in
                     list(zip(xi, eta)) + list(zip(np.ravel(edges[0]), np.ravel(edges[1])))])


@pytest.mark.parametrize("kernel", [2, 8, 11])  # tile, shared-face and patch kernels
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,ny,share", [(1, 1, 1.0), (13, 5, 0.0), (13, 5, 0.05), (25, 25, 1.0)])
def test_every_check_point_stays_physical(oracle, kernel, p, nx, ny, share):
    arrays = meshgen.jittered_box(nx, jitter=0.1, seed=nx, ny=ny)
    c = state(2 * nx * ny, p, share, 7 + p)
    b = check_points(oracle, p)
    kw = dict(polynomial_order=p, boundary="transmissive", precision="mixed", limiting=True,
              sensor_threshold=1e30, mixed_kernel=kernel)
    after = {}
    for always in (False, True) if share == 0.0 else (True,):
        with wasl_b200.Solver(*arrays, positivity_all=always, **kw) as g:
            g.set_state(c)
            g.limit()
            g.step(1e-3 / (nx + ny))
            after[always] = g.get_state().reshape(c.shape)

    def smallest(c):
        """The smallest point density and pressure."""
        u = np.einsum("vme,qm->vqe", c, b)
        return u[0].min(), (0.4 * (u[3] - 0.5 * (u[1] ** 2 + u[2] ** 2) / u[0])).min()

    assert min(smallest(after[True])) > 0.0
    if share == 1.0:
        assert min(smallest(c)) < 0.0  # the data does need the limiter
    if share == 0.0:
        assert np.array_equal(after[False], after[True])
