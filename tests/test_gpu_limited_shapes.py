"""Every launch shape that runs with the limiter, on meshes just below, at and
above its tiles' and patches' sizes: the second pass (elements with a face across
a jump of the cell means) against the FP64 oracle, and the listed positivity
against the plain form's, which tests every element."""
import functools

import numpy as np
import pytest

import golden_cases as gc
import wasl_b200
from test_gpu_rough_pass import jumping_state
from test_gpu_suspects import check_points
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu

# mixed_kernel values: tile 2-5, shared-face 6-9, patch 10-13, persistent 16-17
# (tiles and patches of 64, 96, 128, 192 and 256 elements).
KERNELS = [*range(2, 14), 16, 17]
MESHES = [(31, 1), (16, 2), (33, 1), (24, 2), (13, 5), (97, 1), (16, 8), (43, 3)]
FLOOR = 0.2


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,ny", MESHES)
def test_second_pass_in_every_shape(oracle, kernel, p, nx, ny):
    """Tolerance: one step moves the state by about CFL x |u|; the perturbations
    are FP32 sums of at most 256 rounded terms of that size, the rest is FP64."""
    cfl = 0.2
    arrays = meshgen.jittered_box(nx, jitter=0.1, seed=nx + p, ny=ny)
    om = oracle.tri_mesh(*arrays)
    c = jumping_state(om.ne, p, 10 * p + nx)
    with wasl_b200.Solver(*arrays, polynomial_order=p, boundary="transmissive", precision="mixed",
                          limiting=True, sensor_threshold=1e30, mixed_kernel=kernel) as g:
        g.set_state(c)
        dt = g.stable_dt(cfl)
        g.step(dt)
        got = g.get_state()
    om.euler_step(gc.GAMMA, p, dt, c, boundary="transmissive")
    assert np.max(np.abs(got - c)) <= 256 * 2.0 ** -24 * cfl * np.max(np.abs(c))


def low_state(oracle, p, ne, seed):
    """A gas at rest whose density and pressure fall to half the floor at a check
    point of every third element (positive everywhere), with jumps of the means
    across some faces."""
    rng = np.random.Generator(np.random.PCG64(seed))
    b = check_points(oracle, p)
    high = rng.standard_normal((b.shape[1] - 1, ne))
    mean = np.where(rng.uniform(size=ne) < 0.2, 1.5, 1.0)
    lowest = np.where(np.arange(ne) % 3 == 0, 0.5 * FLOOR, 0.9 * mean)
    swing = (b[:, 1:] @ high).min(axis=0)
    rho = np.vstack([np.sqrt(2.0) * mean, high * ((mean - lowest) / -swing)])
    c = np.zeros((4, b.shape[1], ne))
    c[0], c[3] = rho, 2.5 * rho
    return c


@functools.lru_cache(maxsize=None)
def plain_result(oracle, p, nx, ny):
    arrays = meshgen.jittered_box(nx, jitter=0.1, seed=nx + p, ny=ny)
    c = low_state(oracle, p, 2 * nx * ny, 3 * nx + p)
    with solver(arrays, p, precision="plain") as g:
        g.set_state(c)
        g.step(1e-200)
        return arrays, c, g.get_state().reshape(c.shape)


def solver(arrays, p, **kw):
    return wasl_b200.Solver(*arrays, polynomial_order=p, boundary="transmissive", limiting=True,
                            sensor_threshold=1e30, positivity_all=True, density_floor=FLOOR,
                            pressure_floor=FLOOR, **kw)


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,ny", MESHES)
def test_listed_positivity_in_every_shape(oracle, kernel, p, nx, ny):
    """A step so short that only the stages' positivity changes the state.  The
    forms' stage combinations differ by their roundings (a few units of 1e-16 of
    states of order one, times ten modes and the limiter's condition of about
    ten): 1e-12."""
    arrays, c, expected = plain_result(oracle, p, nx, ny)
    assert np.max(np.abs(expected - c)) > 0.01  # elements are limited
    with solver(arrays, p, precision="mixed", mixed_kernel=kernel) as g:
        g.set_state(c)
        g.step(1e-200)
        got = g.get_state().reshape(c.shape)
    assert np.max(np.abs(got - expected)) <= 1e-12
