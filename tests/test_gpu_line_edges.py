"""The 1D kernels where their blocks end: the Euler stage's 127-element blocks
(each face evaluated once) and the one-launch run's limits of one element per
thread, bit for bit the oracle's steps and the host loop's runs."""
import numpy as np
import pytest

import golden_cases as gc
import wasl_b200
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu
ENDS = [("periodic", "periodic"), ("outflow", "outflow")]
KINDS = {"periodic": 0, "inflow": 1, "outflow": 2}


def euler_state(ne, p, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    c = 0.05 * rng.standard_normal((4, p + 1, ne))
    c[0, 0] = np.sqrt(2.0) * (1.0 + 0.2 * rng.uniform(-1, 1, ne))
    c[3, 0] = np.sqrt(2.0) * 2.5
    return c.ravel()


@pytest.mark.parametrize("p", [0, 1, 2, 6])
@pytest.mark.parametrize("ends", ENDS)
@pytest.mark.parametrize("n", [2, 126, 127, 128, 253, 254, 255])
def test_euler_stage_blocks(oracle, p, ends, n):
    arrays = meshgen.jittered_line(n, jitter=0.2, seed=n + p)
    om = oracle.line_mesh(*arrays)
    c = euler_state(n, p, n)
    with wasl_b200.Solver(*arrays, dimensions=1, polynomial_order=p, boundary=ends[0],
                          boundary_right=ends[1]) as g:
        g.set_state(c)
        dt = g.stable_dt(0.2)
        for _ in range(2):
            g.step(dt)
            om.euler_step(gc.GAMMA, p, dt, c, KINDS[ends[0]], KINDS[ends[1]])
        assert np.array_equal(g.get_state(), c, equal_nan=True)


@pytest.mark.parametrize("value", [np.nan, np.inf, 0.0])
def test_euler_stage_not_finite(oracle, value):
    arrays = meshgen.jittered_line(130, jitter=0.2, seed=1)
    om = oracle.line_mesh(*arrays)
    c = euler_state(130, 2, 3).reshape(4, 3, 130)
    c[0, 2, 126] = value
    c[2, 1, 5] = value
    c = c.ravel().copy()
    with wasl_b200.Solver(*arrays, dimensions=1, polynomial_order=2, boundary="outflow") as g:
        g.set_state(c)
        g.step(1e-3)
        om.euler_step(gc.GAMMA, 2, 1e-3, c, 2, 2)
        assert np.array_equal(g.get_state(), c, equal_nan=True)


# (order, sizes around the limits of one element per thread and of the clusters of
# four and eight blocks; 19 steps: the halo is exchanged every eighth)
@pytest.mark.parametrize("p,n", [(0, 1), (2, 31), (2, 32), (2, 95), (2, 96), (0, 97),
                                 (2, 400), (2, 416), (2, 417), (2, 1023), (2, 1024), (1, 2345),
                                 (3, 511), (3, 512), (3, 1952), (3, 1953), (6, 300)])
@pytest.mark.parametrize("ends,speed", [(("periodic", "periodic"), 0.7),
                                        (("inflow", "outflow"), 0.7),
                                        (("outflow", "inflow"), -0.9),
                                        (("outflow", "outflow"), 1.3)])
def test_scalar_run_limits(p, n, ends, speed):
    arrays = meshgen.jittered_line(n, jitter=0.2 if n > 1 else 0.0, seed=n)
    c = np.random.Generator(np.random.PCG64(p)).standard_normal(n * (p + 1))
    out = []
    for resident in (False, True):
        with wasl_b200.Solver(*arrays, dimensions=1, equation="scalar", polynomial_order=p,
                              velocity=(speed, 0.0), boundary=ends[0], boundary_right=ends[1],
                              inflow=(0.8, -0.3)) as g:
            g.set_state(c)
            run = g.run_resident if resident else g.run
            out.append((run(0.3, 0.0, 1.0, 19), g.get_state()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("p,n", [(0, 2), (1, 31), (1, 32), (2, 511), (2, 512), (3, 33), (3, 500), (5, 60)])
@pytest.mark.parametrize("ends", ENDS)
def test_euler_run_limits(p, n, ends):
    arrays = meshgen.jittered_line(n, jitter=0.2, seed=n)
    out = []
    for resident in (False, True):
        with wasl_b200.Solver(*arrays, dimensions=1, polynomial_order=p, boundary=ends[0],
                              boundary_right=ends[1]) as g:
            g.set_state(euler_state(n, p, n + p))
            run = g.run_resident if resident else g.run
            out.append((run(0.1, 0.0, 1.0, 6), g.get_state()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n", [2, 127, 128, 3000])
def test_euler_advance_takes_the_next_speed_from_the_last_stage(n):
    """Several steps in one call (each step's CFL speed reduced by the step
    before) and one call per step (each a pass over the state): the same bits."""
    arrays = meshgen.jittered_line(n, jitter=0.2, seed=n)
    out = []
    for calls, steps in ((1, 5), (5, 1)):
        with wasl_b200.Solver(*arrays, dimensions=1, polynomial_order=2, boundary="outflow") as g:
            g.set_state(euler_state(n, 2, n))
            for _ in range(calls):
                g.advance(0.2, steps)
            out.append(g.get_state())
    assert np.array_equal(out[0], out[1])
