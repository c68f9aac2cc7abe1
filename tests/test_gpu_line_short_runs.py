"""Resident advection runs spread over a cluster of blocks, for step counts below,
at and just above the eight that a block takes between two exchanges: a block
writes its cells back only after its neighbour has read the halo it starts from,
so every repetition gives the host loop's bits."""
import numpy as np
import pytest

import wasl_b200
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,n", [(0, 97), (2, 96), (2, 400), (2, 417), (1, 2345), (3, 512)])
@pytest.mark.parametrize("ends,speed", [(("periodic", "periodic"), 0.7),
                                        (("periodic", "periodic"), -0.7),
                                        (("inflow", "outflow"), 0.7),
                                        (("outflow", "inflow"), -0.9)])
def test_short_resident_runs(p, n, ends, speed):
    arrays = meshgen.jittered_line(n, jitter=0.2, seed=n)
    c = np.random.Generator(np.random.PCG64(p + n)).standard_normal(n * (p + 1))
    with wasl_b200.Solver(*arrays, dimensions=1, equation="scalar", polynomial_order=p,
                          velocity=(speed, 0.0), boundary=ends[0], boundary_right=ends[1],
                          inflow=(0.8, -0.3)) as g:
        for steps in (0, 1, 2, 7, 8, 9, 16, 17):
            g.set_state(c)
            taken = g.run(0.3, 0.0, 1.0, steps)
            expected = g.get_state()
            for _ in range(20):
                g.set_state(c)
                assert g.run_resident(0.3, 0.0, 1.0, steps) == taken
                assert np.array_equal(g.get_state(), expected)


def test_short_run_by_its_end_time():
    """The run ends inside its first steps by end_time, not by the step limit."""
    arrays = meshgen.jittered_line(400, jitter=0.2, seed=4)
    c = np.random.Generator(np.random.PCG64(4)).standard_normal(400 * 3)
    with wasl_b200.Solver(*arrays, dimensions=1, equation="scalar", polynomial_order=2,
                          velocity=(0.7, 0.0)) as g:
        end = 2.5 * g.stable_dt(0.3)
        g.set_state(c)
        taken = g.run(0.3, 0.0, end)
        expected = g.get_state()
        assert taken[0] == 3
        for _ in range(50):
            g.set_state(c)
            assert g.run_resident(0.3, 0.0, end) == taken
            assert np.array_equal(g.get_state(), expected)
