"""The plain P2 stage kernel's register bounds by grid size (one wave of three or of
four blocks per SM, or more): bit for bit the oracle's step on meshes of a whole
wave and of a block more, numbered in order and at random."""
import numpy as np
import pytest

import golden_cases as gc
import wasl_b200
from golden.make_golden import seeded_state
from test_gpu_stage_blocks import shuffled
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(111, 128), (98, 145), (128, 148), (45, 421)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_p2_grids_around_a_wave(oracle, nx, ny, shuffle):
    arrays = meshgen.jittered_box(nx, jitter=0.1, seed=nx, ny=ny)
    if shuffle:
        arrays = shuffled(arrays, 5)
    om = oracle.tri_mesh(*arrays)
    c = seeded_state(om.ne, 2, 42)
    donors, basis = om.periodic_trace(2)
    with wasl_b200.Solver(*arrays, polynomial_order=2) as g:
        g.set_state(c)
        dt = g.stable_dt(0.2)
        g.step(dt)
        om.euler_step(gc.GAMMA, 2, dt, c, donors=donors, basis=basis)
        assert np.array_equal(g.get_state(), c)
