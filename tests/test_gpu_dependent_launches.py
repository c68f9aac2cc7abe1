"""Stage kernels launched as programmatic dependents are resident while the launch
before them still writes the state they read: they read it through ordinary loads
after their wait.  Steps enqueued back to back give the bits of steps with the
stream drained and the state read between them, on meshes of several waves whose
rows do not fill whole cache lines."""
import numpy as np
import pytest

import wasl_b200
from golden.make_golden import seeded_state
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,kernel", [("plain", 0), ("mixed", 11), ("mixed", 12)])
@pytest.mark.parametrize("p,nx,ny", [(1, 301, 173), (2, 203, 151), (3, 131, 101)])
@pytest.mark.parametrize("limiting", [False, True])
@pytest.mark.parametrize("boundary", ["periodic", "transmissive"])
def test_back_to_back_steps_match_drained_ones(form, kernel, p, nx, ny, limiting, boundary):
    arrays = meshgen.jittered_box(nx, jitter=0.15, seed=p, ny=ny)
    c = seeded_state(2 * nx * ny, p, 50 + p, amplitude=0.02)
    with wasl_b200.Solver(*arrays, polynomial_order=p, boundary=boundary, limiting=limiting,
                          precision=form, mixed_kernel=kernel) as g:
        g.set_state(c)
        for _ in range(6):
            g.advance(0.05, 1)
            drained = g.get_state()
        assert not np.array_equal(drained, c)
        for _ in range(4):
            g.set_state(c)
            g.advance(0.05, 6)
            assert np.array_equal(g.get_state(), drained)
