"""A state written through the device pointer between two calls is the state the
next call starts from, its first CFL step included: the bits of a fresh handle."""
import numpy as np
import pytest
import torch

import wasl_b200
from golden.make_golden import seeded_state
from wasl_b200 import halo, meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,kernel", [("plain", 0), ("mixed", 1), ("mixed", 2), ("mixed", 8),
                                         ("mixed", 11), ("mixed", 16)])
@pytest.mark.parametrize("faster", [0.5, 4.0])
def test_advance_after_a_write_through_the_device_pointer(form, kernel, faster):
    arrays = meshgen.jittered_box(17, jitter=0.15, seed=5)
    kw = dict(polynomial_order=2, precision=form, mixed_kernel=kernel, element_order="caller")
    c = seeded_state(2 * 17 * 17, 2, 7, amplitude=0.02)
    # The same gas with its sound speed scaled: energy (and pressure) times faster^2.
    other = c.reshape(4, 6, -1).copy()
    other[1:3] = 0.0
    other[3] *= faster ** 2
    with wasl_b200.Solver(*arrays, **kw) as g:
        g.set_state(other.ravel())
        g.advance(0.1, 2)
        expected = g.get_state()
    with wasl_b200.Solver(*arrays, **kw) as g:
        g.set_state(c)
        view = halo.device_state(g)
        for _ in range(2):
            g.advance(0.1, 3)
            view.copy_(torch.from_numpy(other.reshape(24, -1)))
            torch.cuda.synchronize()
            g.advance(0.1, 2)
            assert np.array_equal(g.get_state(), expected)


def test_the_kept_speed_changes_no_bits():
    """Without a device pointer the last stage's CFL speed serves the next call:
    one step a call and all in one call give the same bits."""
    arrays = meshgen.jittered_box(17, jitter=0.15, seed=5)
    c = seeded_state(2 * 17 * 17, 2, 7, amplitude=0.02)
    out = []
    for calls, steps in ((1, 6), (6, 1)):
        with wasl_b200.Solver(*arrays, polynomial_order=2, precision="mixed", mixed_kernel=11) as g:
            g.set_state(c)
            for _ in range(calls):
                g.advance(0.1, steps)
            out.append(g.get_state())
    assert np.array_equal(out[0], out[1])
