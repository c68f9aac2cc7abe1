"""Listed positivity takes a warp per element on a short list and a thread on a long
one (more than 8,192 suspects): both as the plain form, which tests every element."""
import numpy as np
import pytest

from test_gpu_limited_shapes import plain_result, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [2, 8, 11])  # tile, shared-face and patch kernels
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("nx,ny", [(110, 100), (130, 110)])  # 7,333 and 9,533 low elements
def test_short_and_long_lists(oracle, kernel, p, nx, ny):
    """Tolerance as there: the forms' stage combinations differ by their roundings."""
    arrays, c, expected = plain_result(oracle, p, nx, ny)
    limited = (np.abs(expected - c) > 0.01).any((0, 1)).sum()
    assert limited >= nx * ny * 2 // 3
    with solver(arrays, p, precision="mixed", mixed_kernel=kernel) as g:
        g.set_state(c)
        g.step(1e-200)
        got = g.get_state().reshape(c.shape)
    assert np.max(np.abs(got - expected)) <= 1e-12
