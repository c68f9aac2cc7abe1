"""With the limiter the autotuner keeps one kernel family per order at every mesh
size (its shapes agree bit for bit, so what was timed changes no result), and
each order's family is as close to the plain FP64 form at shocks as the other."""
import numpy as np
import pytest

import wasl_b200
from wasl_b200 import cases, meshgen

pytestmark = pytest.mark.gpu
PATCH = range(9, 13)  # tuning values of the patch kernel's shapes
REFERENCE = {1: 2, 2: 11, 3: 2}  # mixed_kernel of one shape of the order's family


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n", [4, 33, 190])  # 32, 2,178 and 72,200 triangles
def test_one_family_per_order(p, n):
    arrays = meshgen.jittered_box(n, jitter=0.15, seed=n + p)
    out = []
    for kernel in (0, REFERENCE[p]):
        with wasl_b200.Solver(*arrays, polynomial_order=p, precision="mixed", limiting=True,
                              positivity_all=True, mixed_kernel=kernel) as g:
            cases.project_initial(g, cases.QuadrantRiemann(seed=2).conserved)
            g.limit()
            for _ in range(3):
                g.step(g.stable_dt(0.1))
            assert (g.tuning()[0] in PATCH) == (p == 2)
            out.append(g.get_state())
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_families_are_equally_close_to_fp64(p, seed):
    """Errors against the plain form, tile and patch family: the mean within 1.5x of
    one another, the largest within 3x (rounding differences that the limiter's
    weights amplify)."""
    arrays = meshgen.jittered_box(40, jitter=0.15, seed=200 + p)
    out = {}
    for kernel in (0, 2, 11):
        kw = dict(precision="mixed", mixed_kernel=kernel) if kernel else {}
        with wasl_b200.Solver(*arrays, polynomial_order=p, limiting=True, positivity_all=True,
                              boundary="transmissive", **kw) as g:
            cases.project_initial(g, cases.QuadrantRiemann(seed=seed).conserved)
            g.limit()
            for _ in range(4):
                g.step(g.stable_dt(0.1))
            out[kernel] = g.get_state()
    tile, patch = np.abs(out[2] - out[0]), np.abs(out[11] - out[0])
    for a, b in ((tile, patch), (patch, tile)):
        assert np.mean(a) <= 1.5 * np.mean(b) + 1e-12
        assert np.max(a) <= 3.0 * np.max(b) + 1e-12
