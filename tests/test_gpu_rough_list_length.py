"""The mixed form's second pass takes lanes for a short list and threads for a long
one: the same bits for an element whatever the length of the list it is on, and
both against the plain FP64 form."""
import numpy as np
import pytest

import wasl_b200
from test_gpu_rough_pass import jumping_state
from wasl_b200 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [2, 11])  # tile and patch family
@pytest.mark.parametrize("boundary", ["periodic", "transmissive"])
# (lists are long from 12,000, 18,000 and 24,000 elements on, on meshes of six times that)
@pytest.mark.parametrize("p,nx,ny", [(1, 371, 100), (2, 451, 121), (3, 481, 151)])
@pytest.mark.parametrize("rule", [0, -1])
def test_same_bits_on_short_and_long_lists(kernel, boundary, p, nx, ny, rule):
    """Most of the domain smooth (a short list) or jumping (a long one); the left
    end's elements, three stages away from it, do not depend on which.
    Tolerance against the plain form: one step moves the state by about CFL x |u|;
    the perturbations are FP32 sums of at most 256 rounded terms of that size."""
    cfl = 0.2
    tags, xy, el = meshgen.jittered_box(nx, jitter=0.1, seed=nx, ny=ny)
    nodes = {int(t): i for i, t in enumerate(tags)}
    corner = np.vectorize(nodes.get)(np.asarray(el).reshape(-1, 3))
    x = np.asarray(xy).reshape(-1, 2)[corner, 0].mean(axis=1)
    jumping = jumping_state(len(x), p, p).reshape(4, -1, len(x))
    smooth = jumping.copy()
    smooth[:, 0, x > 0.12] = np.sqrt(2.0) * np.array([1.0, 0.0, 0.0, 2.5])[:, None]
    inner = (x > 0.03) & (x < 0.09)
    out = {}
    for name, c in (("long", jumping), ("short", smooth)):
        for form, k in (("mixed", kernel), ("plain", 0)):
            with wasl_b200.Solver(tags, xy, el, polynomial_order=p, boundary=boundary,
                                  precision=form, limiting=True, sensor_threshold=1e30,
                                  mixed_kernel=k,
                                  volume_rule_order=rule if k else 0) as g:
                g.set_state(c.ravel())
                dt = out.setdefault("dt", g.stable_dt(cfl))
                g.step(dt)
                out[name, form] = g.get_state().reshape(c.shape)
        if rule == 0:  # (the plain form's rule)
            assert (np.max(np.abs(out[name, "mixed"] - out[name, "plain"]))
                    <= 256 * 2.0 ** -24 * cfl * np.max(np.abs(c)))
    assert np.array_equal(out["long", "mixed"][:, :, inner], out["short", "mixed"][:, :, inner])


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("kernel", [2, 8, 11])
def test_conserves_in_supersonic_flow(p, kernel):
    """Every branch of the flux at the faces between the two passes' elements: mass
    and energy of a periodic run with supersonic quadrants are kept to round-off."""
    from wasl_b200 import cases
    arrays = meshgen.jittered_box(130, jitter=0.15, seed=9)
    rng = np.random.Generator(np.random.PCG64(1))
    states = np.stack([cases.conserved(rng.uniform(0.5, 1.5), *rng.uniform(-3, 3, 2),
                                       rng.uniform(0.3, 1.5)) for _ in range(4)])
    with wasl_b200.Solver(*arrays, polynomial_order=p, limiting=True, positivity_all=True,
                          precision="mixed", mixed_kernel=kernel) as g:
        cases.project_initial(g, lambda x, y: states[(np.asarray(x) >= 0.5).astype(int)
                                                     + 2 * (np.asarray(y) >= 0.5).astype(int)])
        g.limit()
        m0, e0 = g.mass_energy()
        for _ in range(5):
            g.step(g.stable_dt(0.05))
        m1, e1 = g.mass_energy()
    assert abs(m1 - m0) <= 1e-13 * abs(m0) and abs(e1 - e0) <= 1e-13 * abs(e0)


@pytest.mark.parametrize("p,nx,ny", [(1, 371, 100), (2, 451, 121), (3, 481, 151)])
def test_long_lists_in_a_batch(p, nx, ny):
    """Two cases of one order, which share a list: the single-case solver's bits."""
    arrays = [meshgen.jittered_box(nx, jitter=0.1, seed=s, ny=ny) for s in (1, 2)]
    states = [jumping_state(2 * nx * ny, p, p + s) for s in (1, 2)]
    kw = dict(limiting=True, sensor_threshold=1e30, boundary="transmissive")
    with wasl_b200.Batch([(*a, p) for a in arrays], tile_shape=1, **kw) as b:
        for c, state in enumerate(states):
            b.set_state(c, state)
        b.advance(0.2, 1)
        got = [b.get_state(c) for c in range(2)]
    for c, a in enumerate(arrays):
        with wasl_b200.Solver(*a, polynomial_order=p, precision="mixed", mixed_kernel=2,
                              volume_rule_order=p, **kw) as g:
            g.set_state(states[c])
            g.advance(0.2, 1)
            assert np.array_equal(got[c], g.get_state())
