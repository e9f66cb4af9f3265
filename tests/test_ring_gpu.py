"""A ring of z slabs whose periodic normal faces are not refilled
(fix_periodic_normal_faces 0): at the seam the exchange leaves the normal face
field out, so its x and y ghost columns on the seam's ghost planes are the
engine's own to fill.  Against the undivided grid, ghost planes and columns
included, from an upload whose ghosts are not already what the boundary rules
give."""
import numpy as np
import pytest

from cumc3d_b200 import capi, engine, models

pytestmark = pytest.mark.gpu


def _problem(xy, n=(11, 9, 15)):
    spec, prim, eps = models.smooth_state(*n, 3, boundary_flag=xy + (0, 0), recon="weno", riemann="hlld", seed=8)
    inside = np.zeros(prim.shape[:3], dtype=bool)
    inside[3:-3, 3:-3, 3:-3] = True
    rng = np.random.Generator(np.random.PCG64(17))
    prim[~inside] *= rng.uniform(0.9, 1.1, (int((~inside).sum()), 8))
    return spec, prim, eps


@pytest.mark.parametrize("sizes", [(8, 7), (5, 6, 4)])
@pytest.mark.parametrize("xy", [(0, 0, 0, 0), (1, 1, 2, 2)])
def test_seam_planes_carry_the_undivided_ghosts(xy, sizes):
    spec, prim, eps = _problem(xy)
    assert not spec.get("fix_periodic_normal_faces", 0)
    nz = spec["nz"]
    g, s = engine.SlabGroup(spec, sizes), engine.Solver(spec)
    for q in (g, s):
        q.set_state(prim, eps)
        q.initial_update()
    for step in range(3):
        whole, _ = s.get_state()
        lower, _ = g.slabs[0].get_state()
        upper, _ = g.slabs[-1].get_state()
        assert np.array_equal(lower[:3], whole[:3]), step
        assert np.array_equal(upper[-3:], whole[nz + 3:]), step
        # the index-0 layer of the conserved face fields is taken from them
        cons, lower_cons = s.get_array(capi.ARR_CONS), g.slabs[0].get_array(capi.ARR_CONS)
        assert np.array_equal(lower_cons[2, 2:-3, 2:-3, 5:], cons[2, 2:-3, 2:-3, 5:]), step
        dt = s.finddt()
        assert g.finddt() == dt
        g.step(dt)
        s.rungekutta(dt)
    g.close()
    s.close()


def test_captured_step_of_a_slab_follows_its_seam():
    """A slab stepped by itself before it joins a ring keeps no step captured
    with its old z sides."""
    spec, prim, eps = _problem((0, 0, 0, 0))
    out = []
    for alone in (4, 0):
        g = engine.SlabGroup(spec, (8, 7))
        g.set_state(prim, eps)
        if alone:
            for s in g.slabs:
                s.initial_update()
                for _ in range(alone):
                    s.rungekutta(1e-4)
            g.set_state(prim, eps)
        g.initial_update()
        for s in g.slabs:
            s.rungekutta(1e-3)
        out.append([s.get_state() + (s.get_array(capi.ARR_CONS),) for s in g.slabs])
        g.close()
    inner = (slice(3, -3),) * 3
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x[inner], y[inner])
