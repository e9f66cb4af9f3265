"""Slabs large enough for the list of deferred HLLD faces and beyond the size
from which an undivided handle's kernels are launched programmatically
dependent: two slabs of more than 131072 cells and 200000 padded cells, against
the undivided grid bit for bit, ghost planes at the cut included."""
import numpy as np
import pytest

from cumc3d_b200 import capi, engine, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zflags", [(0, 0), (1, 1)])
def test_large_slabs_bitwise(zflags):
    sizes = (49, 50)
    spec, prim, eps = models.smooth_state(63, 55, 99, 3, boundary_flag=(0, 0, 1, 1) + zflags, recon="weno",
                                          riemann="hlld", seed=3, fix_periodic_normal_faces=1)
    # fields that decay to nothing across the grid: some faces go on the list
    decay = 10.0 ** (-6.0 * np.arange(prim.shape[2]))[None, None, :, None]
    prim[..., 1:4] *= decay
    prim[..., 5:8] *= decay
    g1 = spec["model"]["gamma"] - 1.0
    eps = np.ascontiguousarray(prim[..., 4] / prim[..., 0] / g1)
    g, s = engine.SlabGroup(spec, sizes), engine.Solver(spec)
    for q in (g, s):
        q.set_state(prim, eps)
        q.initial_update()
    for _ in range(4):
        dt = s.finddt()
        assert g.finddt() == dt
        g.step(dt)
        s.rungekutta(dt)
    whole, cons = s.get_state()[0], s.get_array(capi.ARR_CONS)
    for slab, o, m in zip(g.slabs, g.offsets, g.sizes):
        part = slab.get_state()[0]
        assert np.array_equal(part[:, 3:-3, 3:-3], whole[o:o + m + 6, 3:-3, 3:-3])
        assert np.array_equal(slab.get_array(capi.ARR_CONS)[3:-3, 3:-3, 3:-3], cons[o + 3:o + m + 3, 3:-3, 3:-3])
    g.close()
    s.close()
