"""The one-pass ghost fill and the edge EMFs that map their own boundary indices:
every cell of the padded arrays, ghosts and corners included, against the
oracle's three sequential fills, for grids down to one and two cells an axis
and every kind of side."""
import numpy as np
import pytest

from cumc3d_b200 import models

pytestmark = pytest.mark.gpu

CASES = [
    # nx, ny, nz, n_dim, geometry, flags, periodic-face option
    (7, 5, 4, 3, 0, (0, 0, 0, 0, 0, 0), 0),
    (7, 5, 4, 3, 0, (0, 0, 0, 0, 0, 0), 1),
    (3, 3, 3, 3, 0, (2, 2, 2, 2, 2, 2), 0),
    (5, 4, 3, 3, 0, (1, 2, 0, 0, 2, 1), 1),
    (6, 5, 4, 3, 0, (2, 1, 4, 1, 1, 4), 0),
    (2, 1, 2, 3, 0, (0, 0, 1, 1, 0, 0), 1),
    (1, 2, 1, 3, 0, (1, 1, 0, 0, 1, 1), 0),
    (9, 6, 1, 2, 0, (2, 2, 0, 0, 1, 1), 0),
    (6, 2, 1, 2, 0, (0, 0, 1, 1, 0, 0), 1),
    (11, 1, 1, 1, 0, (2, 1, 1, 1, 1, 1), 0),
    (5, 1, 1, 1, 0, (0, 0, 0, 0, 0, 0), 0),
    (40, 4, 35, 3, 0, (1, 1, 0, 0, 1, 1), 0),
]


@pytest.mark.parametrize("nx,ny,nz,nd,geo,flags,fixn", CASES)
def test_padded_state_equals_the_sequential_fills(oracle_mod, nx, ny, nz, nd, geo, flags, fixn):
    from cumc3d_b200.engine import Solver
    spec, prim, eps = models.smooth_state(nx, ny, nz, nd, coordinate_flag=geo, boundary_flag=flags, seed=3, recon="ppm",
                                          fix_periodic_normal_faces=fixn)
    out = []
    for s in (Solver(spec), oracle_mod.Oracle(spec)):
        s.set_state(prim, eps)
        s.initial_update()
        for _ in range(2):
            dt = s.finddt()
            (s.rungekutta if hasattr(s, "rungekutta") else s.rk3_step)(dt)
        out.append(s.get_state() + (dt,))
    (pg, eg, dg), (po, eo, do) = out
    assert dg == do
    assert np.array_equal(pg, po, equal_nan=True)
    assert np.array_equal(eg, eo, equal_nan=True)
