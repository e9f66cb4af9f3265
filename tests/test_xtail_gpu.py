"""FP64 WENO-Z staged tiles: the x sweep's columns beyond the last whole 32-cell
tile share blocks.  Every bit of the state against the per-cell kernel, where
the remainder of nx + 2 is 0, 1, 2, 31 or the whole row and where the rows end
inside a block."""
import numpy as np
import pytest

from cumc3d_b200 import engine, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [4, 8, 29, 30, 31, 32, 61, 94])
@pytest.mark.parametrize("ny,nz", [(4, 5), (17, 4), (49, 6)])
def test_staged_tiles_equal_the_per_cell_kernel(nx, ny, nz):
    spec, prim, eps = models.blast_3d(nx, nx=nx, ny=ny, nz=nz)
    spec["positivity_fallback"] = 1
    spec["fix_periodic_normal_faces"] = 1
    out = []
    for tile in (0, 1, 2, 4):
        s = engine.Solver(spec)
        s.set_state(prim, eps)
        s.fallback_count(1)
        s.initial_update()
        s.set_tuning(True, 256, 128, 4, tile)
        s.evolve(1e30, 2)
        out.append((*s.get_state(), s.fallback_count()))
        s.close()
    for p, e, n in out[1:]:
        assert np.array_equal(p.view(np.uint64), out[0][0].view(np.uint64))
        assert np.array_equal(e.view(np.uint64), out[0][1].view(np.uint64))
        assert n == out[0][2]
