"""Self-gravity iterations, two launches each, replayed sixteen at a time: every
bit of phi, the count and the error against the oracle where the iteration
limit meets the end of a chunk and where the grid ends inside a CTA's rows."""
import numpy as np
import pytest

from cumc3d_b200 import engine, models
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(24, 16, 12), (33, 7, 9), (8, 5, 4), (65, 9, 6)])
@pytest.mark.parametrize("limit", [1, 2, 16, 17, 18, 33, 34])
def test_limit_against_the_chunks_of_iterations(dims, limit):
    spec, prim, eps = models.star_sph(*dims)
    s = engine.Solver(spec)
    s.set_state(prim, eps)
    s.poisson_setup(spec["rho_atm"], 1.9)
    it, err, conv = s.poisson_solve(max_iter=limit, tol=1e-14)
    phi = s.poisson_get()
    s.close()
    po, ito, erro, convo = O.poisson_solve(spec, prim[3:-3, 3:-3, 3:-3, 0], spec["rho_atm"], omega=1.9, tol=1e-14,
                                           max_iter=limit)
    assert (it, conv) == (ito, convo)
    # (from phi = 0 the first relative changes are 0 / 0: a NaN's sign is not compared)
    assert err == erro or (np.isnan(err) and np.isnan(erro))
    assert np.array_equal(phi.view(np.uint64), po.view(np.uint64)), int((phi != po).sum())
