"""Self-gravity solves whose last iterations are launched one by one instead of
replayed (up to 8 of them): limits on both sides of that line and of the first
replays, and convergence inside either, against the oracle bit for bit."""
import numpy as np
import pytest

from cumc3d_b200 import engine, models
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(11, 6, 8), (12, 7, 9)])
@pytest.mark.parametrize("limit,tol", [(3, 0.0), (9, 0.0), (10, 0.0), (25, 0.0), (26, 0.0), (81, 0.0), (89, 0.0),
                                       (90, 0.0), (9, 0.5), (9, 1e6), (25, 0.1), (500, 0.1), (500, 1e-4)])
def test_limits_and_tolerances(dims, limit, tol):
    spec, prim, eps = models.star_sph(*dims)
    guess = -np.random.Generator(np.random.PCG64(6)).uniform(0.5, 2.0, (dims[2] + 2, dims[1] + 2, dims[0] + 2))
    s = engine.Solver(spec)
    s.set_state(prim, eps)
    s.poisson_setup(spec["rho_atm"], 1.5)
    for _ in range(2):          # the second solve goes on from the first one's potential
        s.poisson_set(guess)
        it, err, conv = s.poisson_solve(max_iter=limit, tol=tol)
        phi = s.poisson_get()
        po, ito, erro, convo = O.poisson_solve(spec, prim[3:-3, 3:-3, 3:-3, 0], spec["rho_atm"], omega=1.5, tol=tol,
                                               max_iter=limit, phi=guess)
        assert (it, err, conv) == (ito, erro, convo)
        assert np.array_equal(phi.view(np.uint64), po.view(np.uint64)), int((phi != po).sum())
        guess = po
    s.close()
