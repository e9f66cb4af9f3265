"""The branch-free FP64 WENO-Z and HLLD (csrc/fast64.cuh) on the operands where
they hand over to the plain forms: tails that decay through every decade to
zero (subnormals, underflowing products), huge and uniform values, densities
with an all-ones mantissa, still gas without a normal field.  The engine's bits
must be the oracle's, whichever arithmetic a cell or face took, also when more
faces are deferred than the list holds."""
import numpy as np
import pytest

from cumc3d_b200 import models

from parity_util import assert_bitwise, interior, run_pair

pytestmark = pytest.mark.gpu


def _state(kind, recon, n=(21, 9, 10)):
    spec, prim, eps = models.smooth_state(*n, 3, recon=recon, riemann="hlld", seed=5, fix_periodic_normal_faces=1,
                                          positivity_fallback=1)
    rng = np.random.Generator(np.random.PCG64(7))
    shape = prim.shape[:3]
    x = np.arange(shape[2])[None, None, :] * np.ones(shape)
    g1 = spec["model"]["gamma"] - 1.0
    if kind == "tails":          # each cell 10^-10 of the one before: products pass through 1e-323
        for v in (1, 2, 3, 5, 6, 7):
            prim[..., v] = rng.choice([-1.0, 0.0, 1.0], shape) * 10.0 ** (-14.0 * x - rng.uniform(0, 20, shape))
    elif kind == "underflow":    # every product of two fields is subnormal or zero: the list overflows
        for v in (1, 2, 3, 5, 6, 7):
            prim[..., v] = rng.choice([-1.0, 1.0], shape) * 10.0 ** rng.uniform(-163, -140, shape)
    elif kind == "ones":         # uniform, density one ulp below 1: power-of-two quotients over all ones
        prim[..., 0] = 1.0 - 2.0 ** -53
        prim[..., 4] = 1.0
        prim[..., 1:4] = 0.0
        prim[..., 5:8] = 0.5
        prim[3:-3, 3:-3, 6:9, 0] = 1.0
        prim[3:-3, 4:6, 3:-3, 4] = 2.0
    elif kind == "still":        # no normal field, equal states, a pressure jump along z
        prim[..., 0] = 1.0
        prim[..., 1:8] = 0.0
        prim[..., 5] = 0.3
        prim[..., 4] = np.where(np.arange(shape[0])[:, None, None] < shape[0] // 2, 1.0, 0.25)
    elif kind == "scaled":       # far from unity: densities of 1e-17, then pressures beyond the tested range
        prim[..., 0] *= 1e-17
        prim[..., 4] *= np.where(x < 12, 1e-17, 1e-26)
        prim[..., 5:8] *= 1e-9
    eps = prim[..., 4] / prim[..., 0] / g1
    return spec, prim, np.ascontiguousarray(eps)


@pytest.mark.parametrize("recon", ["weno", "ppm"])
@pytest.mark.parametrize("kind", ["tails", "underflow", "ones", "still", "scaled"])
def test_bits_of_the_oracle_on_extreme_operands(oracle_mod, kind, recon):
    spec, prim, eps = _state(kind, recon)
    gpu, orc, dg, do = run_pair(spec, prim, eps, 2, oracle_mod)
    assert dg == do
    assert np.isfinite(interior(orc["prim"], spec)).all()
    assert_bitwise(gpu, orc, spec)


@pytest.mark.parametrize("kind", ["tails", "ones"])
def test_bits_through_the_step_graph(oracle_mod, kind):
    spec, prim, eps = _state(kind, "weno", n=(33, 8, 9))
    gpu, orc, dg, do = run_pair(spec, prim, eps, 3, oracle_mod, use_evolve=True, t_end=1e30)
    assert dg == do
    assert_bitwise(gpu, orc, spec)
