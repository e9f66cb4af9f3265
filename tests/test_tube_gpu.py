"""The batched engine's shared-memory kernel at the edges of its sizes: problems
that fill a CTA, a cluster of 2, 4, 8 and 16 exactly, one cell more or less, the
smallest ones, and beyond the largest cluster, in a small batch (CTAs of 126
cells) and in one that fills the device (254); every bit against the persistent
kernel, whose launch shape cumc_batch_set_cluster selects."""
import numpy as np
import pytest

from cumc3d_b200 import models

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 3, 7, 125, 126, 127, 252, 253, 254, 255, 504, 505, 508, 509, 1008, 1016, 1017, 2016, 2017, 2032, 2033]
LARGE = [4064, 4065]


def _specs(sizes, recon, riemann, precision, t_end):
    params = models.batch_problems(len(sizes), seed=11)
    return [models.riemann_1d(n, p["left"], p["right"], p["bx"], recon=recon, riemann=riemann, precision=precision,
                              t_end=t_end) for n, p in zip(sizes, params)]


def _run(probs, cluster, max_steps):
    from cumc3d_b200.engine import BatchSolver
    b = BatchSolver([p[0] for p in probs], positivity_fallback=1)
    if cluster:
        b.set_cluster(*cluster)
    for i, (_, prim, eps) in enumerate(probs):
        b.set_state(i, prim, eps)
    out = [b.run(max_steps, check=False)]
    out.append(b.run(max_steps, check=False))   # a second run goes on from the first one's state
    states = [b.get_state(i) for i in range(len(probs))]
    b.close()
    return out, states


@pytest.mark.parametrize("sizes,recon,riemann,precision", [
    (EDGES, "ppm", "hlld", "fp64"),
    (EDGES + LARGE, "weno", "hlld", "fp64"),
    (EDGES, "weno", "hllc", "fp32"),
    ([4, 600], "tvdvl", "lf", "fp32"),
    ([n for n in EDGES for _ in range(12)] + LARGE, "tvdmc", "hll", "fp64"),
])
def test_cluster_sizes_keep_the_bits(sizes, recon, riemann, precision):
    probs = _specs(sizes, recon, riemann, precision, t_end=0.05)
    (a, sa), (b, sb) = _run(probs, None, 6), _run(probs, (8, 64), 6)
    for x, y in zip(a, b):
        for p, q in zip(x, y):
            assert np.array_equal(p, q)
    for (pa, ea), (pb, eb) in zip(sa, sb):
        assert np.array_equal(pa, pb, equal_nan=True)
        assert np.array_equal(ea, eb, equal_nan=True)
