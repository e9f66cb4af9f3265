"""Handles on both sides of the sizes from which their stage kernels are launched
programmatically dependent (80,000 cells in 1D and 2D, 100,000 in 3D, 131072 in
3D FP32): the bits of the same handle with concurrent sweeps, which turn it off,
through the step graph and through host-driven steps."""
import numpy as np
import pytest

from cumc3d_b200 import capi, engine, models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [
    ((79999, 1, 1), "fp64"), ((80000, 1, 1), "fp64"), ((80001, 1, 1), "fp32"),
    ((283, 282, 1), "fp64"), ((284, 283, 1), "fp64"), ((284, 283, 1), "fp32"),
    ((47, 46, 46), "fp64"), ((47, 47, 46), "fp64"), ((47, 47, 46), "fp32"), ((51, 51, 51), "fp32"),
])
def test_same_bits_on_both_sides(n, precision):
    dim = 1 if n[1] == 1 else 2 if n[2] == 1 else 3
    spec, prim, eps = models.smooth_state(*n, dim, recon="ppm", precision=precision, fix_periodic_normal_faces=1, seed=9)
    out = []
    for concurrent in (False, True):
        s = engine.Solver(spec)
        s.set_concurrent_sweeps(concurrent)
        s.set_state(prim, eps)
        s.initial_update()
        t = [s.evolve(1e30, 3)]
        for _ in range(4):
            t.append(s.finddt())
            s.rungekutta(t[-1])
        out.append((t, s.get_state() + (s.get_array(capi.ARR_CONS), s.get_array(capi.ARR_CS))))
        s.close()
    (ta, a), (tb, b) = out
    assert ta == tb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
