"""The list of deferred HLLD faces on a handle that has one (above 131072 cells):
some faces on it, more than it holds, and none, through the split and the fused
kernels, concurrent sweeps and the step graph; bit for bit the oracle's."""
import numpy as np
import pytest

from cumc3d_b200 import models

from parity_util import assert_bitwise, interior

pytestmark = pytest.mark.gpu

N, STEPS = (57, 52, 49), 2      # 145236 cells, odd extents


def _problem(kind):
    spec, prim, eps = models.smooth_state(*N, 3, recon="weno", riemann="hlld", seed=5, fix_periodic_normal_faces=1,
                                          positivity_fallback=1)
    rng = np.random.Generator(np.random.PCG64(7))
    shape = prim.shape[:3]
    x = np.arange(shape[2])[None, None, :] * np.ones(shape)
    # fields that decay to nothing along x, through every decade: on every row, or
    # on the first few
    rows = {"smooth": 0, "few": 8, "many": shape[1]}[kind]
    for v in (1, 2, 3, 5, 6, 7):
        decay = rng.choice([-1.0, 0.0, 1.0], shape) * 10.0 ** (-6.0 * x - rng.uniform(0, 20, shape))
        prim[:, :rows, :, v] = decay[:, :rows]
    eps = prim[..., 4] / prim[..., 0] / (spec["model"]["gamma"] - 1.0)
    return spec, prim, np.ascontiguousarray(eps)


@pytest.fixture(scope="module")
def problems(oracle_mod):
    out = {}

    def get(kind):
        if kind not in out:
            spec, prim, eps = _problem(kind)
            o = oracle_mod.Oracle(spec)
            o.set_state(prim, eps)
            o.initial_update()
            t, n = o.evolve(1e30, STEPS)
            p, e = o.get_state()
            assert np.isfinite(interior(p, spec)).all()
            out[kind] = spec, prim, eps, t, dict(prim=p, eps=e)
            o.close()
        return out[kind]
    return get


@pytest.mark.parametrize("path", ["split", "fused", "sweeps", "host"])
@pytest.mark.parametrize("kind", ["few", "many", "smooth"])
def test_deferred_faces_keep_the_bits(problems, kind, path):
    from cumc3d_b200.engine import Solver
    spec, prim, eps, t, want = problems(kind)
    s = Solver(spec)
    if path == "fused":
        s.set_tuning(0, 256, 128, 1, 0)
    elif path == "sweeps":
        s.set_concurrent_sweeps(True)
    s.set_state(prim, eps)
    s.initial_update()
    if path == "host":
        time = 0.0
        for _ in range(STEPS):
            dt = s.finddt()
            s.rungekutta(dt)
            time += dt
    else:
        time, _ = s.evolve(1e30, STEPS)
    assert time == t
    p, e = s.get_state()
    most, capacity = s.deferred_faces()
    assert 0 < capacity < 3 * N[0] * N[1] * N[2]
    if kind == "few":
        assert 0 < most <= capacity
    elif kind == "many":
        assert most > capacity
    else:
        assert most == 0
    assert_bitwise(dict(prim=p, eps=e), want, spec, what=("prim", "eps"))
    assert s.deferred_faces() == (0, capacity)
    s.close()


def test_no_list_on_a_small_grid():
    from cumc3d_b200.engine import Solver
    spec, prim, eps = models.blast_3d(12)
    s = Solver(spec)
    assert s.deferred_faces() == (0, 0)
    s.close()


@pytest.mark.parametrize("recon", ["ppm", "tvdmm"])
def test_spherical_torus_below_the_general_size(oracle_mod, recon):
    """84,320 cells, whose limited reconstruction leaves many faces for good."""
    from cumc3d_b200.engine import Solver
    spec, prim, eps = models.torus_sph(nr=62, ntheta=34, nphi=40, recon=recon)
    spec["fix_periodic_normal_faces"] = 1
    spec["positivity_fallback"] = 1
    s, o = Solver(spec), oracle_mod.Oracle(spec)
    for q in (s, o):
        q.set_state(prim, eps)
        q.initial_update()
    assert s.evolve(1e30, 20) == o.evolve(1e30, 20)
    most, capacity = s.deferred_faces()
    assert 0.1 * 84320 < most <= capacity
    (p, e), (po, eo) = s.get_state(), o.get_state()
    assert_bitwise(dict(prim=p, eps=e), dict(prim=po, eps=eo), spec, what=("prim", "eps"))
    s.close()
    o.close()
