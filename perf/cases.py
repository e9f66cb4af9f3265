"""The engine's timed cases: whole calls of its public API as a simulation makes them.

A pass of a grid case is one run of ``engine.Solver``: upload of the initial
model from page-locked host memory, INITIAL_UPDATE, the time loop, download of
the final state.  The time loop is ``evolve`` (on the device), or for
``loop = "host"`` the reference's own loop, FINDDT and RUNGEKUTTA called step
by step.  A pass of a batch case does the same for many 1D problems through
``engine.BatchSolver``; a pass of a gravity case re-solves the potential from
a given guess.  Every pass starts from the same inputs, so it can be repeated.

What a program keeps between runs (the handle, its tuning, its host buffers)
is made in ``prepare``.
"""
import math
import random

import numpy as np
import torch

from cumc3d_b200 import models

#: counted operations of one zone-update (one zone, one RK3 step and its
#: FINDDT), by dimensions and reconstruction; HLLD, an add, a multiplication, a
#: division or a root each one operation (profiles/op_counts.json).  A sweep's
#: reconstruction and Riemann solve are a third of the 3D figures' flux part.
FLOPS_3D = {"weno": 16600.0, "ppm": 9580.0, "tvdmc": 6400.0}
REST = 800.0


def listed():
    """The cases, from one shock tube to the 256^3 blast."""
    return [
        # a coupling code or a debugging run: a tiny tube, the host's own loop
        dict(name="tube_100_hostloop", kind="grid", model="tube", nx=100, ny=1, nz=1, recon="ppm", riemann="hlld",
             precision="fp64", steps=20, loop="host", tuned=False, learned=False),
        # the Brio-Wu test at its usual size on the grid engine: latency of the step
        dict(name="tube_800", kind="grid", model="tube", nx=800, ny=1, nz=1, recon="ppm", riemann="hlld",
             precision="fp64", steps=200, loop="device", tuned=False, learned=False),
        # a parameter study of 1D problems of uneven size, each to its end time
        dict(name="batch_64", kind="batch", count=64, nmin=128, nmax=2048, t_end=0.05, recon="ppm", riemann="hlld",
             precision="fp64"),
        # the same in single precision with the other reconstruction
        dict(name="batch_160_weno_fp32", kind="batch", count=160, nmin=100, nmax=1000, t_end=0.05, recon="weno",
             riemann="hlld", precision="fp32"),
        # a 2D test problem (Orszag-Tang)
        dict(name="vortex_256x256", kind="grid", model="vortex", nx=256, ny=256, nz=1, recon="ppm", riemann="hlld",
             precision="fp64", steps=60, loop="device", tuned=False, learned=False),
        # a 3D blast as a first production run is made: no tuning, odd extents
        dict(name="blast_101x96x90", kind="grid", model="blast", nx=101, ny=96, nz=90, recon="weno", riemann="hlld",
             precision="fp64", steps=16, loop="device", tuned=False, learned=False),
        # the headline workload: 256^3 blast, WENO-Z + HLLD + CT, tuned
        dict(name="blast_256", kind="grid", model="blast", nx=256, ny=256, nz=256, recon="weno", riemann="hlld",
             precision="fp64", steps=12, loop="device", tuned=True, learned=False),
        # smooth MHD waves in a periodic box, PPM
        dict(name="waves_128_ppm", kind="grid", model="waves", nx=128, ny=128, nz=128, recon="ppm", riemann="hlld",
             precision="fp64", steps=16, loop="device", tuned=True, learned=False),
        # the same in the FP32 form, WENO-Z
        dict(name="waves_160_weno_fp32", kind="grid", model="waves", nx=160, ny=160, nz=160, recon="weno",
             riemann="hlld", precision="fp32", steps=16, loop="device", tuned=True, learned=False),
        # cylindrical torus: floors, source terms, outflow and clamps
        dict(name="torus_96x64x96", kind="grid", model="torus_cyl", nx=96, ny=64, nz=96, recon="weno", riemann="hlld",
             precision="fp64", steps=24, loop="device", tuned=True, learned=False),
        # spherical torus, pole to pole on its refined grid, as the model ships (PPM)
        dict(name="torus_sph_124x44x128", kind="grid", model="torus_sph", nx=124, ny=44, nz=128, recon="ppm",
             riemann="hlld", precision="fp64", steps=24, loop="device", tuned=True, learned=False),
        # the self-gravity solve of the collapsar model on its grid
        dict(name="gravity_156x44x128", kind="gravity", nx=156, ny=44, nz=128, iters=400),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, its options, and sizes over the listed ranges."""
    kind = rng.choice(["tube", "batch", "vortex", "blast", "blast", "waves", "waves", "torus", "torus_sph", "gravity"])
    recon = rng.choice(["weno", "ppm", "weno", "ppm", "tvdmc"])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    riemann = rng.choice(["hlld", "hlld", "hlld", "hllc", "hll"])
    base = dict(kind="grid", recon=recon, riemann=riemann, precision=precision, loop="device", learned=False)
    if kind == "tube":
        host = rng.random() < 0.5
        return dict(base, model="tube", nx=_log(rng, 40, 4000), ny=1, nz=1, steps=rng.randint(10, 60) * (1 if host else 4),
                    loop="host" if host else "device", tuned=False)
    if kind == "batch":
        return dict(kind="batch", count=_log(rng, 8, 200), nmin=64 + rng.randint(0, 64), nmax=_log(rng, 400, 2000),
                    t_end=0.01 * rng.randint(2, 5), recon=recon, riemann=riemann, precision=precision)
    if kind == "vortex":
        return dict(base, model="vortex", nx=_log(rng, 48, 600), ny=_log(rng, 48, 600), nz=1, steps=rng.randint(20, 60),
                    tuned=rng.random() < 0.3)
    if kind in ("blast", "waves"):
        learned = kind == "waves" and recon == "weno" and rng.random() < 0.4
        return dict(base, model=kind, nx=_log(rng, 24, 180), ny=_log(rng, 24, 180), nz=_log(rng, 24, 180),
                    riemann="hlld" if learned else riemann, steps=rng.randint(8, 16), tuned=rng.random() < 0.5,
                    learned=learned)
    if kind == "torus":
        return dict(base, model="torus_cyl", nx=_log(rng, 48, 160), ny=_log(rng, 16, 96), nz=_log(rng, 48, 160),
                    recon=rng.choice(["weno", "ppm"]), riemann="hlld", steps=rng.randint(10, 24), tuned=rng.random() < 0.5)
    if kind == "torus_sph":
        return dict(base, model="torus_sph", nx=_log(rng, 48, 140), ny=_log(rng, 20, 60), nz=_log(rng, 48, 140),
                    recon="ppm", riemann="hlld", steps=rng.randint(10, 24), tuned=rng.random() < 0.5)
    return dict(kind="gravity", nx=_log(rng, 48, 384), ny=_log(rng, 32, 128), nz=_log(rng, 64, 160),
                iters=rng.randint(100, 400))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _box(nx, ny, nz, n_dim, flags, lo, hi, **kw):
    return dict(nx=nx, ny=ny, nz=nz, n_dim=n_dim, coordinate_flag=0, boundary_flag=list(flags),
                xF=models.faces(lo, hi, nx), yF=models.faces(lo, hi, ny), zF=models.faces(lo, hi, nz), **kw)


def _tube_sides(rng):
    def side():
        return [math.exp(rng.uniform(math.log(0.1), math.log(10.0))), rng.uniform(-0.5, 0.5), rng.uniform(-1, 1),
                rng.uniform(-1, 1), math.exp(rng.uniform(math.log(0.1), math.log(10.0))), 0.0, rng.uniform(-2, 2),
                rng.uniform(-2, 2)]
    left, right = side(), side()
    left[5] = right[5] = rng.uniform(-1, 1)
    return left, right


def _tube(nx, rng, case):
    """One 1D Riemann problem on [0, 1] (gamma 5/3), states as the batched workload draws them."""
    spec = _box(nx, 1, 1, 1, (1,) * 6, 0.0, 1.0, cfl=0.8, recon=case["recon"], riemann=case["riemann"],
                precision=case["precision"], model=dict(gamma=5.0 / 3.0, floor="eps"), t_end=case.get("t_end", 0.1),
                positivity_fallback=1)
    left, right = _tube_sides(rng)
    x = models.centers(spec["xF"])
    row = np.where((x <= 0.5)[:, None], np.array(left), np.array(right))
    prim = np.broadcast_to(row, (7, 7) + row.shape).copy()
    eps = prim[..., 4] / prim[..., 0] / (5.0 / 3.0 - 1.0)
    return spec, prim, eps


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid_xyz(spec, dev):
    c = [torch.from_numpy(models.centers(spec[k])).to(dev) for k in ("xF", "yF", "zF")]
    f = [torch.from_numpy(np.asarray(spec[k])[1:].copy()).to(dev) for k in ("xF", "yF", "zF")]
    view = ((1, 1, -1), (1, -1, 1), (-1, 1, 1))
    return [a.view(v) for a, v in zip(c, view)], [a.view(v) for a, v in zip(f, view)]


def _blast(case, rng):
    """The periodic MHD blast (p 10 inside r = 0.1, 0.1 outside, oblique field),
    with the strength and the ambient density varied by the seed."""
    spec = _box(case["nx"], case["ny"], case["nz"], 3, (0,) * 6, -0.5, 0.5, cfl=0.4, recon=case["recon"],
                riemann=case["riemann"], precision=case["precision"], model=dict(gamma=5.0 / 3.0, floor="eps"),
                fix_periodic_normal_faces=1, positivity_fallback=1)
    dev = _device()
    (x, y, z), _ = _grid_xyz(spec, dev)
    r = torch.sqrt(x * x + y * y + z * z)
    prim = torch.zeros(tuple(r.shape) + (8,), dtype=torch.float64, device=dev)
    prim[..., 0] = rng.uniform(0.9, 1.1)
    prim[..., 4] = torch.where(r <= 0.1, rng.uniform(8.0, 12.0), rng.uniform(0.08, 0.12))
    prim[..., 5] = prim[..., 6] = 1.0 / math.sqrt(2.0)
    return spec, prim, prim[..., 4] / prim[..., 0] / (5.0 / 3.0 - 1.0)


def _waves(case, rng):
    """A periodic box of smooth MHD waves around a uniform field (seeded modes;
    face B is the curl of an edge-centred vector potential)."""
    spec = _box(case["nx"], case["ny"], case["nz"], 3, (0,) * 6, 0.0, 1.0, cfl=0.4, recon=case["recon"],
                riemann=case["riemann"], precision=case["precision"], learned=int(case["learned"]),
                model=dict(gamma=5.0 / 3.0, floor="eps"), fix_periodic_normal_faces=1)
    dev = _device()
    c, f = _grid_xyz(spec, dev)
    tau = 2.0 * math.pi
    modes = [([rng.randint(-2, 2) for _ in range(3)], [rng.uniform(0.0, tau) for _ in range(8)],
              [rng.uniform(-1.0, 1.0) for _ in range(8)]) for _ in range(4)]

    def field(q, x, y, z, amp):
        out = torch.zeros(torch.broadcast_shapes(x.shape, y.shape, z.shape), dtype=torch.float64, device=dev)
        for k, ph, a in modes:
            out += amp * a[q] * torch.cos(tau * (k[0] * x + k[1] * y + k[2] * z) + ph[q])
        return out

    h = [(a[1:] - a[:-1]).mean().item() for a in (t.flatten() for t in f)]
    prim = torch.zeros(tuple(field(0, *c, 1.0).shape) + (8,), dtype=torch.float64, device=dev)
    prim[..., 0] = 1.0 + field(0, *c, 0.02)
    for v in range(3):
        prim[..., 1 + v] = field(1 + v, *c, 0.05)
    prim[..., 4] = 0.3 + field(4, *c, 0.01)
    b0 = (0.6, 0.5, 0.4)
    for v in range(3):  # B_v = d_a A_b - d_b A_a on the faces of axis v
        a, b = (v + 1) % 3, (v + 2) % 3

        def at(q, axis, sign):
            p = [f[i] if i == v else c[i] for i in range(3)]
            p[axis] = p[axis] + sign * 0.5 * h[axis]
            return field(5 + q, *p, 0.02)
        prim[..., 5 + v] = b0[v] + (at(b, a, 1) - at(b, a, -1)) / h[a] - (at(a, b, 1) - at(a, b, -1)) / h[b]
    return spec, prim, prim[..., 4] / prim[..., 0] / (5.0 / 3.0 - 1.0)


def _vortex(case, rng):
    """The Orszag-Tang vortex, its velocity scaled by the seed."""
    spec, prim, eps = models.riemann_2d(15, case["nx"], case["ny"], recon=case["recon"], riemann=case["riemann"],
                                        precision=case["precision"])
    prim[..., 1:4] *= rng.uniform(0.9, 1.1)
    return spec, prim, eps


def _problem(case, seed):
    """(spec, prim, eps) of a grid case; prim and eps as torch tensors."""
    rng = random.Random(int(seed))
    if case["model"] == "tube":
        spec, prim, eps = _tube(case["nx"], rng, case)
    elif case["model"] == "vortex":
        spec, prim, eps = _vortex(case, rng)
    elif case["model"] == "blast":
        return _blast(case, rng)
    elif case["model"] == "waves":
        return _waves(case, rng)
    elif case["model"] == "torus_cyl":
        spec, prim, eps = models.torus_cyl(case["nx"], case["ny"], case["nz"], recon=case["recon"],
                                           riemann=case["riemann"], precision=case["precision"], seed=seed)
        spec["fix_periodic_normal_faces"] = 1
        spec["positivity_fallback"] = 1
    else:
        refined = (case["nx"], case["ny"], case["nz"]) == (124, 44, 128)
        size = {} if refined else dict(nr=case["nx"], ntheta=case["ny"], nphi=case["nz"])
        spec, prim, eps = models.torus_sph(recon=case["recon"], riemann=case["riemann"], precision=case["precision"],
                                           seed=seed, **size)
        spec["fix_periodic_normal_faces"] = 1
        spec["positivity_fallback"] = 1
    return spec, torch.from_numpy(np.ascontiguousarray(prim)), torch.from_numpy(np.ascontiguousarray(eps))


def _pinned(t):
    out = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    return out.copy_(t)


def prepare(case, seed):
    """The handle, its tuning and the host buffers a program holds before a run."""
    from cumc3d_b200 import engine
    if case["kind"] == "batch":
        rng, sizes = random.Random(int(seed)), random.Random(case["count"])  # one study's sizes, new states
        probs = [_tube(_log(sizes, case["nmin"], case["nmax"]), rng, case) for _ in range(case["count"])]
        return dict(case=case, b=engine.BatchSolver([p[0] for p in probs], positivity_fallback=1),
                    states=[(p[1], p[2]) for p in probs])
    if case["kind"] == "gravity":
        spec, prim, eps = models.star_sph(case["nx"], case["ny"], case["nz"], seed=seed)
        s = engine.Solver(spec)
        s.set_state(prim, eps)
        s.poisson_setup(spec["rho_atm"], 1.9)
        return dict(case=case, s=s, guess=_guess(case, seed))
    spec, prim, eps = _problem(case, seed)
    s = engine.Solver(spec)
    prim, eps = _pinned(prim), _pinned(eps)
    st = dict(case=case, s=s, prim=prim, eps=eps, out_prim=torch.empty_like(prim, pin_memory=True),
              out_eps=torch.empty_like(eps, pin_memory=True))
    if case["tuned"] or case["learned"]:
        s.set_state_ptr(prim.data_ptr(), eps.data_ptr())
        s.initial_update()
        if case["learned"]:
            s.learn_set(np.load("cumc3d_b200/data/flag_mlp.npy"), threshold=-4.0, audit_interval=24, audit_tol=1e-5,
                        flag_interval=8)
        if case["tuned"]:
            s.autotune()
    return st


def _guess(case, seed):
    """The potential a re-solve starts from: about -M/r with a seeded ripple."""
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    r = models.centers(models.faces(2.0, 40.0, case["nx"]))[2:-2]
    phi = np.broadcast_to(-40.0 / r, (case["nz"] + 2, case["ny"] + 2, case["nx"] + 2)) * 1.0
    return phi * (1.0 + 1e-3 * (rng.random(phi.shape) - 0.5))


def run(state):
    """One whole run through the public API."""
    case = state["case"]
    if case["kind"] == "batch":
        b = state["b"]
        for p, (prim, eps) in enumerate(state["states"]):
            b.set_state(p, prim, eps)
        t, steps, _ = b.run()  # raises where a problem ends in a bad state
        out = [b.get_state(p) for p in range(case["count"])]
        return dict(prim=np.concatenate([o[0] for o in out]), eps=np.concatenate([o[1] for o in out]), t=t, steps=steps)
    s = state["s"]
    if case["kind"] == "gravity":
        s.poisson_set(state["guess"])
        n, err, _ = s.poisson_solve(max_iter=case["iters"], tol=1e-10)
        return dict(phi=s.poisson_get(), n=n, err=err)
    s.set_state_ptr(state["prim"].data_ptr(), state["eps"].data_ptr())
    s.initial_update()
    if case["loop"] == "host":
        t = 0.0
        for _ in range(case["steps"]):
            dt = s.finddt()
            s.rungekutta(dt)
            t = t + dt
    else:
        s.time = 0.0
        t, _ = s.evolve(1e30, case["steps"])
    s.get_state_ptr(state["out_prim"].data_ptr(), state["out_eps"].data_ptr())
    return dict(prim=state["out_prim"], eps=state["out_eps"], t=t)


def work(case):
    """Bytes and operations of a pass.  A step reads and writes the eight
    conserved variables once a stage and the saved state twice: 512 B a zone."""
    if case["kind"] == "gravity":
        cells = float(case["nx"] * case["ny"] * case["nz"])
        return dict(bytes=cells * (16.0 + 56.0 * case["iters"]), flops=cells * 18.0 * case["iters"])
    if case["kind"] == "batch":
        # mean of n and of n^2 over the log-uniform sizes; a zone is crossed in
        # about 1/15 of a time unit at CFL 0.8 (the median problem's fast speed)
        lo, hi = float(case["nmin"]), float(case["nmax"])
        ln = math.log(hi / lo)
        n1, n2 = (hi - lo) / ln, (hi * hi - lo * lo) / (2.0 * ln)
        updates = case["count"] * n2 * case["t_end"] * 8.0
        return dict(bytes=case["count"] * n1 * 144.0, flops=updates * (FLOPS_3D[case["recon"]] / 3.0 + REST))
    zones = float(case["nx"] * case["ny"] * case["nz"])
    dims = 1 + (case["ny"] > 1) + (case["nz"] > 1)
    per = (FLOPS_3D[case["recon"]] - REST) * dims / 3.0 + REST
    resident = zones * 8.0 * 8.0 * 2.0 < 100e6  # a state and its saved copy that stay in L2
    return dict(bytes=zones * (144.0 + (0.0 if resident else 512.0 * case["steps"])), flops=zones * case["steps"] * per)


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    """The outputs of ``run`` in 64 bits for the Cartesian grids with PPM or
    WENO-Z and HLLD and for the gravity solve.  None for the batches (each
    problem's thousands of steps would take minutes here), the curvilinear
    grids (their model hooks would have to be written a second time) and the
    other schemes."""
    if case["kind"] == "gravity":
        return _exact_gravity(case, seed)
    if case["kind"] == "batch" or case["model"] in ("torus_cyl", "torus_sph"):
        return None
    if case["recon"] not in ("ppm", "weno") or case["riemann"] != "hlld":
        return None
    if case["nx"] * case["ny"] * case["nz"] * case["steps"] > 3e8:
        return None
    spec, prim, eps = _problem(case, seed)
    m = _Plain(spec, prim.to(_device()), eps.to(_device()))
    t = m.evolve(case["steps"])
    return dict(prim=m.prim().cpu(), eps=m.eps.cpu(), t=t)


def _exact_gravity(case, seed):
    """Red-black SOR of the spherical Poisson equation, omega 1.9."""
    spec, prim, _ = models.star_sph(case["nx"], case["ny"], case["nz"], seed=seed)
    dev = _device()
    x, y, z = (torch.from_numpy(models.centers(spec[k])).to(dev) for k in ("xF", "yF", "zF"))
    r, th, ph = x[2:-2].view(1, 1, -1), y[2:-2].view(1, -1, 1), z[2:-2].view(-1, 1, 1)   # cells 0..n+1

    def near(a, axis):
        m = a.shape[axis]
        return a.narrow(axis, 0, m - 2), a.narrow(axis, 1, m - 2), a.narrow(axis, 2, m - 2)
    (rm, rc, rp), (tm, tc, tp), (pm, pc, pp) = near(r, 2), near(th, 1), near(ph, 0)
    ty, s2 = torch.tan(tc), torch.sin(tc) ** 2
    eps = (2 * (rp + rm - 3 * rc) / rc / (rp - rc) / (rc - rm)
           + (tp + tm - 2 * tc - 2 * ty) / rc ** 2 / ty / (tp - tc) / (tc - tm) - 2 / rc ** 2 / s2 / (pp - pc) / (pc - pm))
    a1, a0 = (2 * (2 * rc - rm) / (rp - rm) / (rp - rc) / rc, 2 * (2 * rc - rp) / (rp - rm) / (rc - rm) / rc)
    b1 = (2 * ty + tc - tm) / rc ** 2 / ty / (tp - tc) / (tp - tm)
    b0 = (2 * ty + tc - tp) / rc ** 2 / ty / (tp - tm) / (tc - tm)
    c1, c0 = 2 / rc ** 2 / s2 / (pp - pm) / (pp - pc), 2 / rc ** 2 / s2 / (pp - pm) / (pc - pm)
    rho = torch.from_numpy(np.ascontiguousarray(prim[3:-3, 3:-3, 3:-3, 0])).to(dev)
    src = 4 * math.pi * torch.where(rho - spec["rho_atm"] > 0, rho, torch.zeros_like(rho))
    phi = torch.from_numpy(_guess(case, seed)).to(dev)
    nz, ny, nx = rho.shape
    par = (torch.arange(1, nz + 1, device=dev).view(-1, 1, 1) + torch.arange(1, ny + 1, device=dev).view(1, -1, 1)
           + torch.arange(1, nx + 1, device=dev).view(1, 1, -1)) % 2
    n = 0
    for n in range(1, case["iters"] + 1):
        old = phi[1:-1, 1:-1, 1:-1].clone()
        for colour in (0, 1):
            p = phi[1:-1, 1:-1, 1:-1]
            s = a1 * phi[1:-1, 1:-1, 2:] + a0 * phi[1:-1, 1:-1, :-2] + b1 * phi[1:-1, 2:, 1:-1] + b0 * phi[1:-1, :-2, 1:-1]
            s = s + c1 * phi[2:, 1:-1, 1:-1] + c0 * phi[:-2, 1:-1, 1:-1]
            p.copy_(torch.where(par == colour, -0.9 * p + 1.9 * ((src - s) / eps), p))
        i = slice(1, -1)
        phi[i, i, 0], phi[i, i, -1] = phi[i, i, 1], -1.0
        phi[i, 0, i], phi[i, -1, i] = phi[i, 1, i], phi[i, -2, i]
        phi[0, i, i], phi[-1, i, i] = phi[-2, i, i], phi[1, i, i]
        err = torch.max(torch.abs((phi[i, i, i] - old) / old)).item()
        if err <= 1e-10:
            break
    return dict(phi=phi.cpu(), n=n, err=err)


class _Plain:
    """The finite-volume CT scheme on a Cartesian grid with periodic and outflow
    sides: reconstruction, HLLD, constrained transport, SSP-RK3, on padded
    arrays indexed [z, y, x] with three ghost cells a side."""

    def __init__(self, spec, prim, eps):
        self.spec, self.nd = spec, spec["n_dim"]
        self.n = (spec["nx"], spec["ny"], spec["nz"])
        self.g = spec["model"]["gamma"]
        self.fixn, self.fallback = spec.get("fix_periodic_normal_faces", 0), spec.get("positivity_fallback", 0)
        self.P = [prim[..., v].clone() for v in range(8)]
        self.eps = eps.clone()
        z = torch.zeros_like(self.eps)
        self.z, self.cs, self.BC = z, z.clone(), [z.clone() for _ in range(3)]
        self.dev = eps.device
        self.d = [torch.from_numpy(np.diff(np.asarray(spec[k]))).to(self.dev) for k in ("xF", "yF", "zF")]
        self.dv = [a.view(v) for a, v in zip(self.d, ((1, 1, -1), (1, -1, 1), (-1, 1, 1)))]
        self.w = [self._weights(a) for a in self.d]
        self.U = [z.clone() for _ in range(8)]
        I = self._cells((1, 1, 1), self.n)
        self.eps[I] = torch.clamp(self.eps[I], min=0.0)
        self.from_prim(I, [self.P[5 + a] for a in range(3)])
        for v in range(3):
            self.U[5 + v][I] = self.P[5 + v][I]
        self.low_faces()
        self.fill(self.state_arrays)

    def prim(self):
        return torch.stack(self.P, dim=-1)

    @staticmethod
    def _cells(lo, hi):
        """Slices of the cells lo..hi (reference numbering, axes x, y, z)."""
        return tuple(slice(lo[a] + 2, hi[a] + 3) for a in (2, 1, 0))

    @staticmethod
    def _moved(I, axis, by):
        s = list(I)
        a = 2 - axis
        s[a] = slice(s[a].start + by, s[a].stop + by)
        return tuple(s)

    def state_arrays(self, axis):
        out = self.P[:5] + self.BC + [self.P[5 + i] for i in range(3) if i != axis] + [self.cs, self.eps]
        return out + ([self.P[5 + axis]] if self.fixn and self.spec["boundary_flag"][2 * axis] == 0 else [])

    def emf_arrays(self, axis):
        f = self.EF
        return self.EC + [f[k] for k in (("xz", "xy", "yz", "zy"), ("xz", "yx", "yz", "zx"), ("xy", "yx", "zx", "zy"))[axis]]

    def fill(self, arrays):
        for axis in range(3):
            n, a, flags = self.n[axis], 2 - axis, self.spec["boundary_flag"][2 * axis:2 * axis + 2]
            for arr in arrays(axis):
                for g in (1, 2, 3):
                    for dst, flag, edge in ((1 - g, flags[0], 1), (n + g, flags[1], n)):
                        src = (dst - 1) % n + 1 if flag == 0 else edge
                        arr.select(a, dst + 2).copy_(arr.select(a, src + 2))

    def low_faces(self):
        for axis in range(3):
            hi = list(self.n)
            hi[axis] = 0
            I = self._cells((0, 0, 0), hi)
            for v in (5, 6, 7):
                self.U[v][I] = self.P[v][I]

    def from_prim(self, I, low):
        """Cell B from the faces (low: the arrays that hold the lower ones), the
        conserved state, the pressure and the sound speed."""
        for a in range(3):
            self.BC[a][I] = 0.5 * (self.P[5 + a][I] + low[a][self._moved(I, a, -1)])
        rho, v, b, e = self.P[0][I], [p[I] for p in self.P[1:4]], [c[I] for c in self.BC], self.eps[I]
        v2, b2 = sum(q * q for q in v), sum(q * q for q in b)
        self.U[0][I] = rho
        for a in range(3):
            self.U[1 + a][I] = rho * v[a]
        self.U[4][I] = rho * (e + 0.5 * v2) + 0.5 * b2
        p = rho * e * (self.g - 1)
        self.P[4][I] = p
        self.cs[I] = torch.sqrt(e * (self.g - 1) + rho * (self.g - 1) * p / (rho * rho))

    def _weights(self, d):
        """Per-cell interpolation weights for the cells 0..n+1 (rows), from the spacings."""
        m = d.numel() - 4
        m2, m1, c, p1, p2 = (d[i:i + m] for i in range(5))
        if self.spec["recon"] == "weno":
            a12, a01, a10, a21 = p2 / (p1 + p2), p1 / (c + p1), c / (m1 + c), m1 / (m2 + m1)
            return [1 - a01, a01, 1 - a12, a12, 1 - a10, a10, 1 - a21, a21, 1 - a21, a12]
        xr, xl = m1 + c + p1 + p2, m2 + m1 + c + p1
        ar, al = 2 * p1 * c / (p1 + c), 2 * c * m1 / (c + m1)
        z1r, z1l, zr, zl = (m1 + c) / (2 * c + p1), (m2 + m1) / (2 * m1 + c), (p2 + p1) / (2 * p1 + c), (p1 + c) / (2 * c + m1)
        return [m1 / (m1 + c), al * (z1l - zl) / xl, -m1 * z1l / xl, c * zl / xl,
                c / (c + p1), ar * (z1r - zr) / xr, -c * z1r / xr, p1 * zr / xr,
                m1 / (m2 + m1 + c) * (2 * m2 + m1) / (c + m1), m1 / (m2 + m1 + c) * (m1 + 2 * c) / (m2 + m1),
                c / (m1 + c + p1) * (2 * m1 + c) / (p1 + c), c / (m1 + c + p1) * (c + 2 * p1) / (m1 + c),
                p1 / (c + p1 + p2) * (2 * c + p1) / (p2 + p1), p1 / (c + p1 + p2) * (p1 + 2 * p2) / (c + p1)]

    def edges(self, axis, q, I):
        """Left and right edge values of the cells I."""
        w = [a.view([-1 if k == 2 - axis else 1 for k in range(3)]) for a in self.w[axis]]
        a, b, c, d, e = (q[self._moved(I, axis, s)] for s in (-2, -1, 0, 1, 2))
        if self.spec["recon"] == "ppm":
            def slope(lo, mid, hi, w0, w1):
                s = w0 * (hi - mid) + w1 * (mid - lo)
                lim = torch.minimum(s.abs(), 2 * torch.minimum((mid - lo).abs(), (hi - mid).abs()))
                return torch.where((hi - mid) * (mid - lo) > 0, lim * torch.sign(s), torch.zeros_like(s))
            dp, dc, dm = slope(c, d, e, w[12], w[13]), slope(b, c, d, w[10], w[11]), slope(a, b, c, w[8], w[9])
            right = c + (w[4] + w[5]) * (d - c) + w[6] * dp + w[7] * dc
            left = b + (w[0] + w[1]) * (c - b) + w[2] * dc + w[3] * dm
            flat = (right - c) * (c - left) <= 0
            lo = torch.where((right - left) * (left - 3 * c + 2 * right) < 0, 3 * c - 2 * right, left)
            hi = torch.where((right - lo) * (3 * c - 2 * left - right) < 0, 3 * c - 2 * left, right)
            return torch.where(flat, c, lo), torch.where(flat, c, hi)
        u01, u12, u10, u21 = w[0] * c + w[1] * d, w[2] * d + w[3] * e, w[4] * b + w[5] * c, w[6] * a + w[7] * b
        u00, u11 = b + w[8] * (b - a), d + w[9] * (d - e)

        def side(near, far, out, mid, last):
            """near: the mid value on the face's side; far: the other; out: the far extrapolation."""
            p = [(6 * c - far - 2 * out) / 3, (2 * c - far + 2 * near) / 3, (2 * near + 2 * mid - last) / 3]
            r = 13.0 / 12.0
            s = [4 * r * (far - out) ** 2 + (2 * c - far - out) ** 2, 4 * r * (far - 2 * c + near) ** 2 + (near - far) ** 2,
                 4 * r * (near - 2 * mid + last) ** 2 + (4 * mid - 3 * near - last) ** 2]
            tau5 = (s[0] - s[2]).abs()
            k = [gw * (1 + (tau5 / (1e-40 + b)) ** 2) for gw, b in zip((0.1, 0.6, 0.3), s)]
            return sum(x * y for x, y in zip(k, p)) / sum(k)
        return side(u10, u01, u11, b, u21), side(u01, u10, u00, d, u12)

    def sweep(self, axis):
        """Face fluxes of one direction on the faces 0..n; EMFs on the faces."""
        n, hi = self.n, list(self.n)
        lo = [1, 1, 1]
        lo[axis], hi[axis] = 0, n[axis] + 1
        C = self._cells(lo, hi)
        t = [i for i in range(3) if i != axis]
        src = self.P[:5] + [self.BC[t[0]], self.BC[t[1]]]
        ed = [self.edges(axis, q, C) for q in src]
        if self.fallback:
            bad = ~((ed[0][0] > 0) & (ed[0][1] > 0) & (ed[4][0] > 0) & (ed[4][1] > 0))
            ed = [tuple(torch.where(bad, q[C], x) for x in e) for q, e in zip(src, ed)]
        a, m = 2 - axis, n[axis] + 1
        L = [e[1].narrow(a, 0, m) for e in ed]
        R = [e[0].narrow(a, 1, m) for e in ed]
        hi[axis] = n[axis]
        F = self._cells(lo, hi)
        flux, fb = self.hlld(axis, t, L, R, self.P[5 + axis][F])
        for i in range(5):
            self.F[axis][i][F] = flux[i]
        x, y, zz = fb  # fluxes of Bx, By, Bz
        if axis == 0:
            self.EF["yx"][F], self.EF["zx"][F] = zz, -y
        elif axis == 1:
            self.EF["xy"][F], self.EF["zy"][F] = -zz, x
        else:
            self.EF["xz"][F], self.EF["yz"][F] = y, -x

    def hlld(self, axis, t, L, R, bn):
        g = self.g

        def side(q):
            rho, v, p = q[0], q[1:4], q[4]
            b = [None] * 3
            b[axis], b[t[0]], b[t[1]] = bn, q[5], q[6]
            b2, v2, vb = sum(c * c for c in b), sum(c * c for c in v), sum(c * d for c, d in zip(b, v))
            e = p / rho / (g - 1)
            u = [rho] + [rho * c for c in v] + [rho * (0.5 * v2 + e) + 0.5 * b2]
            pt, vn = p + 0.5 * b2, v[axis]
            f = [c * vn for c in u]
            for i in range(3):
                f[1 + i] = f[1 + i] - bn * b[i]
            f[1 + axis] = f[1 + axis] + pt
            f[4] = f[4] + pt * vn - bn * vb
            a2, bb = e * (g - 1) + rho * (g - 1) * p / rho ** 2, b2 / rho
            cf = torch.sqrt(0.5 * (a2 + bb + torch.sqrt(torch.clamp((a2 + bb) ** 2 - 4 * a2 * bn * bn / rho, min=0))))
            return dict(rho=rho, v=v, b=b, u=u + b, f=f + [vn * b[i] - v[i] * bn for i in range(3)], pt=pt, vn=vn, cf=cf, vb=vb)
        l, r = side(L), side(R)
        wl, wr = torch.sqrt(l["rho"]), torch.sqrt(r["rho"])
        ub, cb = (wl * l["vn"] + wr * r["vn"]) / (wl + wr), (wl * l["cf"] + wr * r["cf"]) / (wl + wr)
        sl, sr = torch.minimum(l["vn"] - l["cf"], ub - cb), torch.maximum(r["vn"] + r["cf"], ub + cb)
        dl, dr = l["rho"] * (sl - l["vn"]), r["rho"] * (sr - r["vn"])
        sm = (dr * r["vn"] - dl * l["vn"] + l["pt"] - r["pt"]) / (dr - dl)
        rl, rr = dl / (sl - sm), dr / (sr - sm)
        al, ar = sm - bn.abs() / torch.sqrt(rl), sm + bn.abs() / torch.sqrt(rr)
        weak = ((al - sl) < 1e-4 * (sm - sl)) | ((ar - sr) > -1e-4 * (sr - sm))
        al, ar = torch.where(weak, sm, al), torch.where(weak, sm, ar)

        def star(q, s, ds, rs):
            u, b, v, vs = q["u"], list(q["b"]), q["v"], [None] * 3
            us = [rs] + [c * (s - q["vn"]) / (s - sm) for c in u[1:5]]
            fac = ds * (s - sm) - bn * bn
            for i in t:
                hll = (sr * r["b"][i] - sl * l["b"][i] - (r["f"][5 + i] - l["f"][5 + i])) / (sr - sl)
                b[i] = torch.where(weak, hll, q["b"][i] * (ds * (s - q["vn"]) - bn * bn) / fac)
                us[1 + i] = us[1 + i] - (bn * b[i] - bn * q["b"][i]) / (s - sm)
                vs[i] = us[1 + i] / rs
            us[1 + axis], vs[axis] = rs * sm, sm
            ps = ds * (sm - q["vn"]) + q["pt"]
            vb = sum(c * d for c, d in zip(b, vs))
            us[4] = us[4] + ((ps * sm - q["pt"] * q["vn"]) - (vb - q["vb"]) * bn) / (s - sm)
            return us + b, vs, vb
        ul, vl, vbl = star(l, sl, dl, rl)
        ur, vr, vbr = star(r, sr, dr, rr)
        ql, qr, sg = torch.sqrt(rl), torch.sqrt(rr), torch.copysign(torch.ones_like(bn), bn)
        vv, bb = [None] * 3, [None] * 3
        vv[axis], bb[axis] = sm, bn
        for i in t:
            vv[i] = (ql * vl[i] + qr * vr[i] + (ur[5 + i] - ul[5 + i]) * sg) / (ql + qr)
            bb[i] = (ql * ur[5 + i] + qr * ul[5 + i] + torch.sqrt(rl * rr) * (vr[i] - vl[i]) * sg) / (ql + qr)
        vbb = sum(c * d for c, d in zip(vv, bb))
        ull = [rl] + [rl * c for c in vv] + [ul[4] - ql * (vbl - vbb) * sg] + bb
        urr = [rr] + [rr * c for c in vv] + [ur[4] + qr * (vbr - vbb) * sg] + bb
        out = []
        for i in range(8):
            fl, fr = l["f"][i] + sl * (ul[i] - l["u"][i]), r["f"][i] + sr * (ur[i] - r["u"][i])
            mid = torch.where(sm >= 0, fl + al * (ull[i] - ul[i]), fr + ar * (urr[i] - ur[i]))
            mid = torch.where(al >= 0, fl, torch.where(ar <= 0, fr, mid))
            out.append(torch.where(sl >= 0, l["f"][i], torch.where(sr <= 0, r["f"][i], mid)))
        return out[:5], out[5:]

    def stage(self, k, dt):
        I = self._cells((1, 1, 1), self.n)
        new = lambda: torch.zeros_like(self.z)  # noqa: E731
        self.F = [[new() for _ in range(5)] for _ in range(self.nd)]
        self.EF = {a: new() for a in ("yx", "zx", "xy", "zy", "xz", "yz")}
        self.EC = [new() for _ in range(3)]
        v, b = self.P[1:4], self.BC
        for a in range(3):
            p, q = (a + 1) % 3, (a + 2) % 3
            self.EC[a][I] = v[q][I] * b[p][I] - v[p][I] * b[q][I]
        for axis in range(self.nd):
            self.sweep(axis)
        comp = dict(x=0, y=1, z=2)
        for axis, names in ((1, ("xy", "zy")), (2, ("xz", "yz"))):
            if axis >= self.nd:  # a direction without cells takes the cell EMFs on both of its faces
                for f in names:
                    self.EF[f][I] = self.EC[comp[f[0]]][I]
                    self.EF[f][self._moved(I, axis, -1)] = self.EC[comp[f[0]]][I]
        self.fill(self.emf_arrays)
        E = [new() for _ in range(3)]
        J = self._cells((0, 0, 0), self.n)
        for c, (p, q) in enumerate(((1, 2), (0, 2), (0, 1))):
            fp, fq, e = self.EF["xyz"[c] + "xyz"[p]], self.EF["xyz"[c] + "xyz"[q]], self.EC[c]
            Jp, Jq = self._moved(J, p, 1), self._moved(J, q, 1)
            E[c][J] = (0.5 * (fp[J] + fp[Jq] + fq[J] + fq[Jp])
                       - 0.25 * (e[J] + e[Jq] + e[Jp] + e[self._moved(Jp, q, 1)]))
        dv = self.dv
        sl = lambda a, S: dv[a][S[0] if a == 2 else slice(None), S[1] if a == 1 else slice(None), S[2] if a == 0 else slice(None)]  # noqa: E731
        rate = [new() for _ in range(8)]
        for axis in range(self.nd):
            for i in range(5):
                f = self.F[axis][i]
                rate[i][I] -= (f[I] - f[self._moved(I, axis, -1)]) / sl(axis, I)
        for a in range(3):
            p, q = (a + 1) % 3, (a + 2) % 3
            rate[5 + a][J] = -((E[q][J] - E[q][self._moved(J, p, -1)]) / sl(p, J)
                               - (E[p][J] - E[p][self._moved(J, q, -1)]) / sl(q, J))
        if k == 1:
            self.U0 = [u.clone() for u in self.U]
        w = ((0.0, 1.0, 1.0), (0.75, 0.25, 0.25), (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0))[k - 1]
        for i in range(8):
            self.U[i][J] = w[0] * self.U0[i][J] + w[1] * self.U[i][J] + w[2] * dt * rate[i][J]
        # recovery: the velocity and the energy from the new state and faces
        b = [0.5 * (self.U[5 + a][I] + self.U[5 + a][self._moved(I, a, -1)]) for a in range(3)]
        rho = self.U[0][I]
        vel = [self.U[1 + a][I] / rho for a in range(3)]
        e = (self.U[4][I] - 0.5 * sum(c * c for c in b)) / rho - 0.5 * sum(c * c for c in vel)
        self.eps[I] = torch.clamp(e, min=0.0)
        self.P[0][I] = rho
        for a in range(3):
            self.P[1 + a][I] = vel[a]
            self.P[5 + a][I] = self.U[5 + a][I]
        self.from_prim(I, [self.P[5 + a] for a in range(3)])
        self.low_faces()
        self.fill(self.state_arrays)

    def finddt(self):
        I = self._cells((1, 1, 1), self.n)
        rho, a2, b = self.P[0][I], self.cs[I] ** 2, [c[I] for c in self.BC]
        b2 = sum(c * c for c in b) / rho
        lam = None
        for a in range(3):
            c = torch.sqrt(0.5 * (a2 + b2 + torch.sqrt((a2 + b2) ** 2 - 4 * a2 * b[a] * b[a] / rho)))
            c = c + self.P[1 + a][I].abs()
            lam = c if lam is None else torch.maximum(lam, c)
        h = min(self.d[a][3:-3].min().item() for a in range(self.nd))
        return min(1e5, (h * self.spec["cfl"] / lam).min().item())

    def evolve(self, steps):
        t = 0.0
        for _ in range(steps):
            dt = self.finddt()
            for k in (1, 2, 3):
                self.stage(k, dt)
            t += dt
        return t
