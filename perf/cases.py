"""Performance cases: what a user of the framework has it do, through its public entry points.

A pass is what a tsunami model's main loop does between two write-outs: some
time steps from the state that the GPU already holds, then a look at the
results.  The state (``Domain``, ``Batch``, ``Multidomain``) is made once, as a
model's setup makes it; further passes go on from where the last one ended.

    listed()            the cases, by name
    draw(rng)           another case of the same ranges
    prepare(case, seed) the model as set up, its initial state made from the seed
    run(state)          one pass, and the whole of its results
    exact(case, seed)   the same results in 64 bits, in plain torch
    work(case)          bytes and floating-point operations of a pass
"""
import ctypes
import functools
import math

import numpy as np
import torch

from ptha_b200 import Domain, Multidomain, _lib, workloads
from ptha_b200.batch import Batch
from ptha_b200.nesting import NestDomain

G, MAD, WALL = 9.8, 1.0e-5, 1.0e6
RADIUS, OMEGA = 6371000.0, 7.292115e-05
# the nested configuration's time-step refinement of its four domains
NEST_REFINEMENT = (1, 3, 9, 8)
SERIES = 8   # passes that a batch's gauge series holds
OCEAN = ("linear", "leapfrog_linear_plus_nonlinear_friction")
FV = ("rk2", "midpoint", "euler")


def _domain(name, method, nx, ny, steps, real_bytes=8, spherical=False, loop=False, gauges=0):
    return dict(name=name, kind="domain", method=method, nx=nx, ny=ny, steps=steps, real_bytes=real_bytes,
                spherical=spherical, loop=loop, gauges=gauges)


def listed():
    return [
        # A small inundation grid advanced step by step from the host's own
        # loop (the drop-in use of evolve_one_step): launches and latency.
        _domain("beach_small_step_calls", "rk2", 300, 200, 15, loop=True),
        # The 400 x 400 plain leapfrog with its nine gauges: a grid in L2.
        _domain("linear_400_gauges", "linear", 400, 400, 120, gauges=9),
        # A regional ocean at one arc minute, single precision, Coriolis.
        _domain("linear_ocean_fp32", "linear", 3600, 2400, 150, real_bytes=4, spherical=True),
        # The plain FP64 leapfrog on a grid far beyond L2.
        _domain("linear_4096", "linear", 4096, 4096, 120),
        # Linear leapfrog with Manning friction, the usual choice for long
        # ocean-wide runs; odd sizes.
        _domain("linear_friction_ocean", "leapfrog_linear_plus_nonlinear_friction", 1501, 1001, 100, spherical=True),
        # Nonlinear leapfrog over a wet/dry beach.
        _domain("leapfrog_nonlinear_beach", "leapfrog_nonlinear", 1024, 768, 60),
        # The 2048 x 2048 wet/dry beach with the CFL time step: the headline.
        _domain("rk2_beach_2048", "rk2", 2048, 2048, 30, gauges=9),
        # The same solver with FP32 state on a smaller, odd-sized grid.
        _domain("rk2_beach_fp32", "rk2", 1531, 1021, 30, real_bytes=4),
        # The midpoint method on a spherical coastal patch, fixed time step,
        # the size of a nested grid.
        _domain("midpoint_coast", "midpoint", 930, 930, 30, spherical=True),
        # Many earthquake sources on one ocean grid, advanced together, by
        # the kernel that the batch's own tuner picked.
        dict(name="batch_sources", kind="batch", nx=1800, ny=1200, count=12, steps=120, gauges=50, tuned=True),
        # Gradient of a gauge misfit for a source inversion (backward).
        dict(name="misfit_gradient", kind="adjoint", nx=1200, ny=800, steps=100, every=25, gauges=30),
        # The four-domain nest, three outer steps as one captured graph.
        dict(name="nested_4_domains", kind="nested", scale=1, replays=1),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["ocean", "ocean", "friction", "lfnl", "rk2", "rk2", "fv", "batch", "adjoint", "nested"])
    real_bytes = rng.choice([8, 8, 4])
    if kind in ("ocean", "friction"):
        n = size(200 * 150, 3800 * 3800)
        nx = max(100, min(n // 100, int(math.sqrt(n * rng.uniform(0.6, 2.0)))))
        return _nameless(_domain("", OCEAN[kind == "friction"], nx, n // nx, rng.choice([40, 75, 110]), real_bytes,
                                 rng.random() < 0.7, rng.random() < 0.2, rng.choice([0, 0, 9, 50])))
    if kind in ("rk2", "fv", "lfnl"):
        n = size(120 * 80, 2000 * 1900)
        nx = max(90, min(n // 70, int(math.sqrt(n * rng.uniform(0.6, 2.0)))))
        method = "rk2" if kind == "rk2" else "leapfrog_nonlinear" if kind == "lfnl" else rng.choice(FV)
        return _nameless(_domain("", method, nx, n // nx, rng.choice([12, 20, 30]), real_bytes,
                                 method != "leapfrog_nonlinear" and rng.random() < 0.4, rng.random() < 0.3,
                                 rng.choice([0, 9])))
    if kind == "batch":
        nx = size(300, 1800)
        return dict(kind="batch", nx=nx, ny=max(200, int(nx * rng.uniform(0.5, 0.66))), count=rng.randint(2, 12),
                    steps=rng.choice([40, 75, 110]), gauges=rng.choice([0, 20, 50]), tuned=rng.random() < 0.5)
    if kind == "adjoint":
        nx = size(240, 1200)
        return dict(kind="adjoint", nx=nx, ny=max(160, int(nx * rng.uniform(0.5, 0.66))), steps=rng.randint(40, 100),
                    every=rng.choice([20, 25, 33]), gauges=rng.randint(5, 30))
    scale = rng.choice([1, 3, 5, 15])
    return dict(kind="nested", scale=scale, replays=rng.randint(1, min(scale, 3)))


def _nameless(case):
    del case["name"]
    return case


# ------------------------------------------------------------------- inputs
def _waves(rng, X, Y, count, amplitude, longest):
    """A sum of `count` random sinusoids of wavelength `longest` and shorter on the grid X (row) x Y (column)."""
    out = np.zeros((Y.size, X.size))
    for _ in range(count):
        k = 2.0 * np.pi / (longest * rng.uniform(0.3, 1.0))
        a, p = rng.uniform(0.0, 2.0 * np.pi), rng.uniform(0.0, 2.0 * np.pi)
        kx, ky = k * np.cos(a), k * np.sin(a)
        # cos(kx x + ky y + p), as outer products
        out += amplitude / count * (np.outer(np.cos(ky * Y + p), np.cos(kx * X)) -
                                    np.outer(np.sin(ky * Y + p), np.sin(kx * X)))
    return out


def _ocean(nx, ny, spherical, seed, instances=1):
    """An ocean with islands behind walls, and `instances` uplift patterns: Domain arguments, elevation, stages."""
    rng = np.random.default_rng(seed)
    if spherical:
        dl = 60.0 / max(nx, 1.5 * ny)
        lw, ll = (nx * dl, ny * dl), (140.0, -45.0)
    else:
        lw, ll = (nx * 1000.0, ny * 1000.0), (0.0, 0.0)
    X, Y = np.arange(nx) / max(nx, ny), np.arange(ny) / max(nx, ny)
    elv = -3000.0 + _waves(rng, X, Y, 6, 6000.0, 0.7)
    elv = np.maximum(elv, -6500.0)
    elv[elv > -20.0] = 100.0
    elv[:2], elv[-2:], elv[:, :2], elv[:, -2:] = 100.0, 100.0, 100.0, 100.0
    kw = dict(nx=(nx, ny), lw=lw, lower_left=ll, spherical=spherical)
    return kw, elv, [np.where(elv < 0.0, _waves(rng, X, Y, 5, 3.0, 0.25), 0.0) for _ in range(instances)]


def _beach(nx, ny, spherical, seed):
    """A planar beach from -50 m to +10 m with bumps behind walls, a wave field on it and a solitary wave entering
    from the west (Cartesian grids): Domain arguments, elevation, stage, momenta."""
    rng = np.random.default_rng(seed)
    if spherical:
        dl = 1.0 / 180.0
        lw, ll = (nx * dl, ny * dl), (141.0, -39.0)
    else:
        lw, ll = (20480.0, 20480.0 * ny / nx), (0.0, 0.0)
    X, Y = (np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / nx
    elv = np.clip(-50.0 + 512.0 * (X - 0.83), -50.0, 10.0)[None, :] + _waves(rng, X, Y, 6, 2.0, 0.1)
    stage = _waves(rng, X, Y, 6, 1.5, 0.3)
    u, v = _waves(rng, X, Y, 4, 0.8, 0.4), _waves(rng, X, Y, 4, 0.4, 0.4)
    kw = dict(nx=(nx, ny), lw=lw, lower_left=ll, spherical=spherical)
    edge = (slice(None), 0), (slice(None), -1), (0, slice(None)), (-1, slice(None))
    if spherical:
        for e in edge:
            elv[e] = 100.0
    else:
        x0 = 0.5 * lw[0] / nx - 5.0 / math.sqrt(15.0 / (4.0 * 50.0 ** 3))
        kw.update(boundary_kind=_lib.BC_STAGE_TRANSMISSIVE_NORMAL_MOMENTUM,
                  boundary_function_kind=_lib.BF_SOLITARY_WEST_WALLS, boundary_function_params=(5.0, 50.0, x0))
        for e, z in zip(edge, (-50.0, WALL, WALL, WALL)):
            elv[e] = z
    stage = np.maximum(stage, elv)
    depth = stage - elv
    return kw, elv, stage, depth * u, depth * v


def _spacing(kw):
    """distance_bottom_edge, distance_left_edge, area, coriolis, coriolis at bottom edges, tan(lat)/R by row."""
    nx, ny = kw["nx"]
    dx, dy = kw["lw"][0] / nx, kw["lw"][1] / ny
    if not kw["spherical"]:
        one, z = np.ones(ny), np.zeros(ny)
        return dx * np.ones(ny + 1), dy, dx * dy * one, z, np.zeros(ny + 1), z
    d2r = math.pi / 180.0
    lat = (kw["lower_left"][1] + (np.arange(ny) + 0.5) * dy) * d2r
    edge = (kw["lower_left"][1] + np.arange(ny + 1) * dy) * d2r
    area = RADIUS ** 2 * np.cos(lat) * (dy * d2r) * (dx * d2r)
    return (dx * d2r * RADIUS * np.cos(edge), dy * d2r * RADIUS, area, 2.0 * OMEGA * np.sin(lat),
            2.0 * OMEGA * np.sin(edge), np.tan(lat) / RADIUS)


def _timestep(kw, depth, cfl):
    dxb, dyl = _spacing(kw)[:2]
    return cfl * min(float(dxb.min()), dyl) / math.sqrt(G * float(np.max(np.where(depth < 1.0e4, depth, 0.0))))


def _gauge_cells(kw, n, seed):
    """(n, 2) row and column of gauges, and their coordinates (cell centres)."""
    nx, ny = kw["nx"]
    rng = np.random.default_rng([seed, 7])
    c = np.stack([rng.integers(4, ny - 4, n), rng.integers(4, nx - 4, n)], axis=1)
    xy = np.stack([kw["lower_left"][0] + (c[:, 1] + 0.5) * kw["lw"][0] / nx,
                   kw["lower_left"][1] + (c[:, 0] + 0.5) * kw["lw"][1] / ny], axis=1)
    return c, xy


def _inputs(case, seed):
    """What a "domain" or "adjoint" case starts from: Domain arguments, U (4, ny, nx), dt or None (the CFL step)."""
    method = case.get("method", "linear")
    nx, ny, sph = case["nx"], case["ny"], case.get("spherical", True)
    U = np.zeros((4, ny, nx))
    if method in OCEAN:
        kw, U[3], (U[0],) = _ocean(nx, ny, sph, seed)
        dt = _timestep(kw, -U[3], 0.63)
    else:
        kw, U[3], U[0], U[1], U[2] = _beach(nx, ny, sph, seed)
        if method == "leapfrog_nonlinear":
            kw = {k: v for k, v in kw.items() if not k.startswith("boundary")}
        cfl = {"leapfrog_nonlinear": 0.5, "midpoint": 0.3, "euler": 0.25}.get(method)
        dt = cfl and _timestep(kw, U[0] - U[3], cfl)
    return dict(kw, timestepping_method=method, real_bytes=case.get("real_bytes", 8)), U, dt


@functools.lru_cache(maxsize=4)
def _nest_elevations(scale):
    specs, coasts = workloads.nested_specs(NEST_REFINEMENT, scale)
    md = Multidomain([NestDomain(s.lower_left, s.lw, s.nx, s.timestepping_method, s.timestepping_refinement_factor)
                      for s in specs], periodic_xs=(0.0, 360.0))
    return [workloads.nested_elevation(s, k, coasts) for k, s in enumerate(md.specs)]


def prepare(case, seed):
    if case["kind"] == "domain":
        kw, U, dt = _inputs(case, seed)
        d = Domain(**kw)
        d.set_U(U)
        if case["method"] != "linear":
            d.set_manning_squared(0.025 ** 2)
        if case["gauges"]:
            d.gauges_setup(_gauge_cells(kw, case["gauges"], seed)[1], case["steps"])
        peak = torch.empty((case["ny"], case["nx"]), dtype=torch.float64 if case["real_bytes"] == 8 else torch.float32,
                           pin_memory=True)
        return dict(case=case, domain=d, dt=dt, peak=peak)
    if case["kind"] == "batch":
        kw, elv, stages = _ocean(case["nx"], case["ny"], True, seed, case["count"])
        grid = Domain(**kw, timestepping_method="linear", real_bytes=4)
        grid.set_var(4, elv)
        b = Batch(grid, case["count"])
        U = np.zeros((1, 3) + elv.shape, dtype=np.float32)
        for q, s in enumerate(stages):
            U[0, 0] = s
            b.set_U(U, first=q)
        if case["tuned"]:
            b.tune()
        xy = _gauge_cells(kw, case["gauges"], seed)[1]
        if case["gauges"]:
            b.gauges_setup(xy, SERIES * case["steps"])
        peak = torch.empty((case["count"],) + elv.shape, dtype=torch.float32, pin_memory=True)
        return dict(case=case, batch=b, gauges=xy, passes=0, dt=_timestep(kw, -elv, 0.63), peak=peak)
    if case["kind"] == "adjoint":
        kw, U, dt = _inputs(case, seed)
        d = Domain(**kw)
        d.set_U(U)
        d.gauges_setup(_gauge_cells(kw, case["gauges"], seed)[1], case["steps"])
        return dict(case=case, domain=d, dt=dt, target=_target(case, seed))
    specs, coasts = workloads.nested_specs(NEST_REFINEMENT, case["scale"])
    md = Multidomain(specs, [dict(real_bytes=4 if k == 0 else 8, spherical=True) for k in range(4)],
                     periodic_xs=(0.0, 360.0))
    elv = _nest_elevations(case["scale"])
    for k, (s, d) in enumerate(zip(md.specs, md.domains)):
        d.set_U(workloads.nested_initial_state(s, k, coasts, source_seed=seed, elevation=elv[k]))
        if k:
            d.set_manning_squared(0.025 ** 2)
    dt = md.domains[0].linear_timestep_max()
    dt = 0.95 * min([dt] + [n * d.stationary_timestep_max() for n, d in zip(NEST_REFINEMENT, md.domains)][1:])
    md.capture_graph(3, dt)
    return dict(case=case, md=md)


def _target(case, seed):
    t = np.arange(case["steps"])[:, None]
    return 0.3 * np.sin(0.1 * t + np.random.default_rng([seed, 3]).uniform(0.0, 6.0, case["gauges"])[None, :])


# --------------------------------------------------------------------- pass
class _Plane:
    """Device memory of `owner` as torch takes it; a tensor made of it keeps the owner."""

    def __init__(self, owner, address, shape, strides, size):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(address, False), shape=shape, strides=tuple(size * s for s in strides),
                                             typestr="<f%d" % size, version=2)


def _state_planes(d):
    size = d.dtype().itemsize
    planes, pitch = d.device_planes()
    return [torch.as_tensor(_Plane(d, p, (d.nx[1], d.nx[0]), (pitch, 1), size), device="cuda") for p in planes[:3]]


def run(state):
    case = state["case"]
    if case["kind"] == "domain":
        d, dt, n = state["domain"], state["dt"], case["steps"]
        if case["gauges"]:
            d.gauges_reset()
        if case["loop"]:
            for _ in range(n):
                d.evolve_one_step(dt)
        else:
            d.evolve_steps(n, dt)
        _lib.check(_lib.lib().swals_gpu_download_max_stage(d.handle, ctypes.c_void_p(state["peak"].data_ptr())))
        out = dict(U=_state_planes(d), max_stage=state["peak"])
        if case["gauges"]:
            out["gauges"] = d.gauges_read()
        return out
    if case["kind"] == "batch":
        b = state["batch"]
        if case["gauges"] and state["passes"] == SERIES:   # the series is full: a new one
            b.gauges_setup(state["gauges"], SERIES * case["steps"])
            state["passes"] = 0
        state["passes"] += 1
        b.evolve(case["steps"], state["dt"])
        _lib.check(_lib.lib().swals_gpu_batch_download_max_stage(b._h, 0, case["count"],
                                                                 ctypes.c_void_p(state["peak"].data_ptr())))
        address, pitch, plane, stride = b.device_state()
        U = torch.as_tensor(_Plane(b, address, (case["count"], 3, case["ny"], case["nx"]), (stride, plane, pitch, 1), 4),
                            device="cuda")
        out = dict(U=U, max_stage=state["peak"])
        if case["gauges"]:
            out["gauges"] = b.gauges_read()[-case["steps"]:]
        return out
    if case["kind"] == "adjoint":
        loss, gradient = state["domain"].misfit_gradient(case["steps"], state["dt"], state["target"], case["every"])
        return dict(loss=loss, gradient=gradient)
    md = state["md"]
    md.replay(case["replays"])
    md.synchronize()
    return [_state_planes(d) for d in md.domains]


def _cells(case):
    if case["kind"] == "nested":
        sizes = ((5400, 1800), (900, 900), (1197, 801), (702, 1098))
        return [(nx // case["scale"]) * (ny // case["scale"]) * n for (nx, ny), n in zip(sizes, NEST_REFINEMENT)]
    return [case["nx"] * case["ny"]]


def work(case):
    """Per cell and step, the state in and out once, with the elevation, the friction coefficient and max_stage where
    the method has them; operations as the reference's statements have them."""
    if case["kind"] == "nested":
        c = _cells(case)
        n = 3 * case["replays"]
        return dict(bytes=n * (9 * 4 * c[0] + 10 * 8 * sum(c[1:])), flops=n * (30.0 * c[0] + 1050.0 * sum(c[1:])))
    n = _cells(case)[0] * case["steps"]
    if case["kind"] == "batch":
        return dict(bytes=4.0 * n * (8 * case["count"] + 1), flops=40.0 * n * case["count"])
    if case["kind"] == "adjoint":
        return dict(bytes=2.0 * 7 * 8 * n, flops=2.0 * 40 * n)
    planes, flops = {"linear": (9, 40), OCEAN[1]: (10, 90), "leapfrog_nonlinear": (10, 200)}.get(case["method"], (10, 1050))
    return dict(bytes=float(planes * case["real_bytes"] * n), flops=float(flops * n))


# --------------------------------------------------- the same in plain torch
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rows(kw):
    dxb, dyl, area, cor, cor_be, tan = _spacing(kw)
    col = [torch.as_tensor(a, device=_device())[:, None] for a in (dxb, area, cor, cor_be, tan)]
    return col[0], dyl, col[1], col[2], col[3], col[4]


def _shift(a, dj, di):
    """a[j + dj, i + di], the edge repeated."""
    j = torch.arange(a.shape[-2], device=a.device).add(dj).clamp(0, a.shape[-2] - 1)
    i = torch.arange(a.shape[-1], device=a.device).add(di).clamp(0, a.shape[-1] - 1)
    return a.index_select(-2, j).index_select(-1, i)


def _leapfrog(kw, elv, dt, nsq=None):
    """One step (stage, UH, VH) -> (stage, UH, VH) of the truly linear leapfrog, with Manning friction if nsq is given."""
    dxb, dyl, area, cor, cor_be, _ = _rows(kw)
    wet = elv < -MAD
    east, north = _shift(elv, 0, 1), _shift(elv, 1, 0)
    h_e = torch.where(wet & (east < -MAD), -0.5 * (east + elv), 0.0)
    h_n = torch.where(wet & (north < -MAD), -0.5 * (north + elv), 0.0)
    area_n = 0.5 * (area + torch.cat([area[1:], area[-1:]]))
    inner = torch.zeros_like(elv)
    inner[1:-1, 1:-1] = 1.0
    lower = torch.zeros_like(elv)
    lower[:-1, :-1] = 1.0
    if nsq is not None:
        work_e, work_n = (G * nsq * (-0.5 * (elv + z)).clamp_min(MAD) ** (-7.0 / 3.0) for z in (east, north))

    def step(s, u, v):
        div = (u - _shift(u, 0, -1)) * dyl + v * dxb[1:] - _shift(v, -1, 0) * dxb[:-1]
        s = s - inner * (dt / area) * div
        v_e = 0.5 * (_shift(v, -1, 0) + _shift(v, -1, 1) + v + _shift(v, 0, 1))
        u_n = 0.5 * (u + _shift(u, 0, -1) + _shift(u, 1, 0) + _shift(u, 1, -1))
        un = u - G * dt / area * h_e * (_shift(s, 0, 1) - s) * dyl + 0.5 * dt * cor * (h_e > 0) * v_e
        vn = v - G * dt / area_n * h_n * (_shift(s, 1, 0) - s) * dxb[1:] - 0.5 * dt * cor_be[1:] * (h_n > 0) * u_n
        if nsq is not None:
            un = un / (1.0 + dt * work_e * torch.sqrt(u * u + 0.25 * v_e * v_e))
            vn = vn / (1.0 + dt * work_n * torch.sqrt(v * v + 0.25 * u_n * u_n))
        return s, u + lower * (un - u), v + lower * (vn - v)

    return step


def _limited(lo, c, up, th):
    a, b = up - c, c - lo
    d = torch.minimum(a.abs(), b.abs()) * 0.5 * (torch.copysign(torch.ones_like(a), a) + torch.copysign(torch.ones_like(b), b)) * th
    e = torch.where(d == 0, 0.0, 0.5 * (a + b))
    return torch.where(d > 0, torch.minimum(e, d), torch.maximum(e, d))


def _fv_fluxes(kw, s, uh, vh, elv, theta, cfl):
    """DE1_low_fr_diffusion: the fixed-up state, the flux sums, the sources and the largest 1/dt."""
    dxb, dyl, area, cor, _, tan = _rows(kw)
    h = s - elv
    wet = h > MAD
    s, h = torch.where(h < 0, elv, s), h.clamp_min(0)
    uh, vh = torch.where(wet, uh, 0.0), torch.where(wet, vh, 0.0)
    u, v = torch.where(wet, uh / h, 0.0), torch.where(wet, vh / h, 0.0)
    flux, source, rate = [torch.zeros_like(s) for _ in range(3)], [torch.zeros_like(s), torch.zeros_like(s)], 0.0
    for axis in (0, 1):   # north-south edges, then east-west
        def to(a, k):
            return _shift(a, k, 0) if axis == 0 else _shift(a, 0, k)
        n = s.shape[axis]
        h3 = torch.stack([to(h, -1), h, to(h, 1)])
        th = (theta * (((h3.amin(0) - MAD) / (h3.amax(0) + 100.0 * MAD) - 0.1) / 0.2).clamp_max(1.0)).clamp_min(0.0)
        inside = torch.ones(n, device=s.device, dtype=s.dtype)
        inside[0] = inside[-1] = 0.0
        th = th * (inside[:, None] if axis == 0 else inside[None, :])
        gr = [torch.where(th > 0, 0.5 * _limited(to(q, -1), q, to(q, 1), th), 0.0) for q in (s, h, u, v)]
        # the edge below (west of) each cell: '-' side from the neighbour
        sm, hm, um, vm = (to(q + g, -1) for q, g in zip((s, h, u, v), gr))
        sp, hp, up, vp = (q - g for q, g in zip((s, h, u, v), gr))
        zm, zp = sm - hm, sp - hp
        z = torch.maximum(zm, zp)
        sms, sps = torch.maximum(sm, z), torch.maximum(sp, z)
        dm, dp = sms - z, sps - z
        um, vm, up, vp = (torch.where(d == 0, 0.0, q) for q, d in ((um, dm), (vm, dm), (up, dp), (vp, dp)))
        gm, gp = torch.sqrt(G * dm), torch.sqrt(G * dp)
        nm, np_ = (vm, vp) if axis == 0 else (um, up)
        hi = torch.maximum(nm + gm, np_ + gp).clamp_min(0)
        lo = torch.minimum(nm - gm, np_ - gp).clamp_max(0)
        length = dxb[:-1] if axis == 0 else torch.full_like(dxb[:-1], dyl)
        ok = (hi - lo > 1e-12) & (torch.maximum(gm, gp) > math.sqrt(G * MAD))
        inv = torch.where(ok, length / (hi - lo), 0.0)
        fr2 = (vm * vm + vp * vp + um * um + up * up) / (gm * gm + gp * gp + 1e-10)
        fr2 = torch.sqrt(fr2.clamp(0.001, 1.0))
        q = [(sps - sms, None), (um * dm, up * dp), (vm * dm, vp * dp)]
        normal = q[2] if axis == 0 else q[1]
        f = [((hi * normal[0] - lo * normal[1]) + hi * lo * q[0][0]) * inv]
        f += [(hi * a * nm - lo * b * np_ + fr2 * hi * lo * (b - a)) * inv for a, b in q[1:]]
        p = 0.5 * G * inv * (hi * dm * dm - lo * dp * dp)
        hc, hcm, ec, ecm = h, to(h, -1), elv, to(elv, -1)
        below = 0.5 * G * ((dm - hm) * (dm + hm) - (hm + hcm) * (zm - ecm)) * length - p
        above = p - 0.5 * G * ((dp - hp) * (dp + hp) - (hp + hc) * (zp - ec)) * length
        edge = torch.ones_like(s)   # no edges on row 0 and column 0
        edge[0], edge[:, 0] = 0.0, 0.0

        def difference(a):   # the edges above and below each cell, none above the last
            a = a * edge
            nxt = to(a, 1).clone()
            nxt[(-1, slice(None)) if axis == 0 else (slice(None), -1)] = 0.0
            return nxt, a
        for k in range(3):
            nxt, own = difference(f[k])
            flux[k] = flux[k] + nxt - own
        nxt, own = difference(below)[0], above * edge
        source[1 - axis] = source[1 - axis] + own + nxt
        speed = torch.maximum(hi, -lo) * edge
        rate = max(rate, float((speed / ((torch.full_like(length, dyl) if axis == 0 else dxb[:-1]) * 0.5 * cfl)).max()))
    if kw["spherical"]:
        inner = torch.ones_like(s)
        inner[0], inner[:, 0] = 0.0, 0.0
        source[1] = source[1] + inner * (0.5 * G * h * h * (dxb[1:] - dxb[:-1]) - area * (cor + tan * u) * uh)
        source[0] = source[0] + inner * area * (cor + tan * u) * vh
    return s, h, u, v, uh, vh, flux, source, rate


def _fv_update(kw, base, parts, elv, dt, t, nsq):
    _, _, area, _, _, _ = _rows(kw)
    s, h, u, v, uh, vh, flux, source, _ = parts
    s, uh, vh = base if base is not None else (s, uh, vh)
    s, uh, vh = (q - dt / area * f for q, f in zip((s, uh, vh), flux))
    drag = 1.0 / (1.0 + dt * G * h * nsq * torch.sqrt(u * u + v * v) * h.clamp_min(MAD) ** (-7.0 / 3.0))
    wet = s > elv + MAD
    uh = torch.where(wet, (uh + dt / area * source[0]) * drag, 0.0)
    vh = torch.where(wet, (vh + dt / area * source[1]) * drag, 0.0)
    if kw.get("boundary_kind"):
        H, d, x0 = kw["boundary_function_params"]
        arg = math.sqrt(3.0 * H / (4.0 * d ** 3)) * (0.5 * kw["lw"][0] / kw["nx"][0] - x0 - math.sqrt(G * (d + H)) * t)
        west = H / math.cosh(min(abs(arg), 300.0)) ** 2
        s[:, 0], uh[:, 0], vh[:, 0] = west, uh[:, 1].clone(), 0.0
        s[:, -1], uh[:, -1], vh[:, -1] = WALL, uh[:, -2].clone(), 0.0
        for j, inner in ((0, 1), (-1, -2)):
            s[j], uh[j], vh[j] = WALL, 0.0, vh[inner].clone()
            s[j, 0] = west
            elv[j, 0] = -d
    return s, uh, vh


def _fv(kw, method, elv, dt_fixed, nsq):
    """One step of rk2, midpoint or euler, and its dt, from the time t."""
    theta, cfl = (0.9, 0.9) if method == "euler" else (1.6, 0.99)

    def step(U, t):
        parts = _fv_fluxes(kw, *U, elv, theta, cfl)
        dt = dt_fixed or 1.0 / parts[-1]
        half = 0.5 * dt if method == "midpoint" else dt
        new = _fv_update(kw, None, parts, elv, half, t + half, nsq)
        if method == "midpoint":
            new = _fv_update(kw, U, _fv_fluxes(kw, *new, elv, theta, cfl), elv, dt, t + dt, nsq)
        elif method == "rk2":
            new = _fv_update(kw, None, _fv_fluxes(kw, *new, elv, theta, cfl), elv, dt, t + 2.0 * dt, nsq)
            new = tuple(0.5 * (a + b) for a, b in zip(new, U))
        return new, dt

    return step


def exact(case, seed):
    if case["kind"] == "nested" or case.get("method") == "leapfrog_nonlinear":
        return None
    if case["kind"] == "batch":
        kw, elv, stages = _ocean(case["nx"], case["ny"], True, seed, case["count"])
        dt, cells = _timestep(kw, -elv, 0.63), _gauge_cells(kw, case["gauges"], seed)[0]
        U, peak, series = [], [], []
        for s in stages:
            u, m, g = _march_ocean(kw, elv, np.float32(s), dt, case["steps"], None, cells)
            U.append(torch.stack(u).cpu())
            peak.append(m.cpu())
            series.append(torch.stack(g)[:, :, 0])
        out = dict(U=torch.stack(U), max_stage=torch.stack(peak))
        if case["gauges"]:
            out["gauges"] = torch.stack(series, 1)
        return out
    kw, U, dt = _inputs(case, seed)
    if case["kind"] == "adjoint":
        return _exact_gradient(case, seed, kw, U, dt)
    if case["real_bytes"] == 4:
        U = U.astype(np.float32).astype(np.float64)
    cells = _gauge_cells(kw, case["gauges"], seed)[0] if case["gauges"] else None
    if case["method"] in OCEAN:
        nsq = None if case["method"] == "linear" else 0.025 ** 2
        U, peak, series = _march_ocean(kw, U[3], U[0], dt, case["steps"], nsq, cells)
    else:
        elv = torch.as_tensor(U[3], device=_device())
        U = tuple(torch.as_tensor(U[k], device=_device()) for k in range(3))
        step, t, peak, series = _fv(kw, case["method"], elv, dt, 0.025 ** 2), 0.0, U[0].clone(), []
        for _ in range(case["steps"]):
            U, now = step(U, t)
            t += now
            peak = torch.maximum(peak, U[0])
            if cells is not None:
                series.append(torch.stack([x[cells[:, 0], cells[:, 1]] for x in U], -1).cpu())
    out = dict(U=list(U), max_stage=peak)
    if cells is not None:
        out["gauges"] = torch.stack(series)
    return out


def _march_ocean(kw, elv, stage, dt, steps, nsq, cells):
    elv = torch.as_tensor(np.float64(elv), device=_device())
    U = (torch.as_tensor(np.float64(stage), device=_device()), torch.zeros_like(elv), torch.zeros_like(elv))
    step, peak, series = _leapfrog(kw, elv, dt, nsq), U[0].clone(), []
    for _ in range(steps):
        U = step(*U)
        peak = torch.maximum(peak, U[0])
        if cells is not None:
            series.append(torch.stack([x[cells[:, 0], cells[:, 1]] for x in U], -1).cpu())
    return U, peak, series


def _exact_gradient(case, seed, kw, U, dt):
    from torch.utils.checkpoint import checkpoint
    cells = _gauge_cells(kw, case["gauges"], seed)[0]
    step = _leapfrog(kw, torch.as_tensor(U[3], device=_device()), dt)
    target = torch.as_tensor(_target(case, seed), device=_device())

    def segment(s, u, v, first, count):
        loss = 0.0
        for n in range(first, first + count):
            s, u, v = step(s, u, v)
            loss = loss + 0.5 * (s[cells[:, 0], cells[:, 1]] - target[n]).square().sum()
        return s, u, v, loss

    x = torch.as_tensor(U[:3], device=_device()).clone().requires_grad_()
    now, loss = (x[0], x[1], x[2]), 0.0
    for first in range(0, case["steps"], 10):
        *now, part = checkpoint(segment, *now, first, min(10, case["steps"] - first), use_reentrant=False)
        loss = loss + part
    loss.backward()
    return dict(loss=float(loss), gradient=x.grad)
