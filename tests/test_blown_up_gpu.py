"""Runs that have blown up: states with huge, infinite, subnormal and NaN cells
take the branches that ordinary water never takes (plain operators in place of
the straight-line ones, the limiter as the reference writes it).  Against the
oracle, NaN for NaN and every other cell bit for bit.  In FP32 the GPU's
invalid operations give NaNs of the other sign than the oracle's, which the
limiter's sign products spread differently: one step there."""
import numpy as np
import pytest

from pairs import oracle_from_kw
from ptha_b200 import Domain, workloads

pytestmark = pytest.mark.gpu

NX, NY = 150, 90
INF, NAN = np.inf, np.nan
EXTREME = {8: [1e150, 1e200, 1e281, 1e300, 1e305, INF, -INF, NAN, -1e300, 1e290, 1e-300, 5e-324, -1e-310, 1e-291],
           4: [1e15, 1e19, 1e25, 1e30, 1e37, INF, -INF, NAN, -1e30, 1e33, 1e-40, -1e-42, 1e-38]}


def _beach(method, real_bytes, **more):
    kw, U, _, nsq = workloads.rk2_beach(n=NX, dx=100.0, toe=9000.0)
    kw = {k: v for k, v in kw.items() if not k.startswith("boundary")}
    kw = dict(kw, nx=(NX, NY), lw=(NX * 100.0, NY * 100.0), timestepping_method=method, real_bytes=real_bytes, **more)
    U = np.ascontiguousarray(U[:, :NY, :NX])
    wet = U[0] > U[3]
    U[0] = np.maximum(U[0] + np.where(wet, 0.3 * np.sin(np.arange(NX) / 7.0)[None, :], 0.0), U[3])
    return kw, U, nsq, wet


def _one_by_one(U, real_bytes, nan):
    """An extreme value in one variable of cells eight apart."""
    k = 0
    for v in range(3):
        for h in EXTREME[real_bytes]:
            U[v, 5 + 8 * (k // 17), 5 + 8 * (k % 17)] = nan if np.isnan(h) else h
            k += 1
    return U


def _scattered(U, wet, real_bytes, share, seed):
    rng = np.random.default_rng(seed)
    U[1:3] = np.where(wet, rng.standard_normal((2, NY, NX)), 0.0)
    hit = rng.random((3, NY, NX)) < share
    U[:3] = np.where(hit, rng.choice(EXTREME[real_bytes], (3, NY, NX)), U[:3])
    return U


def _compare(kw, U, nsq, steps):
    real_bytes = kw["real_bytes"]
    o = oracle_from_kw({k: v for k, v in kw.items() if k != "real_bytes"}, real32=real_bytes == 4)
    o.U[:] = U
    o.manning_squared[:] = nsq
    with np.errstate(all="ignore"):
        for _ in range(steps):
            o.evolve_one_step(0.05)
    with Domain(**kw) as d:
        d.set_U(U)
        d.set_manning_squared(nsq)
        d.evolve_steps(steps, 0.05)
        got = d.get_U()
    want = np.array(o.U)
    assert np.isnan(want).any() and np.isfinite(want).any()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("form", ["strip", "tile"])
@pytest.mark.parametrize("method,steps", [("euler", 1), ("euler", 2), ("rk2", 1), ("rk2", 2), ("midpoint", 2)])
@pytest.mark.parametrize("nan", [NAN, -NAN])
def test_extreme_cells_one_by_one(method, steps, nan, form, monkeypatch):
    if form == "tile":
        monkeypatch.setenv("SWALS_FV_KERNEL", "tile")
    kw, U, nsq, _ = _beach(method, 8)
    _compare(kw, _one_by_one(U, 8, nan), nsq, steps)


@pytest.mark.parametrize("real_bytes", [8, 4])
@pytest.mark.parametrize("flux", ["DE1_low_fr_diffusion", "DE1_upwind_transverse"])
@pytest.mark.parametrize("seed", [0, 1])
def test_extreme_cells_scattered_one_stage(real_bytes, flux, seed):
    kw, U, nsq, wet = _beach("euler", real_bytes, compute_fluxes_inner_method=flux)
    _compare(kw, _scattered(U, wet, real_bytes, 0.02, seed), nsq, 1)


@pytest.mark.parametrize("real_bytes", [8, 4])
@pytest.mark.parametrize("method,more", [
    ("linear", dict()),
    ("leapfrog_linear_plus_nonlinear_friction", dict()),
    ("leapfrog_linear_plus_nonlinear_friction", dict(linear_solver_is_truely_linear=False, friction_type="chezy")),
    ("leapfrog_nonlinear", dict()),
    ("leapfrog_nonlinear", dict(friction_type="chezy"))])
def test_extreme_cells_scattered_leapfrog(method, more, real_bytes):
    kw, U, nsq, wet = _beach(method, real_bytes, **more)
    _compare(kw, _scattered(U, wet, real_bytes, 0.02, 2), nsq, 3)
