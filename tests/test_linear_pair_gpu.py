"""evolve_steps takes plain leapfrog steps two at a time (linear_pair.cu):
the state, max_stage, gauges, clock and boundary fluxes must be those of
evolve_one_step, one step at a time, bit for bit -- on grids narrower than a
strip (60 FP64, 120 FP32 columns), of one strip, with ragged last strips and
short last segments; with Coriolis, linear and Manning / Chezy friction, a
sub-region, wetting faces (not truly linear), more gauges than a mask holds."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads

pytestmark = pytest.mark.gpu

FRIC = "leapfrog_linear_plus_nonlinear_friction"
VARIANTS = {
    "plain": dict(),
    "coriolis": dict(spherical=True),
    "wet_faces": dict(linear_solver_is_truely_linear=False),
    "wet_faces_coriolis": dict(linear_solver_is_truely_linear=False, spherical=True),
    "linear_friction_msl": dict(linear_friction_coeff=1.0e-4, msl_linear=0.4),
    "region": dict(xL=3, xU=-2, yL=2, yU=-3),
    "manning": dict(timestepping_method=FRIC, linear_friction_coeff=2.0e-5),
    "chezy_coriolis": dict(timestepping_method=FRIC, friction_type="chezy", spherical=True),
    "no_max_stage": dict(record_max_stage=False),
}


def _case(nx, ny, variant, real_bytes):
    rng = np.random.default_rng(nx * 100 + ny)
    if variant.get("spherical"):
        kw, U = workloads.spherical_patch(nx=nx, ny=ny, seed=nx)
    else:
        kw = dict(nx=(nx, ny), lw=(nx * 1000.0, ny * 1000.0), lower_left=(0.0, 0.0))
        U = np.zeros((4, ny, nx))
        U[3] = -2000.0 + 800.0 * rng.standard_normal((ny, nx))
        U[3][rng.random((ny, nx)) < 0.1] = 30.0
    U[0] = np.where(U[3] < 0, rng.standard_normal((ny, nx)), np.minimum(U[3], 0.0))
    U[1:3] = np.where(U[3] < 0, 20.0 * rng.standard_normal((2, ny, nx)), 0.0)
    v = dict(variant)
    for k, n in (("xU", nx), ("yU", ny)):
        if k in v:
            v[k] = n + v[k]
    return dict(kw, timestepping_method="linear", real_bytes=real_bytes) | v, U


def _run(kw, U, ngauges, counts, pairs):
    with Domain(**kw) as d:
        d.set_U(U)
        d.set_manning_squared(0.03 ** 2)
        nx, ny = kw["nx"]
        rng = np.random.default_rng(1)
        cell = np.stack([rng.integers(0, nx, ngauges), rng.integers(0, ny, ngauges)], axis=1)
        cell[:2] = [[0, 0], [nx - 1, ny - 1]]
        d.gauges_setup(np.asarray(kw["lower_left"]) + (cell + 0.5) * np.asarray(kw["lw"]) / [nx, ny], 400)
        dt = 0.5 * d.linear_timestep_max()
        for n in counts:
            if pairs:
                d.evolve_steps(n, dt)
            else:
                for _ in range(n):
                    d.evolve_one_step(dt)
        s = d.state()
        peak = d.max_stage() if kw.get("record_max_stage", True) else None
        return (d.get_U(), peak, d.gauges_read(), s.time, s.nsteps_advanced, list(s.boundary_flux_store),
                s.boundary_flux_time_integral, s.boundary_flux_evolve_integral)


@pytest.mark.parametrize("name", list(VARIANTS))
@pytest.mark.parametrize("nx,ny", [(7, 9), (60, 33), (61, 40), (120, 37), (137, 90), (301, 131)])
@pytest.mark.parametrize("real_bytes", [8, 4])
def test_pairs_equal_single_steps(name, nx, ny, real_bytes):
    kw, U = _case(nx, ny, VARIANTS[name], real_bytes)
    # graphs of 24 and 6 steps, pairs and a single step, from every buffer
    a, b = (_run(kw, U, 70 if nx == 61 else 5, (46, 3, 2, 13), pairs) for pairs in (True, False))
    for x, y in zip(a, b):
        if isinstance(x, np.ndarray):
            assert np.isfinite(x).all()
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("rows", [4, 5, 96])
def test_any_segment_height(rows, monkeypatch):
    monkeypatch.setenv("SWALS_PAIR_ROWS", str(rows))
    kw, U = _case(137, 90, VARIANTS["coriolis"], 8)
    a, b = (_run(kw, U, 5, (20,), pairs) for pairs in (True, False))
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("name", ["plain", "coriolis", "wet_faces_coriolis", "region"])
@pytest.mark.parametrize("real_bytes", [8, 4])
@pytest.mark.parametrize("rows", [1, 2, 7, 33])
def test_segments_away_from_the_sides(rows, name, real_bytes, monkeypatch):
    """Strips and segments with and without a side next to one another."""
    monkeypatch.setenv("SWALS_PAIR_ROWS", str(rows))
    kw, U = _case(430, 90, VARIANTS[name], real_bytes)
    a, b = (_run(kw, U, 5, (10,), pairs) for pairs in (True, False))
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
