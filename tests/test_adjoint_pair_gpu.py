"""An adjoint sweep takes two steps a pass (adjoint_pair.cu): it must give the
bits of as many sweeps of one step, each seeded with the one before -- on grids
narrower than a strip (60 FP64, 120 FP32 columns), of one strip and of several,
with ragged ends; Coriolis, linear friction, a sub-region; repeated gauge cells,
more gauges than a mask holds."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads

pytestmark = pytest.mark.gpu

VARIANTS = {
    "plain": dict(),
    "coriolis": dict(spherical=True),
    "friction_msl": dict(linear_friction_coeff=1.0e-4, msl_linear=0.4),
    "region": dict(xL=3, xU=-2, yL=2, yU=-3, spherical=True),
}


def _domain(nx, ny, variant, real_bytes):
    rng = np.random.default_rng(nx * 100 + ny)
    if variant.get("spherical"):
        kw, U = workloads.spherical_patch(nx=nx, ny=ny, seed=nx)
    else:
        kw = dict(nx=(nx, ny), lw=(nx * 1000.0, ny * 1000.0), lower_left=(0.0, 0.0))
        U = np.zeros((4, ny, nx))
        U[3] = -2000.0 + 800.0 * rng.standard_normal((ny, nx))
        U[3][rng.random((ny, nx)) < 0.1] = 30.0
    U[0] = np.where(U[3] < 0, rng.standard_normal((ny, nx)), np.minimum(U[3], 0.0))
    v = dict(variant)
    for k, n in (("xU", nx), ("yU", ny)):
        if k in v:
            v[k] = n + v[k]
    return dict(kw, timestepping_method="linear", real_bytes=real_bytes) | v, U, rng


def _check(nx, ny, variant, real_bytes, ngauges, nsteps):
    kw, U, rng = _domain(nx, ny, variant, real_bytes)
    cell = np.stack([rng.integers(0, nx, ngauges), rng.integers(0, ny, ngauges)], axis=1)
    cell[:2] = [[0, 0], [nx - 1, ny - 1]]
    cell[2] = cell[3]
    with Domain(**kw) as d:
        d.set_U(U)
        d.gauges_setup(np.asarray(kw["lower_left"]) + (cell + 0.5) * np.asarray(kw["lw"]) / [nx, ny], nsteps)
        dt = 0.5 * d.linear_timestep_max()
        g = rng.standard_normal((nsteps, ngauges))
        seed = rng.standard_normal((3, ny, nx)).astype(d.dtype)
        together = d.adjoint_linear(nsteps, dt, gauge_adjoint=g, lambda_seed=seed)
        lam = seed
        for n in range(nsteps - 1, -1, -1):
            lam = d.adjoint_linear(1, dt, gauge_adjoint=g[n:n + 1], lambda_seed=lam)
    assert np.isfinite(lam).all()
    np.testing.assert_array_equal(together, lam)


@pytest.mark.parametrize("name", list(VARIANTS))
@pytest.mark.parametrize("nx,ny", [(7, 9), (60, 33), (61, 40), (120, 37), (137, 90), (430, 131)])
@pytest.mark.parametrize("real_bytes", [8, 4])
def test_pairs_equal_single_steps(name, nx, ny, real_bytes):
    _check(nx, ny, VARIANTS[name], real_bytes, 70 if nx == 61 else 6, 7)


@pytest.mark.parametrize("real_bytes", [8, 4])
@pytest.mark.parametrize("rows", [1, 2, 7, 33, 131])
def test_any_segment_height(rows, real_bytes, monkeypatch):
    monkeypatch.setenv("SWALS_PAIR_ROWS", str(rows))
    _check(430, 131, VARIANTS["coriolis"], real_bytes, 6, 4)
