"""Repeated misfit gradients on one domain: the segments' graphs are kept
between calls, and each call must give the loss and gradient of a domain that
was made for it, bit for bit -- with other numbers of steps (fewer, and more,
which grows the scratch), another spacing or time step and back, other gauge
cells of the same count, and an adjoint sweep in between."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads

pytestmark = pytest.mark.gpu

NX, NY, NG = 90, 60, 4


def _sites(kw, seed):
    rng = np.random.default_rng(seed)
    cell = np.stack([rng.integers(0, NX, NG), rng.integers(0, NY, NG)], axis=1)
    return np.asarray(kw["lower_left"]) + (cell + 0.5) * np.asarray(kw["lw"]) / [NX, NY]


@pytest.mark.parametrize("real_bytes", [8, 4])
def test_each_call_equals_a_fresh_domain(real_bytes):
    kw, U = workloads.spherical_patch(nx=NX, ny=NY, seed=3)
    kw.update(timestepping_method="linear", real_bytes=real_bytes)

    def gradient(d, sites, nsteps, dt, every):
        d.gauges_setup(_sites(kw, sites), 200)
        target = 0.1 * np.random.default_rng(nsteps).standard_normal((nsteps, NG))
        return d.misfit_gradient(nsteps, dt, target, checkpoint_every=every)

    with Domain(**kw) as d:
        d.set_U(U)
        dt = 0.8 * d.linear_timestep_max()
        for k, (sites, nsteps, step, every) in enumerate(
                [(0, 100, dt, 20), (0, 60, dt, 20), (0, 140, dt, 20), (1, 60, dt, 20), (1, 61, dt, 20),
                 (1, 60, 0.5 * dt, 20), (1, 60, dt, 20), (1, 60, dt, 10), (1, 130, dt, 20)]):
            if k == 3:
                d.adjoint_linear(150, dt, gauge_adjoint=np.ones((150, NG)))
            loss, g = gradient(d, sites, nsteps, step, every)
            with Domain(**kw) as fresh:
                fresh.set_U(U)
                loss1, g1 = gradient(fresh, sites, nsteps, step, every)
            assert loss == loss1 and loss > 0.0, (k, nsteps)
            np.testing.assert_array_equal(g, g1, err_msg=str((k, nsteps)))
            assert np.isfinite(g).all() and np.abs(g).max() > 0.0


@pytest.mark.parametrize("every", [20, 22, 10])
def test_launches_counted_as_launched(every):
    """A replayed segment counts the kernels it holds: as many as when every
    kernel is launched by itself (timers on)."""
    kw, U = workloads.spherical_patch(nx=NX, ny=NY, seed=3)
    kw.update(timestepping_method="linear")
    target = np.zeros((100, NG))
    with Domain(**kw) as d:
        d.set_U(U)
        d.gauges_setup(_sites(kw, 0), 200)
        dt = 0.8 * d.linear_timestep_max()
        counts = []
        for timed in (False, False, True):
            d.timers_enable(timed)
            n = d.launch_count()
            d.misfit_gradient(100, dt, target, checkpoint_every=every)
            counts.append(d.launch_count() - n)
    assert counts[0] == counts[1] == counts[2] > 0
