"""The kernel timers time what an untimed run launches: evolve_steps of a linear
domain takes its steps by pairs with timers on as well, to the same bits."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["linear", "leapfrog_linear_plus_nonlinear_friction"])
@pytest.mark.parametrize("real_bytes", [8, 4])
def test_timed_steps_are_the_untimed_ones(method, real_bytes):
    kw, U = workloads.spherical_patch(nx=137, ny=90, seed=5)
    kw.update(timestepping_method=method, real_bytes=real_bytes)
    out = []
    for timed in (False, True):
        with Domain(**kw) as d:
            d.set_U(U)
            d.set_manning_squared(0.03 ** 2)
            dt = 0.5 * d.linear_timestep_max()
            d.evolve_steps(1, dt)
            d.timers_enable(timed)
            n = d.launch_count()
            d.evolve_steps(11, dt)
            tm = d.timers_read()
            s = d.state()
            out.append((d.launch_count() - n, d.get_U(), d.max_stage(), s.time, s.nsteps_advanced,
                        list(s.boundary_flux_store), s.boundary_flux_time_integral))
            if timed:   # five pairs and a single step, whose friction is a kernel of the edge's kind
                assert tm["leapfrog_step"][1] == 6 and tm["leapfrog_step"][0] > 0.0
                assert tm["leapfrog_edge"][1] == 6 + (method != "linear") and tm["leapfrog_edge"][0] > 0.0
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
