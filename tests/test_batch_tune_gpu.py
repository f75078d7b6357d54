"""The batch's tuner times the two-step pass beside the kernels of a single step
and evolve takes the winner; a kernel set afterwards takes every step, one
tuned afterwards replaces the set one.  The state keeps its bits throughout."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads
from ptha_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,real_bytes", [(121, 90, 8), (241, 77, 4)])
def test_tuner_times_pairs_and_evolve_takes_the_winner(nx, ny, real_bytes):
    kw, U = workloads.spherical_patch(nx=nx, ny=ny)
    kw.update(timestepping_method="linear", real_bytes=real_bytes)
    grid = Domain(**kw)
    grid.set_U(U)
    dt = 0.8 * grid.linear_timestep_max()
    rng = np.random.default_rng(nx)
    ics = np.where(U[3] < 0, rng.standard_normal((3, 3, ny, nx)), 0.0)
    forms = Batch.tile_config_count()

    def launches(call):
        n = grid.launch_count()
        call()
        return grid.launch_count() - n

    plain, b = Batch(grid, 3), Batch(grid, 3)
    for x in (plain, b):
        x.set_U(ics)
    for x in (b.get_U(), plain.get_U()):
        np.testing.assert_array_equal(x, ics.astype(x.dtype))
    b.set_tile_config(forms - 1)
    got = []
    assert launches(lambda: got.append(b.tune())) == 8 * (forms + 1)
    cfg, ms = got[0]
    assert 0 <= cfg < forms and ms > 0.0
    np.testing.assert_array_equal(b.get_U(), ics.astype(b.dtype))
    assert launches(lambda: plain.evolve(12, dt)) == 6
    assert launches(lambda: b.evolve(12, dt)) in (6, 12)
    b.set_tile_config(cfg)
    assert launches(lambda: b.evolve(13, dt)) == 13
    plain.evolve(13, dt)
    np.testing.assert_array_equal(b.get_U(), plain.get_U())
    np.testing.assert_array_equal(b.max_stage(), plain.max_stage())
    for x in (plain, b):
        x.close()
    grid.close()
