"""A batch takes its steps two at a time unless a kernel was chosen for it:
the state, max_stage and gauge series of every instance must be those of a
chosen single-step kernel, bit for bit, for step counts that leave the graph,
single pairs and a single step over, with and without max_stage and gauges."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads
from ptha_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,real_bytes", [(64, 48, 8), (121, 90, 8), (241, 77, 4)])
@pytest.mark.parametrize("gauges,record", [(3, True), (70, True), (0, False)])
def test_batch_pairs_equal_single_steps(nx, ny, real_bytes, gauges, record):
    kw, U = workloads.spherical_patch(nx=nx, ny=ny)
    kw.update(timestepping_method="linear", real_bytes=real_bytes)
    grid = Domain(**kw)
    grid.set_U(U)
    dt = 0.8 * grid.linear_timestep_max()
    rng = np.random.default_rng(nx)
    ics = np.where(U[3] < 0, rng.standard_normal((3, 3, ny, nx)), 0.0)
    cell = np.stack([rng.integers(0, nx, gauges), rng.integers(0, ny, gauges)], axis=1)
    xy = np.asarray(kw["lower_left"]) + (cell + 0.5) * np.asarray(kw["lw"]) / [nx, ny]
    out = []
    for chosen in (None, 0):
        b = Batch(grid, 3, record_max_stage=record)
        if chosen is not None:
            b.set_tile_config(chosen)
        b.set_U(ics)
        if gauges:
            b.gauges_setup(xy, 100)
        for n in (39, 1, 2, 7, 5):
            b.evolve(n, dt)
        out.append((b.get_U(), b.max_stage() if record else None, b.gauges_read() if gauges else None, b.time()))
        b.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    grid.close()
