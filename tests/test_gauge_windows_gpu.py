"""Two-steps-a-pass kernels with many gauges in one warp's rows and columns:
every cell of a block (fewer and more than a window's list holds), every cell
of a row, several gauges in a cell, and a series that ends in the middle of a
pair.  Records, adjoint sweeps and batches must be those of single steps, bit
for bit."""
import ctypes

import numpy as np
import pytest

from ptha_b200 import Domain, _lib, workloads
from ptha_b200.batch import Batch

pytestmark = pytest.mark.gpu

NX, NY = 137, 90


def _cells(kind):
    if kind == "row":
        c = [(i, 41) for i in range(NX)]
    elif kind == "twice":      # each cell of a small block twice, in another order
        c = [(i, j) for j in range(30, 34) for i in range(50, 70)]
        c = c + c[::-1]
    else:                      # 300 / 900 cells of a block of 30 columns
        c = [(40 + k % 30, 20 + k // 30) for k in range(int(kind))]
    return np.array(c)


def _case(real_bytes):
    kw, U = workloads.spherical_patch(nx=NX, ny=NY, seed=5)
    kw.update(timestepping_method="linear", real_bytes=real_bytes)
    rng = np.random.default_rng(2)
    U[0] = np.where(U[3] < 0, rng.standard_normal((NY, NX)), np.minimum(U[3], 0.0))
    U[1:3] = np.where(U[3] < 0, 20.0 * rng.standard_normal((2, NY, NX)), 0.0)
    return kw, U


def _xy(kw, cells):
    return np.asarray(kw["lower_left"]) + (cells + 0.5) * np.asarray(kw["lw"]) / [NX, NY]


KINDS = ["row", "twice", "300", "900"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("real_bytes", [8, 4])
@pytest.mark.parametrize("rows", [None, "3", "90"])
def test_records_equal_single_steps(kind, real_bytes, rows, monkeypatch):
    if rows:
        monkeypatch.setenv("SWALS_PAIR_ROWS", rows)
    kw, U = _case(real_bytes)
    xy = _xy(kw, _cells(kind))
    out = []
    for pairs in (True, False):
        with Domain(**kw) as d:
            d.set_U(U)
            d.gauges_setup(xy, 20)
            dt = 0.5 * d.linear_timestep_max()
            if pairs:
                d.evolve_steps(15, dt)
            else:
                for _ in range(15):
                    d.evolve_one_step(dt)
            out.append((d.gauges_read(), d.get_U()))
    assert out[0][0].shape[0] == 15 and np.abs(out[0][0]).max() > 0.0
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("real_bytes", [8, 4])
def test_sweeps_equal_single_steps(kind, real_bytes):
    kw, U = _case(real_bytes)
    cells = _cells(kind)
    rng = np.random.default_rng(3)
    with Domain(**kw) as d:
        d.set_U(U)
        d.gauges_setup(_xy(kw, cells), 20)
        dt = 0.5 * d.linear_timestep_max()
        g = rng.standard_normal((6, len(cells)))
        lam = rng.standard_normal((3, NY, NX)).astype(d.dtype)
        together = d.adjoint_linear(6, dt, gauge_adjoint=g, lambda_seed=lam)
        for n in range(5, -1, -1):
            lam = d.adjoint_linear(1, dt, gauge_adjoint=g[n:n + 1], lambda_seed=lam)
    np.testing.assert_array_equal(together, lam)


@pytest.mark.parametrize("kind", KINDS)
def test_batch_records_equal_single_steps(kind):
    kw, U = _case(4)
    grid = Domain(**kw)
    grid.set_U(U)
    dt = 0.5 * grid.linear_timestep_max()
    ics = np.stack([U[:3], -0.5 * U[:3], 0.25 * U[:3]])
    out = []
    for chosen in (None, 0):
        b = Batch(grid, 3)
        if chosen is not None:
            b.set_tile_config(chosen)
        b.set_U(ics)
        b.gauges_setup(_xy(kw, _cells(kind)), 20)
        b.evolve(15, dt)
        out.append(b.gauges_read())
        b.close()
    grid.close()
    assert out[0].shape[0] == 15
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("capacity", [1, 7, 8])
def test_series_ending_within_a_pair(capacity):
    """The records that fit are there, and the read says that more were asked for."""
    kw, U = _case(8)
    out = []
    for pairs in (True, False):
        with Domain(**kw) as d:
            d.set_U(U)
            dt = 0.5 * d.linear_timestep_max()
            d.evolve_one_step(dt)
            d.gauges_setup(_xy(kw, _cells("twice")), capacity)
            if pairs:
                d.evolve_steps(10, dt)
            else:
                for _ in range(10):
                    d.evolve_one_step(dt)
            rec = np.zeros((capacity, len(_cells("twice")), 3))
            n = ctypes.c_int32()
            rc = _lib.lib().swals_gpu_gauges_read(d.handle, rec.ctypes.data_as(ctypes.c_void_p), capacity,
                                                  ctypes.byref(n))
            assert rc != _lib.SWALS_OK and "gauge buffer full: 10" in _lib.last_error() and n.value == capacity
            out.append(rec)
    assert np.abs(out[0][-1]).max() > 0.0
    np.testing.assert_array_equal(out[0], out[1])


def test_failed_setup_leaves_no_sites():
    """A gauge outside the domain is refused, and nothing is left of the others."""
    kw, U = _case(8)
    with Domain(**kw) as d:
        d.set_U(U)
        dt = 0.5 * d.linear_timestep_max()
        xy = _xy(kw, _cells("twice"))
        d.gauges_setup(xy, 20)
        with pytest.raises(_lib.SwalsError, match="outside the domain"):
            d.gauges_setup(np.concatenate([xy[:3], [[1.0e9, -1.0e9]]]), 20)
        with pytest.raises(_lib.SwalsError, match="gauges must be set up first"):
            d.misfit_gradient(4, dt, np.zeros((4, 4)), checkpoint_every=2)
        d.evolve_steps(6, dt)
        assert np.isfinite(d.get_U()).all()
        d.gauges_setup(xy, 20)
        d.evolve_steps(6, dt)
        assert d.gauges_read().shape == (6, len(xy), 3)
