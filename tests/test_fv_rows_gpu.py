"""The rows per strip segment that the stage kernels choose from the grid
against segments of 8 rows, bit for bit: grids for which the choice is 1, 2,
3, 5 and 14 rows, widths that leave a ragged last strip."""
import numpy as np
import pytest

from ptha_b200 import Domain, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(120, 80), (300, 200), (420, 300), (521, 390), (930, 931)])
@pytest.mark.parametrize("real_bytes", [8, 4])
def test_rows_choice_changes_no_bit(nx, ny, real_bytes, monkeypatch):
    n = max(nx, ny)
    kw, U, _, nsq = workloads.rk2_beach(n=n, dx=20480.0 / n, toe=17580.0)
    U = np.ascontiguousarray(U[:, :ny, :nx])
    U[0] += np.where(U[0] > U[3], 0.3 * np.sin(np.arange(nx) / 7.0)[None, :], 0.0)
    U[0] = np.maximum(U[0], U[3])
    kw = dict(kw, nx=(nx, ny), lw=(20480.0 * nx / n, 20480.0 * ny / n), real_bytes=real_bytes)
    out = []
    for rows in (None, "8"):
        monkeypatch.delenv("SWALS_FV_ROWS", raising=False)
        if rows:
            monkeypatch.setenv("SWALS_FV_ROWS", rows)
        with Domain(**kw) as d:
            d.set_U(U)
            d.set_manning_squared(nsq)
            for _ in range(3):
                d.evolve_one_step()
            out.append((d.get_U(), d.max_stage(), d.max_dt))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2] and np.isfinite(out[0][0]).all()
