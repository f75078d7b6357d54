"""The straight-line FP32 reciprocal and square root of the friction terms
against the correctly rounded operators: every significand (and for roots both
parities of the exponent), the ends of the range, subnormals and zero."""
import numpy as np
import pytest

from test_rounded_gpu import _rounded, _same

pytestmark = pytest.mark.gpu

RECIPROCAL, ROOT = 3, 4
ALL = (np.arange(1 << 23, dtype=np.int32) | (127 << 23)).view(np.float32)   # 1 .. 2


def _check(op, x, want):
    _same(_rounded(op, x.astype(np.float64)), want.astype(np.float64))


@pytest.mark.parametrize("exponent", [-125, -60, 0, 77, 124])
def test_every_reciprocal(exponent):
    x = np.ldexp(ALL, exponent)
    _check(RECIPROCAL, x, np.float32(1) / x)


@pytest.mark.parametrize("exponent", [-126, -81, -80, -79, 0, 1, 126, 127])
def test_every_root(exponent):
    x = np.ldexp(ALL, exponent)
    _check(ROOT, x, np.sqrt(x))


def test_subnormal_roots_and_zero():
    x = np.arange(1, 1 << 23, dtype=np.int32).view(np.float32)
    _check(ROOT, x, np.sqrt(x))
    assert _rounded(ROOT, np.zeros(1))[0] == 2.0 ** -111
    assert np.isnan(_rounded(ROOT, np.array([np.inf, np.nan]))).all()


def test_friction_pairs_with_fading_momenta():
    """Momenta fading from 10 to subnormals and zero across the grid: the pairs'
    straight-line friction against single steps, bit for bit."""
    from ptha_b200 import Domain
    nx, ny = 240, 60
    kw = dict(nx=(nx, ny), lw=(nx * 1000.0, ny * 1000.0), lower_left=(0.0, 0.0), real_bytes=4,
              timestepping_method="leapfrog_linear_plus_nonlinear_friction")
    rng = np.random.default_rng(4)
    U = np.zeros((4, ny, nx))
    U[3] = -10.0 ** rng.uniform(-4, 3.5, (ny, nx))
    U[1:3] = rng.standard_normal((2, ny, nx)) * 10.0 ** np.linspace(1, -45, nx)
    U[:3, :, -20:] = 0.0
    out = []
    for pairs in (True, False):
        with Domain(**kw) as d:
            d.set_U(U)
            d.set_manning_squared(0.04 ** 2)
            dt = 0.4 * d.linear_timestep_max()
            if pairs:
                d.evolve_steps(7, dt)
            else:
                for _ in range(7):
                    d.evolve_one_step(dt)
            out.append(d.get_U())
    assert np.isfinite(out[0]).all() and np.abs(out[0][1, :, 100:200]).max() > 0.0
    np.testing.assert_array_equal(out[0], out[1])
