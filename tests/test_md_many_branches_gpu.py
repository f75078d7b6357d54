"""More domains than branches: ten domains advance on eight streams, two of
which carry two domains each.  State, clocks, boundary fluxes, nesting flux
integrals and halo buffers must be those of the domains advancing one after
another (a domain's timers on), bit for bit, step by step and from a graph."""
import numpy as np
import pytest

from ptha_b200 import Multidomain
from ptha_b200.nesting import NestDomain

pytestmark = pytest.mark.gpu

N, DX = 90, 1000.0
METHODS = ["rk2", "linear", "euler", "euler", "rk2", "leapfrog_nonlinear", "rk2", "linear", "rk2"]


def _nest():
    specs = [NestDomain((0.0, 0.0), (N * DX, N * DX), (N, N), "rk2", 1)]
    for k, method in enumerate(METHODS):
        ll = ((7 + 28 * (k % 3)) * DX, (7 + 28 * (k // 3)) * DX)
        specs.append(NestDomain(ll, (15 * DX, 15 * DX), (45, 45), method, 3 + k % 2))
    return specs


def _run(graph, timed):
    specs = _nest()
    md = Multidomain(specs, domain_kwargs=[dict(real_bytes=8 if k % 3 else 4) for k in range(len(specs))],
                     use_wetdry_limiting=True, flux_correction=True)
    for d, s in zip(md.domains, specs):
        X, Y = np.meshgrid(s.x(), s.y())
        U = np.zeros((4, s.nx[1], s.nx[0]))
        U[3] = np.clip(-50.0 + (X - 40000.0) / 500.0, -50.0, 5.0)
        U[0] = np.maximum(np.exp(-((X - 40000.0) ** 2 + (Y - 45000.0) ** 2) / (2 * 9000.0 ** 2)), U[3])
        d.set_U(U)
        if d.timestepping_method != "linear":
            d.set_manning_squared(0.025 ** 2)
    if timed:
        md.domains[4].timers_enable()
    if graph:
        md.capture_graph(3, 10.0)
        md.replay(3)
    else:
        for _ in range(9):
            md.evolve_one_step(10.0)
    md.synchronize()
    states = [d.state() for d in md.domains]
    out = [np.array([md.time])]
    out += [d.get_U() for d in md.domains]
    out.append(np.array([[s.time, s.boundary_flux_evolve_integral, s.boundary_flux_time_integral,
                          s.nsteps_advanced] for s in states]))
    out.append(np.array([list(s.boundary_flux_store) for s in states]))
    for e in range(len(md.exchanges)):
        out.append(md.buffer(e))
        out += [md.flux(e, which) for which in ("send", "recv", "error")]
    md.close()
    return out


def test_ten_domains_side_by_side_equal_one_after_another():
    serial = _run(False, True)
    assert sum(np.abs(x).max() > 0.0 for x in serial[-40:]) > 10
    for graph in (False, True):
        both = _run(graph, False)
        assert len(both) == len(serial)
        for k, (a, b) in enumerate(zip(both, serial)):
            assert np.isfinite(b).all(), k
            np.testing.assert_array_equal(a, b, err_msg=str((graph, k)))
