"""Between two exchanges the domains of a multidomain advance side by side, on
streams of their own; with a domain's kernel timers on they advance one after
another.  Both must give the same bits, step by step and from a graph, and
leave the time, the fluxes and the corrections the same."""
import numpy as np
import pytest

from ptha_b200 import Multidomain

from nest_cases import two_level_nest

pytestmark = pytest.mark.gpu


def _run(method, graph, timed):
    specs = two_level_nest(ratio=3, child_method=method, parent_method="linear")
    md = Multidomain(specs, domain_kwargs=[dict(real_bytes=4), dict(real_bytes=8)], use_wetdry_limiting=True,
                     flux_correction=True)
    for k, (d, s) in enumerate(zip(md.domains, specs)):
        X, Y = np.meshgrid(s.x(), s.y())
        U = np.zeros((4, s.nx[1], s.nx[0]))
        U[3] = np.clip(-50.0 + (X - 25000.0) / 200.0, -50.0, 5.0)
        U[0] = np.maximum(np.exp(-((X - 18000.0) ** 2 + (Y - 20000.0) ** 2) / (2 * 4000.0 ** 2)), U[3])
        d.set_U(U)
        if d.timestepping_method != "linear":
            d.set_manning_squared(0.025 ** 2)
    if timed:
        md.domains[1].timers_enable()
    if graph:
        md.capture_graph(3, 10.0)
        md.replay(3)
    else:
        for _ in range(9):
            md.evolve_one_step(10.0)
    md.synchronize()
    out = md.time, [d.get_U() for d in md.domains], [d.state().time for d in md.domains]
    md.close()
    return out


@pytest.mark.parametrize("method", ["rk2", "euler", "linear"])
def test_side_by_side_equals_one_after_another(method):
    serial = _run(method, False, True)
    for graph in (False, True):
        both = _run(method, graph, False)
        assert both[0] == serial[0] and both[2] == serial[2]
        for a, b in zip(both[1], serial[1]):
            assert np.isfinite(a).all()
            np.testing.assert_array_equal(a, b)
