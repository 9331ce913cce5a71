"""The persistent PCG cuts a solve into launches of 2048 iterations: limits at and around that number stop
after exactly their count (every one of a failing increment's five attempts), a solve of several launches
is bit-reproducible, and in a batch an instance that runs into its limit after several launches disturbs
no other.  Near-incompressible systems (bulk / shear 1e6) take about 9000 iterations (7^3) and more than
10000 (9^3) to 1e-10, the others below 300."""
import numpy as np
import pytest

from conftest import rel_err
from neon_b200 import mesh as M
from neon_b200 import problem as P

pytestmark = pytest.mark.gpu


def _problem(n, ratio, maxit):
    mesh = M.structured_hex8(n, n, n, jitter=0.05, seed=3)
    bcs = [{"name": "bottom", "time": [0.0, 1.0], "x": [0.0, 0.0], "y": [0.0, 0.0],
            "z": [0.0, 0.0]},
           {"name": "top", "time": [0.0, 1.0], "z": [0.0, 1e-3]}]
    opts = P.Options(residual_tolerance=1e9, displacement_tolerance=1e9, linear_iterations=2,
                     initial=1.0, minimum=1.0, maximum=1.0, adaptive=False, cg_tolerance=1e-10,
                     cg_maximum_iterations=maxit)
    return P.Problem("turns", mesh, P.Material(P.LINEAR_ELASTIC, ratio, 1.0),
                     P.dirichlet_boundaries(mesh, bcs), opts)


@pytest.mark.parametrize("n", [2, 7])  # one CTA, a group
@pytest.mark.parametrize("maxit", [1, 2047, 2048, 2049, 4096, 4097])
def test_iteration_limit_is_exact(n, maxit):
    from neon_b200 import api
    pr = _problem(n, 1e6 if n > 2 else 1e9, maxit)
    if n == 2:
        pr.options.cg_tolerance = 1e-300  # never met
    sm = api.StaticMatrix(pr)
    with pytest.raises(api.ComputationalError):
        sm.solve()
    assert sm.report["cg_iterations"] == 5 * maxit


def test_several_launches_are_bit_reproducible():
    from neon_b200 import api
    sm = api.StaticMatrix(_problem(7, 1e6, 60000))
    u = sm.solve()
    assert sm.report["cg_iterations"] > 2 * 2048
    assert np.array_equal(u, sm.solve())


@pytest.mark.parametrize("precision", [0, 1])
def test_a_long_instance_disturbs_no_other(precision):
    """Twelve times as many CTAs as the GPU has are wanted, so groups take turns on the same CTAs."""
    from neon_b200 import api
    maxit = 7000
    slow = _problem(9, 1e6, maxit)
    good = [_problem(n, 10.0, maxit) for n in (8, 7, 6, 5) for _ in range(60)]
    b = api.BatchedStaticMatrix([slow] + good, precision=precision, autotune=False)
    with pytest.raises(api.ComputationalError):
        b.solve()
    assert b.reports[0]["status"] == api.E_CUTBACK_LIMIT
    assert b.reports[0]["cg_iterations"] == 5 * maxit
    assert all(r["status"] == 0 for r in b.reports[1:])
    for i in (1, 61, 121, 181):
        pr = good[i - 1]
        u = api.StaticMatrix(pr).solve()
        assert rel_err(b.instance_displacement(i), u) < 1e-8
