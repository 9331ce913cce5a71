"""Mixed-precision Newton solves at sizes past the rule that runs smaller ones in FP64 (an assembled K beyond
100 MB for hex8, 130 MB for tet4), for the elements and models whose FP32 PCG runs only there: tet4 (its own
kernel for the search direction, products summed from lists, blocks of 128 elements with a partial last
one) and the anisotropic microspheres (FP64 residual by the element kernels).

Against the FP64 solution, which for these runs on the assembled K: Newton tolerance 1e-8 on both sides, no
path dependence (J2 stays elastic)."""
import numpy as np
import pytest

from conftest import rel_err
from neon_b200 import mesh as M
from neon_b200 import problem as P

pytestmark = pytest.mark.gpu

MATERIALS = {
    "linear": (P.Material(P.LINEAR_ELASTIC, 175e3, 80e3), 1e-3),
    "j2": (P.Material(P.J2_SMALL_STRAIN, 175e3, 80e3, 200.0, 1e3), 2.5e-4),
    "neohooke": (P.Material(P.NEO_HOOKE, 10.0, 1.0), 0.02),
    "langevin": (P.Material(P.LANGEVIN_AFFINE_MICROSPHERE, 10.0, 1.0, segments_per_chain=50.0), 0.02),
    "nonaffine": (P.Material(P.NONAFFINE_MICROSPHERE, 10.0, 1.0, segments_per_chain=50.0,
                             nonaffine_stretch_parameter=1.5), 0.02),
}


def _problem(model, mesh):
    mat, load = MATERIALS[model]
    bcs = [{"name": "bottom", "time": [0.0, 1.0], "x": [0.0, 0.0], "y": [0.0, 0.0],
            "z": [0.0, 0.0]},
           {"name": "top", "time": [0.0, 1.0], "z": [0.0, load]}]
    opts = P.Options(residual_tolerance=1e-8, displacement_tolerance=1e-8, linear_iterations=15,
                     cg_tolerance=1e-10, cg_maximum_iterations=20000)
    return P.Problem("mixed", mesh, mat, P.dirichlet_boundaries(mesh, bcs), opts)


@pytest.mark.parametrize("element,model", [("tet4", "linear"), ("tet4", "j2"), ("tet4", "neohooke"),
                                           ("tet4", "langevin"), ("hex8", "langevin"),
                                           ("hex8", "nonaffine")])
def test_mixed_newton_beyond_the_fp64_rule(element, model):
    from neon_b200 import api
    mesh = M.structured_tet4(50) if element == "tet4" else M.structured_hex8(41, 37, 39)
    if element == "tet4":
        assert mesh.num_elements % 128 == 48
    pr = _problem(model, mesh)
    u = api.StaticMatrix(pr).solve()
    sm = api.StaticMatrix(pr, precision=api.MIXED)
    assert 72 * sm.mesh.nnzb > (130e6 if element == "tet4" else 100e6)
    assert rel_err(sm.solve(), u) < 1e-8


@pytest.mark.parametrize("precision", [0, 1])
def test_plastic_hex8_newton_is_bit_reproducible(precision):
    """Newton steps into the plastic range (top displacement 2e-3, yield strain about 1e-3).  Whether neon's
    path-dependent update converges there is not the question: every step and the displacement that
    the solve ends with have the same bits."""
    from neon_b200 import api
    pr = _problem("j2", M.structured_hex8(41, 37, 39))
    for t in pr.dirichlet:
        if t.values[-1] > 0:
            t.values = np.array([0.0, 2e-3])
    pr.options.linear_iterations = 4
    runs = []
    for _ in range(2):
        sm = api.StaticMatrix(pr, precision=precision)
        u = sm.solve(raise_on_error=False)
        assert (sm.mesh.quadrature_values("accumulated_plastic_strain") > 0).mean() > 0.3
        runs.append((u, sm.log))
    assert len(runs[0][1]) >= 4
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])


def test_two_contexts_solve_from_two_threads():
    """Each persistent launch wants every SM at once; two threads with a context each take turns and get
    the solutions that they get alone (bit for bit: the Newton path is reproducible)."""
    import threading
    from neon_b200 import api
    solvers = [api.StaticMatrix(_problem("neohooke", M.structured_hex8(*s))) for s in ((12, 11, 10),
                                                                                    (14, 9, 8))]
    alone = [sm.solve() for sm in solvers]
    got = [[], []]

    def work(i):
        for _ in range(5):
            got[i].append(solvers[i].solve())

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        assert len(got[i]) == 5
        assert all(np.array_equal(u, alone[i]) for u in got[i])
