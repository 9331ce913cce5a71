"""The persistent PCG (cg_group.cu) at the sizes where its work is cut differently: a system on one
CTA (up to 96 block rows) or on a group of CTAs, one or two exchange levels (up to 16 CTAs, more),
partial tiles of 8 rows, K resident in shared memory or streamed, hex8 (27 blocks per row) and
tet4.  Newton solutions against the CPU oracle within 1e-10 relative, the bar of the other
static-solve parity tests (same equilibrium, CG at rtol 1e-10)."""
import numpy as np
import pytest

from conftest import rel_err
from neon_b200 import mesh as M
from neon_b200 import problem as P

pytestmark = pytest.mark.gpu


def _problem(element, shape, load=0.02):
    make = M.structured_hex8 if element == "hex8" else M.structured_tet4
    mesh = make(*shape)
    mat = P.make_material({"shear_modulus": 1.0, "bulk_modulus": 10.0}, {"name": "neohooke"})
    bcs = [{"name": "bottom", "time": [0.0, 1.0], "x": [0.0, 0.0], "y": [0.0, 0.0],
            "z": [0.0, 0.0]},
           {"name": "top", "time": [0.0, 1.0], "z": [0.0, load]}]
    opts = P.Options(residual_tolerance=1e-8, displacement_tolerance=1e-8, linear_iterations=15,
                     cg_tolerance=1e-10, cg_maximum_iterations=20000)
    return P.Problem("group_cg", mesh, mat, P.dirichlet_boundaries(mesh, bcs), opts)


# block rows: 8, 27, 96 | 120 (15 CTAs), 128 (16), 150 (two levels), 336, 1190, 9261
@pytest.mark.parametrize("element,shape", [
    ("hex8", (1, 1, 1)), ("hex8", (2, 2, 2)), ("hex8", (3, 5, 3)), ("hex8", (3, 5, 4)),
    ("hex8", (3, 3, 7)), ("tet4", (4, 4, 5)), ("hex8", (6, 7, 5)), ("tet4", (6, 9, 16)),
    ("hex8", (20, 20, 20)),
])
def test_persistent_pcg_parity(element, shape, oracle):
    from neon_b200 import api, build
    build.build()
    pr = _problem(element, shape)
    sm = api.StaticMatrix(pr)
    u = sm.solve()
    rep, uo, _, _, _ = oracle.static_solve(pr)
    assert rep["status"] == 0
    assert sm.report["newton_iterations"] == rep["newton_iterations"]
    assert rel_err(u, uo) < 1e-10


def test_persistent_pcg_batch_of_one_and_many_ctas(oracle):
    """Instances of one CTA and of several in one schedule, in both precisions."""
    from neon_b200 import api
    shapes = [(2, 2, 2), (5, 4, 6), (3, 3, 3), (8, 9, 7), (2, 3, 2)]
    problems = [_problem("tet4", s) for s in shapes]
    for precision in (api.FP64, api.MIXED):
        b = api.BatchedStaticMatrix(problems, precision=precision)
        u = b.solve()
        for i, pr in enumerate(problems):
            _, uo, _, _, _ = oracle.static_solve(pr)
            assert rel_err(b.instance_displacement(i, u), uo) < 1e-10


def test_persistent_pcg_iteration_limit():
    """A limit that the solve reaches is reported as neon's computational error, with the count."""
    from neon_b200 import api
    pr = _problem("hex8", (6, 7, 5))
    pr.options.cg_maximum_iterations = 3
    sm = api.StaticMatrix(pr)
    with pytest.raises(api.ComputationalError):
        sm.solve()
    assert sm.report["cg_iterations"] % 3 == 0


def test_persistent_pcg_is_bit_reproducible():
    from neon_b200 import api
    pr = _problem("hex8", (12, 11, 10))
    sm = api.StaticMatrix(pr)
    assert np.array_equal(sm.solve(), sm.solve())


def test_persistent_pcg_with_vectors_in_global_memory():
    """Systems on so few CTAs each (about 500 rows a part) that their vectors do not all fit in shared
    memory, against the same system on all of them: two solutions at CG rtol 1e-10 each, within the
    1e-10 of the parity tests above."""
    from neon_b200 import api
    pr = _problem("tet4", (20, 20, 20))
    u1 = api.StaticMatrix(pr).solve()
    for precision in (api.FP64, api.MIXED):
        b = api.BatchedStaticMatrix([pr] * 16, precision=precision)
        u = b.solve()
        for i in range(16):
            assert rel_err(b.instance_displacement(i, u), u1) < 1e-10
