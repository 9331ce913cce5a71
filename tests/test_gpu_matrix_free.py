"""The matrix-free Newton solves (mf_cg.cu) at sizes past the rule that selects them (an assembled K
beyond 100 MB): ragged boxes whose last element block and warp are partial, every model with an
FP64 operator, both precisions, and a mesh numbered at random, where no neighbouring elements'
products merge and nodes collect theirs from lists of more than four.

The solution is checked through the element kernels and the assembled K, not the operator under
test: at the equilibrium of a solve with Newton tolerance 1e-8 and CG rtol 1e-10 the internal force
of the free DOFs is below 1e-8 of its norm (the residual left by the last correction is its size,
1e-8 of u, times the tangent's nonlinearity and the CG tolerance)."""
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
    "microsphere": (P.Material(P.GAUSS_AFFINE_MICROSPHERE, 10.0, 1.0, segments_per_chain=50.0),
                    0.02),
}


def _problem(model, mesh):
    mat, load = MATERIALS[model]
    bcs = [{"name": "bottom", "time": [0.0, 1.0], "x": [0.0, 0.0], "y": [0.0, 0.0],
            "z": [0.0, 0.0]},
           {"name": "top", "time": [0.0, 1.0], "z": [0.0, load]}]
    opts = P.Options(residual_tolerance=1e-8, displacement_tolerance=1e-8, linear_iterations=15,
                     cg_tolerance=1e-10, cg_maximum_iterations=20000)
    return P.Problem("mf", mesh, mat, P.dirichlet_boundaries(mesh, bcs), opts)


def _free_residual(api, pr, u):
    g = api.SolidMesh(pr.mesh.X, pr.mesh.conn, pr.material)
    g.update_internal_variables(u)
    _, f = g.assemble()
    free = np.ones(len(u), bool)
    for t in pr.dirichlet:
        free[t.dofs] = False
    return np.linalg.norm(f[free]) / np.linalg.norm(f)


@pytest.fixture(scope="module")
def api():
    from neon_b200 import api, build
    build.build()
    return api


@pytest.mark.parametrize("model", list(MATERIALS))
def test_matrix_free_newton_equilibrium(model, api):
    pr = _problem(model, M.structured_hex8(41, 37, 39, jitter=0.05, seed=3))
    u = {}
    for name, precision in (("fp64", api.FP64), ("mixed", api.MIXED)):
        sm = api.StaticMatrix(pr, precision=precision)
        u[name] = sm.solve()
        assert _free_residual(api, pr, u[name]) < 1e-8
    assert rel_err(u["mixed"], u["fp64"]) < 1e-8


def test_matrix_free_newton_on_a_random_numbering(api):
    mesh = M.structured_hex8(41, 37, 39)
    rng = np.random.Generator(np.random.PCG64(5))
    nodes = rng.permutation(mesh.num_nodes)          # new index of every node
    elements = rng.permutation(mesh.num_elements)
    X = np.empty_like(mesh.X)
    X[nodes] = mesh.X
    shuffled = M.Mesh(X=X, conn=nodes[mesh.conn][elements].astype(np.int32),
                      faces={k: nodes[v].astype(np.int32) for k, v in mesh.faces.items()})
    u0 = api.StaticMatrix(_problem("neohooke", mesh)).solve().reshape(-1, 3)
    for precision in (api.FP64, api.MIXED):
        u = api.StaticMatrix(_problem("neohooke", shuffled), precision=precision).solve()
        assert rel_err(u.reshape(-1, 3)[nodes], u0) < 1e-8


def test_the_resident_stiffness_after_a_matrix_free_solve(api):
    """The context holds the last tangent assembled, as after an assembled solve: linear elasticity
    at the last linearisation point, within the parity bar of the assembly."""
    pr = _problem("linear", M.structured_hex8(41, 37, 39))
    sm = api.StaticMatrix(pr)
    u = sm.solve()
    K, _ = sm.mesh.download_system(K=True, f=False)
    g = api.SolidMesh(pr.mesh.X, pr.mesh.conn, pr.material)
    g.update_internal_variables(u)
    K0, _ = g.assemble()
    assert rel_err(K, K0) < 1e-8  # K moves with u, which the last Newton step changes by 1e-8
    assert np.array_equal(u, sm.mesh.displacement())


def test_a_matrix_free_solve_needs_no_second_k_buffer(api):
    """The FP64 K buffer that is zeroed in the background is for assemblies that follow one another; the
    one assembly at the end of an increment goes without.  Free memory falls by that buffer with the
    first assembling pass afterwards, not with the solve."""
    import torch
    pr = _problem("neohooke", M.structured_hex8(41, 37, 39))
    sm = api.StaticMatrix(pr)
    sm.solve()
    after_solve = torch.cuda.mem_get_info()[0]
    sm.mesh.update_assemble_device()
    sm.mesh.synchronize()
    k_bytes = 72 * sm.mesh.nnzb
    assert after_solve - torch.cuda.mem_get_info()[0] >= 0.9 * k_bytes
    K, _ = sm.mesh.download_system(K=True, f=False)
    sm.mesh.update_assemble_device()  # the other buffer
    K1, _ = sm.mesh.download_system(K=True, f=False)
    assert rel_err(K1, K) < 1e-13  # the order of atomic additions
