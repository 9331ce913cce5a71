"""The matrix-free J2 operators at plastic points, hardening and softening.  With a negative hardening
modulus mu' = G sigma_y / q is negative where the yield stress of the present state is, and b positive
where that of the last one is; the operators have to be the assembled K there too.

FP32: the product against the assembled K, to the rounding bar of the FP32 product's other tests.
Newton solves, FP64 and mixed (whose residuals are FP64): past the size that runs matrix-free, with every
DOF prescribed but those of a few interior nodes (a linear system that CG solves exactly whatever its
signs), against the same Newton steps with the downloaded K and a dense solve.  Both solve the same linear
systems, CG to 1e-12, so the norms of the log agree to 1e-8 relative while they are within 1e-6 of the
largest (1e-12 of rounding over 1e-6, with a factor of 100 for the Newton map), and the displacements to
1e-10."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import random_displacement, rel_err
from neon_b200 import mesh as M
from neon_b200 import problem as P

pytestmark = pytest.mark.gpu


def _material(hardening):
    return P.make_material({"elastic_modulus": 200e3, "poissons_ratio": 0.3, "yield_stress": 200.0,
                            "isotropic_hardening_modulus": hardening},
                           {"name": "J2_plasticity", "finite_strain": False})


@pytest.fixture(scope="module")
def api():
    from neon_b200 import api, build
    build.build()
    return api


@pytest.mark.parametrize("topo", ["hex8", "tet4"])
@pytest.mark.parametrize("hardening", [1e3, -1e5])
def test_fp32_product_at_plastic_points(api, topo, hardening):
    m = M.structured_hex8(4, 3, 3, jitter=0.1, seed=3) if topo == "hex8" else \
        M.structured_tet4(3, 2, 2)
    g = api.SolidMesh(m.X, m.conn, _material(hardening))
    u = random_displacement(m, 1.0, 11)
    u *= 0.03 / np.abs(u).max()
    v = np.random.Generator(np.random.PCG64(9)).standard_normal(g.ndofs)
    for scale in (0.02, 0.5, 1.0, 1.2):  # elastic; plastic; and on from a plastic state, twice
        g.update_internal_variables(scale * u)
        K, _ = g.assemble()
        rp, col = g.sparsity_pattern()
        y = sp.csr_matrix((K, col, rp), shape=(g.ndofs, g.ndofs)) @ v
        assert rel_err(g.apply_tangent_fp32(v), y) < 2e-5, scale
        g.save_internal_variables(True)
    ebar = g.quadrature_values("accumulated_plastic_strain")
    assert (ebar > 0).mean() > 0.5 and ((200.0 + hardening * ebar) < 0).any() == (hardening < 0)


def _prescribed(hardening):
    """A box stretched along z by a quadratic displacement in two increments, everywhere prescribed
    but at four interior nodes."""
    m = M.structured_hex8(41, 37, 39)
    node = np.arange(m.num_nodes).reshape(40, 38, 42)
    free = np.array([node[5, 9, 11], node[17, 20, 20], node[17, 21, 20], node[33, 30, 7]])
    held = np.setdiff1d(np.arange(m.num_nodes), free)
    tables = [P.DofTable(np.sort(np.concatenate([3 * held, 3 * held + 1])).astype(np.int32),
                         np.array([0.0, 1.0]), np.zeros(2))]
    for k in range(40):
        z = k / 39.0
        layer = np.setdiff1d(node[k].reshape(-1), free)
        tables.append(P.DofTable((3 * layer + 2).astype(np.int32), np.array([0.0, 1.0]),
                                 np.array([0.0, 0.012 * z * z])))
    # softening diverges sooner or later: its first increment, three steps, and no convergence asked for
    soft = hardening < 0
    opts = P.Options(residual_tolerance=1e-30 if soft else 1e-7, displacement_tolerance=1e-9,
                     absolute_tolerance=True, linear_iterations=3 if soft else 12, initial=0.5,
                     minimum=0.5, maximum=0.5, adaptive=False, cg_tolerance=1e-12,
                     cg_maximum_iterations=200)
    dofs = (3 * free[:, None] + np.arange(3)).reshape(-1)
    return P.Problem("j2", m, _material(hardening), tables, opts), dofs


def _reference(api, pr, free):
    g = api.SolidMesh(pr.mesh.X, pr.mesh.conn, pr.material)
    rp, col = g.sparsity_pattern()
    n = g.ndofs
    top = np.zeros(n)
    for t in pr.dirichlet:
        top[t.dofs] = t.values[-1]
    u_old, log = np.zeros(n), []
    g.update_internal_variables(u_old)
    for _ in range(2):
        u = u_old.copy()
        for k in range(pr.options.linear_iterations):
            g.update_internal_variables(u)
            K, f = g.assemble()
            A = sp.csr_matrix((K, col, rp), shape=(n, n))
            rhs = -f
            if k == 0:
                rhs -= A @ (0.5 * top)
                u += 0.5 * top
            du = np.linalg.solve(A[free][:, free].toarray(), rhs[free])
            u[free] += du
            log.append((np.linalg.norm(du), np.linalg.norm(rhs[free])))
            if log[-1][0] <= 1e-9 and log[-1][1] <= pr.options.residual_tolerance:
                break
        else:
            break
        g.update_internal_variables(u)
        g.save_internal_variables(True)
        u_old = u
    ebar = g.quadrature_values("accumulated_plastic_strain")
    assert (ebar > 0).mean() > 0.2
    assert (200.0 + pr.material.hardening * ebar < 0).any() == (pr.material.hardening < 0)
    return u, np.array(log)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("hardening", [1e3, -1e5])
def test_newton_at_plastic_points(api, hardening, precision):
    pr, free = _prescribed(hardening)
    ur, ref = _reference(api, pr, free)
    sm = api.StaticMatrix(pr, precision=api.MIXED if precision == "mixed" else api.FP64)
    u = sm.solve(raise_on_error=False)
    got = sm.log[:len(ref), 3:5]
    far = ref > 1e-6 * ref.max(0)
    assert far.sum() >= 6
    np.testing.assert_allclose(got[far], ref[far], rtol=1e-8)
    if hardening > 0:
        assert len(sm.log) == len(ref)
        assert rel_err(u, ur) < 1e-10
