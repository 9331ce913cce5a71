"""Newton solves that run out of device memory for what they can do without: the matrix-free operator (its
plan, the scratch of its sort, its coefficients), the tiled copy of K, the second K buffer.  They take
the path that needs less and reach the same solution, to the 1e-8 between two paths of the other tests.

A child process fills the device but for a given number of MB before each solve; its kernels are loaded
up front, since loading one needs memory too."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
import torch
from conftest import rel_err
from neon_b200 import api, mesh as M, problem as P

m = M.structured_hex8(*map(int, sys.argv[2].split(",")))
bcs = [{"name": "bottom", "time": [0.0, 1.0], "x": [0.0, 0.0], "y": [0.0, 0.0], "z": [0.0, 0.0]},
       {"name": "top", "time": [0.0, 1.0], "z": [0.0, 0.02]}]
opts = P.Options(residual_tolerance=1e-8, displacement_tolerance=1e-8, linear_iterations=15,
                 cg_tolerance=1e-10, cg_maximum_iterations=20000)
pr = P.Problem("low", m, P.Material(P.NEO_HOOKE, 10.0, 1.0), P.dirichlet_boundaries(m, bcs), opts)
precision = api.MIXED if sys.argv[1] == "mixed" else api.FP64
ref = api.StaticMatrix(pr)
u0 = ref.solve()
ref.mesh.close()
for left in map(int, sys.argv[3:]):
    g = api.SolidMesh(m.X, m.conn, pr.material)
    g.update_internal_variables(np.zeros(g.ndofs))
    if precision == api.FP64:
        g.assemble()
    sm = api.StaticMatrix(pr, precision=precision, mesh=g)
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - (left << 20), dtype=torch.uint8, device="cuda")
    u = sm.solve()
    del fill
    torch.cuda.empty_cache()
    e = rel_err(u, u0)
    print(left, sm.report["newton_iterations"], e, flush=True)
    assert e < 1e-8
    g.close()
print("complete")
"""


BATCH = """
import sys
import ctypes as C
import numpy as np
import torch
from conftest import rel_err
from neon_b200 import api, problem as P

problems = [P.config_c5_instance(m, mu, increments=1) for m, mu in ((24, 0.7), (23, 1.9), (22, 1.2))]
for pr in problems:
    pr.options.residual_tolerance = pr.options.displacement_tolerance = 1e-8
precision = api.MIXED if sys.argv[1] == "mixed" else api.FP64
ref = api.BatchedStaticMatrix(problems, precision=precision, autotune=False)

def launches(g):
    n = C.c_int64()
    api.lib().nb2_launch_count(g.h, C.byref(n))
    return n.value

u0 = ref.solve()
few = launches(ref.mesh)
ref.mesh.close()
b = api.BatchedStaticMatrix(problems, precision=precision, autotune=False)
b.mesh.update_internal_variables(np.zeros(b.mesh.ndofs))
b.mesh.update_assemble_device(precision)
b.mesh.synchronize()
free = torch.cuda.mem_get_info()[0]
fill = torch.empty(free - (int(sys.argv[2]) << 20), dtype=torch.uint8, device="cuda")
u = b.solve()
many = launches(b.mesh)
for i in range(3):
    e = rel_err(b.instance_displacement(i, u), ref.instance_displacement(i, u0))
    print(i, e, b.reports[i]["cg_iterations"], ref.reports[i]["cg_iterations"], few, many, flush=True)
    assert e < 1e-8
    assert abs(b.reports[i]["cg_iterations"] / ref.reports[i]["cg_iterations"] - 1) < 0.05
assert many > 3 * few
print("complete")
"""


def _run(code, precision, *args):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, CUDA_MODULE_LOADING="EAGER",
               PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", code, precision, *args], cwd=root, env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "complete" in r.stdout, r.stdout + r.stderr


def test_small_solve_beside_a_full_device():
    """A few hundred KB are enough for what a call of this size allocates."""
    _run(CHILD, "fp64", "6,7,5", "12", "20", "28")


@pytest.mark.parametrize("precision,left", [("fp64", (20, 24, 26, 28, 30, 40, 56, 72)),
                                            ("mixed", (64, 72, 80, 88, 96))])
def test_matrix_free_solve_with_little_memory(precision, left):
    _run(CHILD, precision, "41,37,39", *map(str, left))


@pytest.mark.parametrize("precision,left", [("fp64", 30), ("mixed", 22)])
def test_batch_without_the_tiled_copy(precision, left):
    """The copy of K that the persistent PCG reads (54 MB here, 27 in FP32) does not fit: the chunk
    kernels solve the batch, with the same iterations but for the order of sums."""
    _run(BATCH, precision, str(left))
