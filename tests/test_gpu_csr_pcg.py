"""The CSR solve at the row lengths where its SpMV changes path: rows inside, at and beyond the 96
entries it requests at once, single-entry rows, sizes that leave warps without a row or with several.

Diagonally dominant symmetric systems: |off-diagonal row sum| <= 1/2 diagonal, so after Jacobi scaling
the condition number is at most 3 and a relative residual of 1e-13 leaves at most sqrt(ratio of diagonals)
* 3e-13 in x; 1e-11 covers the diagonal ratio (up to ~200) with a margin."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, width, seed):
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for i in range(n):
        if i % 5 == 4:  # a row with its diagonal alone
            continue
        j = np.arange(i + 1, min(n, i + 1 + width // 2))
        j = j[j % 5 != 4]
        A[i, j] = rng.uniform(-1, 1, j.size)
    A += A.T
    A[np.arange(n), np.arange(n)] = 2.0 * np.abs(A).sum(1) + 1.0
    rows = [np.flatnonzero(A[i]) for i in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    return A, rp, col, A[np.repeat(np.arange(n), np.diff(rp)), col]


@pytest.mark.parametrize("n,width", [(1, 2), (33, 8), (130, 120), (500, 240), (4801, 100)])
def test_csr_solve_over_row_lengths(n, width):
    from neon_b200 import api
    A, rp, col, val = _system(n, width, 11)
    b = np.random.default_rng(3).standard_normal(n)
    x = np.zeros(n)
    api.ConjugateGradient(1e-13, 1000).solve((rp, col, val), x, b)
    ref = np.linalg.solve(A, b)
    assert np.linalg.norm(x - ref) <= 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("bad", [-1, 33])
def test_csr_solve_refuses_columns_outside_the_matrix(bad):
    from neon_b200 import api
    _, rp, col, val = _system(33, 8, 5)
    col[len(col) // 2] = bad
    x = np.full(33, 7.0)
    it, err, rhs = C.c_int32(-3), C.c_double(-3.0), np.ones(33)
    st = api.lib().nb2_pcg_solve(33, rp.ctypes.data, col.ctypes.data, val.ctypes.data,
                                 rhs.ctypes.data, x.ctypes.data, 1e-12, 100,
                                 C.byref(it), C.byref(err))
    assert st == api.E_INPUT and (x == 7.0).all() and it.value == -3 and err.value == -3.0
