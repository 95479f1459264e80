"""GMRES with a step's orthogonalisation in one kernel.

The kernel keeps w in registers and exchanges the coefficients through grid
barriers; the modified Gram-Schmidt order is that of the reference
(intel/mpisolver-C-v1.cpp:982-1010, flexible form :1089-1247).  Sizes sit
around the edges of its split: less than a thread's vector, odd sizes (no
16-byte loads), one CTA and around it, every CTA, several chunks per thread.
Both solutions solve a system with condition number below 4 to 1e-13, so
they agree to 1e-12."""
import numpy as np
import pytest

import oracle
from xsolver_b200 import CSRMatrix
from xsolver_b200 import stencils as st

pytestmark = pytest.mark.gpu


def tridiag(n, seed):
    rng = np.random.default_rng(seed)
    lo, up = -rng.uniform(0.5, 1.5, n), -rng.uniform(0.5, 1.5, n)
    v = np.stack([lo, np.full(n, 6.0), up], 1)
    c = np.arange(n)[:, None] + np.array([-1, 0, 1])
    ok = (c >= 0) & (c < n)
    return CSRMatrix(n, np.concatenate([[0], np.cumsum(ok.sum(1))]), c[ok], v[ok])


@pytest.mark.parametrize("n", [1, 2, 3, 5, 1023, 1024, 2047, 2048, 2049, 4097, 151552, 151553, 303104, 303106, 606211,
                               700002, 1212416])
@pytest.mark.parametrize("restart", [1, 5])
def test_fgmres_matches_oracle(cuda, n, restart):
    from xsolver_b200.api import Solver

    A = tridiag(n, n)
    b = st.rhs_uniform(n, 1)
    S = Solver(A).ksp_settype("gmres").ksp_setoption(1e-13, 200, restart).pc_settype("jacobi")
    x = S.solve(b)
    assert np.array_equal(S.solve(b), x)  # the barrier is re-armed, the graph replayed
    xo, _, _ = oracle.solve("fgmres", A, b, tol=1e-13, maxiter=200, restart=restart, pc="jacobi", quirk=0)
    assert np.linalg.norm(x - xo) <= 1e-12 * np.linalg.norm(xo)


@pytest.mark.parametrize("n", [5, 2051, 303105, 606212])
def test_fp32_inner_iteration(cuda, n):
    from xsolver_b200.api import Solver

    A = tridiag(n, n)
    b = st.rhs_uniform(n, 1)
    S = Solver(A).ksp_settype("gmres").ksp_setoption(1e-12, 200, 6).pc_settype("jacobi")
    S.set_precision("fp64", "fp32", "fp32").set_inner(1e-4, 60)
    x = S.solve(b)
    xo, _, _ = oracle.solve("fgmres", A, b, tol=1e-13, maxiter=200, restart=30, pc="jacobi", quirk=0)
    assert np.linalg.norm(x - xo) <= 1e-11 * np.linalg.norm(xo)
