"""New values on a handle whose iterations are captured in graphs.

The reference re-reads its matrix on every solve (hip/xsolver_c.cpp:274-292);
here the iteration bodies are captured into CUDA graphs, and new values can
replace buffers those graphs name: the adjoint's transposed operator and
factors are rebuilt, a ParILUT factor gets a new pattern.  A graph must then
be captured anew: every pass has to equal the first pass of a new handle."""
import numpy as np
import pytest

from xsolver_b200 import stencils as st

pytestmark = pytest.mark.gpu


def _solver(A, ksp, pc):
    from xsolver_b200.api import Solver

    S = Solver(A).ksp_settype(ksp).ksp_setoption(1e-12, 1000, 30).pc_settype(pc)
    if pc == "parilut":
        S.pc_setparilut(2.0, 3, 1e-4)
    return S


@pytest.mark.parametrize("ksp,pc,grid", [("cg", "ilu0", 14), ("bicgstab", "parilut", 14), ("gmres", "parilut", 12),
                                         ("bicgstab", "jacobi", 14)])
def test_update_solve_adjoint_repeated(cuda, ksp, pc, grid):
    fields = [st.varcoef3d_7pt(grid, s) for s in range(4)]
    S = _solver(fields[0], ksp, pc)
    b, g = st.rhs_uniform(fields[0].n, 1), st.rhs_uniform(fields[0].n, 2)
    for A in fields[1:] + fields[1:2]:
        S.mat_update(A.val)
        x = S.solve(b)
        db, dA = S.adjoint(g)
        N = _solver(A, ksp, pc)
        assert np.array_equal(x, N.solve(b))
        db1, dA1 = N.adjoint(g)
        assert np.array_equal(db, db1) and np.array_equal(dA, dA1)
        N.close()


def test_update_batch_repeated(cuda):
    fields = [st.varcoef3d_7pt(14, s) for s in range(3)]
    S = _solver(fields[0], "cg", "ilu0")
    B = np.stack([st.rhs_uniform(fields[0].n, c) for c in range(3)])
    for A in fields[1:] + fields[1:2]:
        S.mat_update(A.val)
        X = S.solve_batch(B)
        DB, DA = S.adjoint_batch(X, X - 0.5)
        N = _solver(A, "cg", "ilu0")
        assert np.array_equal(X, N.solve_batch(B))
        DB1, DA1 = N.adjoint_batch(X, X - 0.5)
        assert np.array_equal(DB, DB1) and np.array_equal(DA, DA1)
        N.close()
