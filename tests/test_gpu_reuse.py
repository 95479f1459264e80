"""One handle or plan given another matrix or another kind of factor.

The reference keeps one global matrix and preconditioner and builds them
anew on every xsolver_mat_setup and preconditioner setup
(hip/xsolver_c.cpp:274-292), so a program may change both at any time.  Here
a handle rebuilds its plans in place, and the schedule of the exact
triangular solves follows the pattern: whatever the handle did before, every
result has to equal that of a handle that did nothing else, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_cluster import mesh
from test_lines import P5, P7, _stencil
from xsolver_b200 import stencils as st

pytestmark = pytest.mark.gpu


def _setup(S, A):
    """A new matrix on the handle of S."""
    from xsolver_b200.api import check

    S.A, S._rp, S._ci, S._v = A, A.rowptr, A.colidx, A.val
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    check(S._L.xs_mat_setup(S.h, A.n, p(S._rp, C.c_int), p(S._ci, C.c_int), p(S._v, C.c_double), 0), "xs_mat_setup")


def _fresh(A, ksp="bicgstab", pc="ilu0"):
    from xsolver_b200.api import Solver

    return Solver(A).ksp_settype(ksp).ksp_setoption(1e-10, 300, 20).pc_settype(pc)


class tuning:
    """Lines off (boxes from 65536 rows) and / or the single-CTA and cluster solves off."""

    def __init__(self, lines=1, one_cta=1):
        self.lines, self.one_cta = lines, one_cta

    def __enter__(self):
        from xsolver_b200 import _lib

        L = _lib.lib()
        if not self.lines:
            L.xs_set_trsv_lines(0, 0)
        if not self.one_cta:
            L.xs_set_trsv_block_rows(0)
            L.xs_set_trsv_cluster(0)

    def __exit__(self, *exc):
        from xsolver_b200 import _lib

        L = _lib.lib()
        L.xs_set_trsv_lines(1, 512)
        L.xs_set_trsv_block_rows(1 << 30)
        L.xs_set_trsv_cluster(1)


def _patterns():
    """(matrix, tuning at its analysis): cluster, lines, boxes, one CTA, sync-free."""
    M, G, S = mesh(26000, 300, 3, 1), _stencil((24, 25, 26), P7), mesh(300, 20, 2, 2)
    B = _stencil((41, 41, 41), P7)
    return {"cluster": (M, {}), "lines": (G, {}), "boxes": (B, dict(lines=0)), "one_cta": (S, {}),
            "sync_free": (M, dict(one_cta=0))}


@pytest.mark.parametrize("order", [("cluster", "lines", "one_cta", "cluster"), ("one_cta", "lines", "cluster"),
                                   ("cluster", "boxes", "cluster", "lines", "boxes"), ("boxes", "one_cta", "lines")])
def test_matrices_of_different_schedules_on_one_handle(cuda, order):
    """A table of an earlier pattern's schedule is never used for a later one."""
    pats = _patterns()
    S = None
    for name in order:
        A, how = pats[name]
        b = st.rhs_uniform(A.n, 3)
        with tuning(**how):
            if S is None:
                S = _fresh(A)
            else:
                _setup(S, A)
            x = S.solve(b)
            N = _fresh(A)
            assert np.array_equal(x, N.solve(b)), name
            assert S.usediter == N.usediter
            N.close()
    S.close()


def test_reference_style_globals_with_a_second_matrix(cuda):
    """The one global handle of the reference's API: a mesh, then a grid."""
    from xsolver_b200 import api

    for name in ("cluster", "lines"):
        A = _patterns()[name][0]
        b, x = st.rhs_uniform(A.n, 3), np.zeros(A.n)
        assert api.xsolver_mat_setup(A.n, A.rowptr, A.colidx, A.val) == 0
        assert api.xsolver_ksp_settype("bicgstab") == 0
        assert api.xsolver_ksp_setoption(1e-10, 300) == 0
        assert api.xsolver_pc_settype("ilu0") == 0
        assert api.xsolver_solve(b, x) == 0
        r = b - A.to_scipy() @ x
        assert np.linalg.norm(r) <= 1e-9 * np.linalg.norm(b)
    assert api.xsolver_free() == 0


def _parts(A, kind="ilu0", **how):
    """A plan factorised under the given tuning."""
    from xsolver_b200.api import Plan

    with tuning(**how):
        return Plan(A).factor(kind, sweeps=3, fill=2.0, droptol=1e-4)


def _lusolve(P, x, cuda):
    import torch

    dx = torch.from_numpy(np.ascontiguousarray(x)).to(cuda)
    z = torch.full_like(dx, float("nan"))
    (P.lusolve_batch if dx.dim() == 2 else P.lusolve)(dx, z)
    P.sync()
    return z.cpu().numpy()


@pytest.mark.parametrize("dtype,cols", [(np.float64, 0), (np.float32, 0), (np.float64, 3)])
@pytest.mark.parametrize("how", [dict(lines=0, one_cta=0), dict(lines=0)])
def test_factor_of_another_schedule_on_one_plan(cuda, dtype, cols, how):
    """ILU(0) on lines and solved, then a threshold factor of another schedule:
    its first solve does not take what the line solve left in the readiness
    buffers for finished rows."""
    A = _stencil((24, 25, 26), P7) if how.get("one_cta") == 0 else _stencil((41, 41, 41), P7)
    x = st.rhs_uniform(A.n, 5).astype(dtype)
    if cols:
        x = np.stack([st.rhs_uniform(A.n, c) for c in range(cols)], 1)
    P = _parts(A)
    _lusolve(P, x, cuda)
    with tuning(**how):
        P.factor("parilut", sweeps=3, fill=2.0, droptol=1e-4)
        z = [_lusolve(P, x, cuda) for _ in range(2)]
        ref = _lusolve(_parts(A, "parilut", **how), x, cuda)
    assert np.array_equal(z[0], ref) and np.array_equal(z[1], ref)


@pytest.mark.parametrize("batch", [False, True])
def test_same_pattern_size_with_another_schedule_on_one_handle(cuda, batch):
    """A grid on lines, then the same system analysed for the sync-free solve."""
    A = _stencil((24, 25, 26), P7)
    B = np.stack([st.rhs_uniform(A.n, c) for c in range(3)])
    solve = (lambda S: S.solve_batch(B)) if batch else (lambda S: S.solve(B[0]))
    S = _fresh(A, "cg")
    solve(S)
    with tuning(lines=0, one_cta=0):
        _setup(S, A)
        N = _fresh(A, "cg")
        assert np.array_equal(solve(S), solve(N))
    N.close()
    S.close()


@pytest.mark.parametrize("first,second", [((96, 96), (16, 25, 25)), ((80, 80), (25, 16, 16))])
def test_stencils_of_equal_slots_on_one_handle(cuda, first, second):
    """A 5-point and a 7-point pattern whose line schedules have as many slots
    (test_equal_slots_of_different_stencils): ILU(0)'s pivot stream of the
    second is larger by half."""
    systems = [_stencil(first, P5, 1), _stencil(second, P7, 2)]
    S = _fresh(systems[0])
    for A in systems + systems[:1]:
        if S.A is not A:
            _setup(S, A)
        b = st.rhs_uniform(A.n, 3)
        N = _fresh(A)
        assert np.array_equal(S.solve(b), N.solve(b))
        N.close()
    S.close()


@pytest.mark.parametrize("own", ["parilut", "ilup", "ict"])
@pytest.mark.parametrize("A", [st.varcoef3d_7pt(24, 1), st.convdiff3d_27pt(14)], ids=lambda A: A.name)
def test_factors_on_the_matrix_pattern_after_one_on_its_own(cuda, A, own):
    """ILU(0), a threshold factor, then ILU(0), ParILU and IC(0) on one plan:
    none of these works on the threshold factor's triangles."""
    from xsolver_b200.api import Plan

    x = st.rhs_uniform(A.n, 5)
    P = Plan(A).factor("ilu0")
    for kind in ("ilu0", "parilu", "ic0"):
        P.factor(own, sweeps=3, fill=3.0 if own == "parilut" else 20, droptol=1e-4)
        _lusolve(P, x, cuda)
        P.factor(kind, sweeps=4)
        N = Plan(A).factor(kind, sweeps=4)
        assert np.array_equal(P.lu_values(), N.lu_values(), equal_nan=True), kind
        assert np.array_equal(_lusolve(P, x, cuda), _lusolve(N, x, cuda), equal_nan=True), kind


def test_preconditioners_in_turn_on_one_handle(cuda):
    A = st.varcoef3d_7pt(24, 1)
    b, g = st.rhs_uniform(A.n, 3), st.rhs_uniform(A.n, 4)
    S = _fresh(A, "cg")
    for pc in ("ilu0", "parilut", "jacobi", "parilut", "ic0", "ilut", "ilu0", "parilu"):
        S.pc_settype(pc)
        N = _fresh(A, "cg", pc)
        assert np.array_equal(S.solve(b), N.solve(b)), pc
        for a, c in zip(S.adjoint(g), N.adjoint(g)):
            assert np.array_equal(a, c), pc
        N.close()
    S.close()


def test_switch_of_the_exact_solve_reaches_captured_iterations(cuda):
    """A handle that has solved (its iterations captured) takes the sync-free
    solve, two launches, once the cluster solve, one launch, is turned off,
    and the other way round."""
    A = mesh(26000, 300, 3, 1)
    b = st.rhs_uniform(A.n, 3)
    S = _fresh(A)
    x, one = S.solve(b), S.launches()
    with tuning(one_cta=0):
        y, two = S.solve(b), S.launches()
        N = _fresh(A)
        assert np.array_equal(N.solve(b), x) and two == N.launches() > one
        N.close()
    assert np.array_equal(x, y)
    S.solve(b)
    assert S.launches() == one
    S.close()


@pytest.mark.parametrize("prec", ["fp64", "bf16"])
def test_sweeps_and_exact_solves_in_turn_on_one_handle(cuda, prec):
    """A handle with Jacobi sweeps has none of the exact solves' buffers; they
    are there once it is set to exact solves, and both work again after that."""
    A = _stencil((24, 25, 26), P7)
    b = st.rhs_uniform(A.n, 3)

    def fresh(mode):
        S = _fresh(A).pc_set_trsv(mode)
        return S.set_precision("fp64", "fp32", prec).set_inner(1e-2, 100) if prec != "fp64" else S

    S = fresh(3)
    for mode in (3, 0, 3, 0):
        S.pc_set_trsv(mode)
        N = fresh(mode)
        assert np.array_equal(S.solve(b), N.solve(b)), mode
        N.close()
    S.close()
