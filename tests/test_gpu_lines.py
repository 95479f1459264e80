"""Line-scheduled exact triangular solves on the GPU.

The schedule (xs_tri_lines) replaces the row-per-thread dependency flags of
the reference's sync-free solves (hip/Precond/gpuparilu.cpp:257-364) on
stencil patterns.  It changes only which thread computes a row, when, and
where a dependency is read from; each row's entries are summed in the same
order with the same operations, so FP64 results are bitwise the oracle's
LUsolve (hip/HostMatrix/HostMatrixCSR.cpp:385-409) and reduced precisions
bitwise the level-ordered solve's."""
import numpy as np
import pytest

import oracle
from test_lines import P5, P7, P9, P27, _stencil
from xsolver_b200 import stencils as st

pytestmark = pytest.mark.gpu


class lines_mode:
    """Line schedule forced for every qualifying triangle (mode 2) or off (0)."""

    def __init__(self, mode):
        self.mode = mode

    def __enter__(self):
        from xsolver_b200 import _lib

        assert _lib.lib().xs_set_trsv_lines(self.mode, 8) == 0

    def __exit__(self, *exc):
        from xsolver_b200 import _lib

        _lib.lib().xs_set_trsv_lines(1, 512)


def _on_lines(P):
    return P.schedule()["L"] == P.schedule()["U"] == "lines" and P.schedule()["lu"] == "halves"


def _dev(a, cuda):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def _lusolve(P, x, cuda, reps=1, t=False):
    import torch

    dx = _dev(x, cuda)
    out = []
    for _ in range(reps):
        z = torch.full_like(dx, float("nan"))
        (P.lusolve_t if t else P.lusolve)(dx, z)
        P.sync()
        out.append(z.cpu().numpy())
    return out


# patterns with a kernel instance of their own beside 5, 7 and 27 points
P19 = [o for o in P27 if sum(map(abs, o)) <= 2]
P13 = P9 + [(0, 2), (0, -2), (2, 0), (-2, 0)]

# one line and one step around a patch (32-128 lines) and a stage (8 steps),
# several patches in Y and Z, lines shorter and longer than the ring (64)
SHAPES = [((9, 11, 10), P7), ((17, 33, 9), P7), ((16, 8, 64), P7), ((33, 17, 71), P7), ((40, 41, 42), P7),
          ((12, 13, 14), P27), ((17, 33, 20), P27), ((129, 63), P5), ((128, 128), P5), ((7, 300), P5), ((300, 9), P9),
          ((11, 12, 13), P19), ((17, 33, 9), P19), ((129, 63), P13), ((9, 300), P13), ((129, 63), P9)]


@pytest.mark.parametrize("shape,offs", SHAPES)
def test_lusolve_fp64_bitwise_vs_oracle(cuda, shape, offs):
    from xsolver_b200.api import Plan

    A = _stencil(shape, offs)
    F = oracle.ilu0(A)
    x = st.rhs_uniform(A.n, 7)
    with lines_mode(2):
        P = Plan(A).factor("ilu0")
        assert _on_lines(P)
        for z in _lusolve(P, x, cuda, reps=4):  # both halves of the exchange buffer, re-armed
            assert np.array_equal(z, oracle.lusolve(F, x))
        (zt,) = _lusolve(P, x, cuda, t=True)
        assert np.allclose(zt, oracle.lusolve_t(F, x), rtol=1e-12, atol=1e-12)


def test_parilut_fill_bitwise_vs_oracle(cuda):
    from xsolver_b200.api import Plan

    A = st.convdiff3d_27pt(24)
    F = oracle.parilut(A, fill=2.0, sweeps=5, droptol=1e-4)
    x = st.rhs_uniform(A.n, 5)
    with lines_mode(2):
        P = Plan(A).factor("parilut", sweeps=5, fill=2.0, droptol=1e-4)
        assert _on_lines(P)
        (z,) = _lusolve(P, x, cuda)
    assert np.array_equal(z, oracle.lusolve(F, x))


@pytest.mark.parametrize("prec", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("shape,offs", [((17, 33, 20), P27), ((33, 17, 71), P7), ((129, 63), P5),
                                        ((17, 33, 20), P19), ((129, 63), P9), ((129, 63), P13)])
def test_reduced_precision_equals_level_ordered(cuda, prec, shape, offs):
    from xsolver_b200 import _lib
    from xsolver_b200.api import Plan

    A = _stencil(shape, offs)
    x = st.rhs_uniform(A.n, 9).astype(np.float32)
    outs = []
    _lib.lib().xs_set_trsv_block_rows(0)
    try:
        for mode in (2, 0):
            with lines_mode(mode):
                P = Plan(A).factor("ilu0").set_factor_precision(prec)
                assert _on_lines(P) == (mode == 2)
                outs.append(_lusolve(P, x, cuda, reps=2))
    finally:
        _lib.lib().xs_set_trsv_block_rows(1 << 30)
    for z in outs[0]:
        assert np.array_equal(z, outs[1][0])


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 16])
@pytest.mark.parametrize("shape,offs", [((33, 17, 30), P7), ((12, 13, 14), P27), ((12, 13, 14), P19), ((33, 40), P9),
                                        ((33, 40), P13)])
def test_several_right_hand_sides_equal_single_solves(cuda, k, shape, offs):
    import torch
    from xsolver_b200.api import Plan

    A = _stencil(shape, offs)
    F = oracle.ilu0(A)
    X = np.stack([st.rhs_uniform(A.n, c) for c in range(k)], 1)
    with lines_mode(2):
        P = Plan(A).factor("ilu0")
        assert _on_lines(P)
        dX = _dev(X, cuda)
        for _ in range(2):
            Z = torch.full_like(dX, float("nan"))
            P.lusolve_batch(dX, Z)
            P.sync()
            for c in range(k):
                assert np.array_equal(Z[:, c].cpu().numpy(), oracle.lusolve(F, X[:, c]))


@pytest.mark.parametrize("shape,offs,ks", [((130, 120, 9), P7, (2, 3, 4, 16)), ((72, 72, 9), P27, (11, 12, 15, 16)),
                                           ((3200, 130), P5, (14, 15, 16))])
def test_columns_on_both_sides_of_two_per_line(cuda, shape, offs, ks):
    """Systems of many patches (135, 90 and 25), with fewer and with more
    columns than give a line two of them (on 148 SMs 370 patches times columns
    for 5- and 7-point patterns, 1036 for 27-point ones), odd counts among them."""
    import torch
    from xsolver_b200.api import Plan

    A = _stencil(shape, offs)
    F = oracle.ilu0(A)
    P = Plan(A).factor("ilu0")
    assert _on_lines(P)
    X = np.stack([st.rhs_uniform(A.n, c) for c in range(max(ks))], 1)
    ref = np.stack([oracle.lusolve(F, X[:, c]) for c in range(max(ks))], 1)
    for k in ks:
        dX = _dev(X[:, :k], cuda)
        Z = torch.full_like(dX, float("nan"))
        P.lusolve_batch(dX, Z)
        P.sync()
        assert np.array_equal(Z.cpu().numpy(), ref[:, :k]), k


@pytest.mark.parametrize("k", [2, 3, 16])
def test_several_right_hand_sides_of_a_long_reach(cuda, k):
    """A skewed 7-point pattern whose steps reach back so far that only one
    column of a line fits in shared memory."""
    import torch
    from xsolver_b200.api import Plan

    offs = [(0, 1), (1, -8), (2, 8)]
    A = _stencil((40, 128), [(0, 0)] + offs + [(-a, -b) for a, b in offs])
    F = oracle.ilu0(A)
    X = np.stack([st.rhs_uniform(A.n, c) for c in range(k)], 1)
    P = Plan(A).factor("ilu0")
    assert _on_lines(P)
    dX = _dev(X, cuda)
    Z = torch.full_like(dX, float("nan"))
    P.lusolve_batch(dX, Z)
    P.sync()
    for c in range(k):
        assert np.array_equal(Z[:, c].cpu().numpy(), oracle.lusolve(F, X[:, c]))


def test_one_triangle_on_lines_the_other_not(cuda):
    """A lower triangle that qualifies beside an upper one that does not: each
    kernel re-arms what the other polls, in either order."""
    from xsolver_b200 import CSRMatrix, _lib
    from xsolver_b200.api import Plan

    A = _stencil((20, 21, 22), P7, 2)
    rows = np.repeat(np.arange(A.n), np.diff(A.rowptr))
    drop = np.random.default_rng(0).random(A.nnz) < 0.5
    x = st.rhs_uniform(A.n, 3)
    _lib.lib().xs_set_trsv_block_rows(0)
    try:
        for part in (A.colidx > rows, A.colidx < rows):
            keep = ~(drop & part)
            rp = np.zeros(A.n + 1, np.int64)
            np.cumsum(np.bincount(rows[keep], minlength=A.n), out=rp[1:])
            B = CSRMatrix(A.n, rp, A.colidx[keep], A.val[keep])
            F = oracle.ilu0(B)
            with lines_mode(2):
                P = Plan(B).factor("ilu0")
                assert (P.schedule()["L"] == "lines") != (P.schedule()["U"] == "lines")
                for z in _lusolve(P, x, cuda, reps=3):
                    assert np.array_equal(z, oracle.lusolve(F, x))
    finally:
        _lib.lib().xs_set_trsv_block_rows(1 << 30)


def test_wait_times_out_and_recovers(cuda):
    """A patch that waits for a value nothing publishes: the bounded wait gives
    up after about 1 s, the error is reported, and the plan works again."""
    from xsolver_b200.api import Plan, XsError

    A = st.poisson3d_7pt(24)
    F = oracle.ilu0(A)
    x = st.rhs_uniform(A.n, 1)
    with lines_mode(2):
        P = Plan(A).factor("ilu0")
        assert _on_lines(P)
        P.debug_break_dependency(A.n - 1, True)
        with pytest.raises(XsError) as e:
            _lusolve(P, x, cuda)
        assert e.value.code == 5  # XS_ERR_TRSV_TIMEOUT
        P.debug_break_dependency(A.n - 1, False)
        for z in _lusolve(P, x, cuda, reps=2):
            assert np.array_equal(z, oracle.lusolve(F, x))


def test_wait_times_out_with_more_patches_than_ctas(cuda):
    """The same in the middle of a system whose CTAs take several patches
    each: every CTA ends with its copies landed and its stage barriers in
    step, and later solves are right."""
    from xsolver_b200.api import Plan, XsError

    A = _stencil((200, 210, 16), P7)  # 350 patches
    x = st.rhs_uniform(A.n, 1)
    with lines_mode(2):
        P = Plan(A).factor("ilu0")
        (ref,) = _lusolve(P, x, cuda)
        P.debug_break_dependency(A.n // 2, True)
        with pytest.raises(XsError) as e:
            _lusolve(P, x, cuda)
        assert e.value.code == 5  # XS_ERR_TRSV_TIMEOUT
        P.debug_break_dependency(A.n // 2, False)
        for z in _lusolve(P, x, cuda, reps=3):
            assert np.array_equal(z, ref)


def test_infinities_and_nans_pass_through(cuda):
    """Infinities and NaNs in the right-hand side spread as in the sequential
    solve; a NaN that is not the marker is published like any value."""
    from xsolver_b200.api import Plan

    A = _stencil((17, 18, 19), P7)
    F = oracle.ilu0(A)
    x = st.rhs_uniform(A.n, 2)
    x[1000], x[3000] = np.inf, np.nan
    with lines_mode(2):
        P = Plan(A).factor("ilu0")
        assert _on_lines(P)
        (z,) = _lusolve(P, x, cuda)
    assert np.array_equal(z, oracle.lusolve(F, x), equal_nan=True)


@pytest.mark.parametrize("shape", [(9, 11, 10), (17, 33, 9), (40, 41, 42), (33, 17, 71), (129, 63), (7, 300), (128, 128)])
def test_ilu0_on_lines_bitwise_vs_oracle(cuda, shape):
    """ILU(0) of 5- and 7-point patterns on the line schedule: the reference's
    factors bit for bit, also where an entry has no transposed one, and a
    pivot near zero takes the reference's substitute."""
    from xsolver_b200 import CSRMatrix
    from xsolver_b200.api import Plan

    A = _stencil(shape, P7 if len(shape) == 3 else P5, 3)
    rows = np.repeat(np.arange(A.n), np.diff(A.rowptr))
    rng = np.random.default_rng(5)
    for M in (A, None):
        if M is None:  # one-sided couplings, and a first pivot of zero
            keep = (A.colidx == rows) | (rng.random(A.nnz) < 0.96)
            rp = np.zeros(A.n + 1, np.int64)
            np.cumsum(np.bincount(rows[keep], minlength=A.n), out=rp[1:])
            M = CSRMatrix(A.n, rp, A.colidx[keep], A.val[keep])
            M.val[0] = 0.0
        with lines_mode(2):
            P = Plan(M).factor("ilu0")
            assert P.schedule()["ilu0"] == "lines"
            assert np.array_equal(P.lu_values(), oracle.ilu0_values(M))
            assert np.array_equal(P.factor("ilu0").lu_values(), oracle.ilu0_values(M))  # refactorised


def test_repeated_columns_keep_their_order(cuda):
    """A row with the same column twice is solved by a schedule that keeps both entries."""
    from xsolver_b200 import CSRMatrix
    from xsolver_b200.api import Plan

    A = _stencil((12, 13, 14), P7, 1)
    e = int(A.rowptr[700])  # repeat the first (lower) entry of row 700
    ci, v = np.insert(A.colidx, e, A.colidx[e]), np.insert(A.val, e, -0.25)
    rp = A.rowptr.copy()
    rp[701:] += 1
    B = CSRMatrix(A.n, rp, ci, v)
    x = st.rhs_uniform(A.n, 1)
    with lines_mode(2):
        P = Plan(B).factor("ilu0")
        assert P.schedule()["L"] != "lines"
        (z,) = _lusolve(P, x, cuda)
        F = P.factors()
    y = np.zeros(A.n)
    for r in range(A.n):
        acc = x[r]
        for q in range(F["lrp"][r], F["lrp"][r + 1]):
            acc = acc - y[F["lci"][q]] * F["lv"][q]
        y[r] = acc
    w = np.zeros(A.n)
    for r in range(A.n - 1, -1, -1):
        acc = y[r] * F["dinv"][r]
        for q in range(F["urp"][r + 1] - 1, F["urp"][r] - 1, -1):
            acc = acc - w[F["uci"][q]] * F["uv"][q]
        w[r] = acc
    assert np.array_equal(z, w)
