"""Exact LU solves on one thread-block cluster (patterns without a grid).

The kernel keeps the solution in the cluster's distributed shared memory in
place of the readiness flags of the reference's sync-free solves
(hip/Precond/gpuparilu.cpp:257-364).  Rows are summed in the same order with
the same operations, so FP64 results are bitwise the oracle's LUsolve
(hip/HostMatrix/HostMatrixCSR.cpp:385-409) and reduced precisions bitwise
the sync-free solve's."""
import numpy as np
import pytest

import oracle
from xsolver_b200 import CSRMatrix
from xsolver_b200 import stencils as st

pytestmark = pytest.mark.gpu


class cluster_mode:
    """Cluster solve (1) or sync-free solve (0), the single-CTA solve off."""

    def __init__(self, on):
        self.on = on

    def __enter__(self):
        from xsolver_b200 import _lib

        assert _lib.lib().xs_set_trsv_cluster(self.on) == 0
        assert _lib.lib().xs_set_trsv_block_rows(0) == 0

    def __exit__(self, *exc):
        from xsolver_b200 import _lib

        _lib.lib().xs_set_trsv_cluster(1)
        _lib.lib().xs_set_trsv_block_rows(1 << 30)


def mesh(n, reach, per_row, seed=0, dense_rows=0):
    """Random couplings within `reach` rows (no grid); dense_rows rows with up to 60 more."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), per_row)
    c = r + rng.integers(-reach, reach + 1, len(r))
    if dense_rows:
        d = rng.integers(0, n, dense_rows)
        r = np.concatenate([r, np.repeat(d, 60)])
        c = np.concatenate([c, np.repeat(d, 60) + rng.integers(-reach, reach + 1, 60 * dense_rows)])
    ok = (c >= 0) & (c < n)
    key = np.unique(np.concatenate([r[ok] * n + c[ok], c[ok] * n + r[ok], np.arange(n) * (n + 1)]))
    r, c = key // n, key % n
    v = rng.uniform(-1.0, -0.3, len(r))
    cnt = np.bincount(r, minlength=n)
    v[r == c] = 1.2 * cnt
    return CSRMatrix(n, np.concatenate([[0], np.cumsum(cnt)]), c, v)


def _lusolve(P, x, cuda, reps=1):
    import torch

    dx = torch.from_numpy(np.ascontiguousarray(x)).to(cuda)
    out = []
    for _ in range(reps):
        z = torch.full_like(dx, float("nan"))
        P.lusolve(dx, z)
        P.sync()
        out.append(z.cpu().numpy())
    return out


# one row, one group, one round of the cluster's groups (16 x 32) and around
# them, several rounds; chains (every row on the one before), rows of more
# than one and more than four chunks of entries, rows without entries
CASES = [(1, 1, 0, 0), (31, 4, 2, 0), (33, 4, 2, 0), (511, 9, 2, 0), (513, 30, 3, 0), (3000, 40, 3, 5), (2000, 1, 2, 0),
         (40000, 700, 3, 20), (70000, 2000, 4, 0), (5000, 2500, 0, 3)]


@pytest.mark.parametrize("n,reach,per_row,dense", CASES)
def test_lusolve_fp64_bitwise_vs_oracle(cuda, n, reach, per_row, dense):
    from xsolver_b200.api import Plan

    A = mesh(n, reach, per_row, n, dense)
    F = oracle.ilu0(A)
    x = st.rhs_uniform(n, 7)
    with cluster_mode(1):
        P = Plan(A).factor("ilu0")
        assert P.schedule()["lu"] == ("cluster" if F.lci.size else "halves")  # one row: nothing to hand over
        for z in _lusolve(P, x, cuda, reps=3):
            assert np.array_equal(z, oracle.lusolve(F, x))


@pytest.mark.parametrize("prec", ["fp32", "bf16", "fp16"])
def test_reduced_precision_equals_sync_free(cuda, prec):
    from xsolver_b200.api import Plan

    A = mesh(9000, 300, 3, 1, 10)
    x = st.rhs_uniform(A.n, 9).astype(np.float32)
    outs = []
    for on in (1, 0):
        with cluster_mode(on):
            P = Plan(A).factor("ilu0").set_factor_precision(prec)
            assert P.schedule()["lu"] == ("cluster" if on else "halves")
            outs += _lusolve(P, x, cuda, reps=2)
    for z in outs[1:]:
        assert np.array_equal(z, outs[0])


def test_wait_times_out_and_recovers(cuda):
    """A row made to wait for itself: the bounded wait gives up after about
    1 s, the error is reported, and the plan works again."""
    from xsolver_b200.api import Plan, XsError

    A = mesh(3000, 40, 3, 2)
    F = oracle.ilu0(A)
    x = st.rhs_uniform(A.n, 1)
    with cluster_mode(1):
        P = Plan(A).factor("ilu0")
        assert P.schedule()["lu"] == "cluster"
        P.debug_break_dependency(A.n - 1, True)
        with pytest.raises(XsError) as e:
            _lusolve(P, x, cuda)
        assert e.value.code == 5  # XS_ERR_TRSV_TIMEOUT
        P.debug_break_dependency(A.n - 1, False)
        for z in _lusolve(P, x, cuda, reps=2):
            assert np.array_equal(z, oracle.lusolve(F, x))


def test_infinities_and_nans_pass_through(cuda):
    from xsolver_b200.api import Plan

    A = mesh(3000, 40, 3, 3)
    F = oracle.ilu0(A)
    x = st.rhs_uniform(A.n, 2)
    x[100], x[2000] = np.inf, np.nan
    with cluster_mode(1):
        (z,) = _lusolve(Plan(A).factor("ilu0"), x, cuda)
    assert np.array_equal(z, oracle.lusolve(F, x), equal_nan=True)


def test_whole_solve_matches_sync_free(cuda):
    from xsolver_b200.api import Solver

    A = mesh(30000, 500, 3, 4)
    b = st.rhs_uniform(A.n, 4)
    res = []
    for on in (1, 0):
        with cluster_mode(on):
            S = Solver(A).ksp_settype("bicgstab").ksp_setoption(1e-10, 500).pc_settype("ilu0")
            res.append((S.solve(b), S.resvec()))
            S.close()
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])


@pytest.mark.parametrize("n,reach,per_row,path",
                         [(4095, 4000, 1, "one_cta"), (4096, 60, 3, "one_cta"), (8000, 7900, 2, "cluster"),
                          (24000, 4000, 6, "cluster"), (25600, 60, 3, "one_cta"), (25601, 60, 3, "cluster"),
                          (10000, 300, 3, "one_cta"), (10000, 300, 5, "cluster"), (10000, 300, 7, "one_cta"),
                          (10000, 60, 5, "one_cta"), (4000, 300, 5, "one_cta")])
def test_default_choice_bitwise_vs_oracle(cuda, n, reach, per_row, path):
    """Where the solve in one CTA hands over to the cluster: never below 4096
    rows, above them where a staged batch holds fewer than three average
    levels, where the solution leaves its shared memory, and on wide enough
    levels of rows with four or five entries."""
    from xsolver_b200.api import Plan

    A = mesh(n, reach, per_row, n)
    x = st.rhs_uniform(n, 3)
    P = Plan(A).factor("ilu0")
    assert P.schedule()["L"] == "levels" and P.schedule()["lu"] == path
    for z in _lusolve(P, x, cuda, reps=2):
        assert np.array_equal(z, oracle.lusolve(oracle.ilu0(A), x))


@pytest.mark.parametrize("shape", [(15, 16, 17), (16, 16, 16), (8, 8, 8)])
def test_default_choice_of_small_grids(cuda, shape):
    """7-point grids around the smallest one on lines."""
    from xsolver_b200.api import Plan

    nx, ny, nz = shape
    i = np.arange(nx * ny * nz)
    x, y, z = i % nx, i // nx % ny, i // (nx * ny)
    r, c = [i], [i]
    for d, on in ((1, x + 1 < nx), (nx, y + 1 < ny), (nx * ny, z + 1 < nz)):
        r += [i[on], i[on] + d]
        c += [i[on] + d, i[on]]
    r, c = np.concatenate(r), np.concatenate(c)
    o = np.lexsort((c, r))
    r, c = r[o], c[o]
    v = np.where(r == c, 6.5, -np.random.default_rng(1).uniform(0.3, 1.0, r.size))
    A = CSRMatrix(i.size, np.concatenate([[0], np.cumsum(np.bincount(r))]), c, v)
    b = st.rhs_uniform(A.n, 3)
    P = Plan(A).factor("ilu0")
    s = P.schedule()
    assert (s["L"], s["U"], s["lu"]) == (("lines", "lines", "halves") if A.n >= 4096 else ("levels", "levels", "one_cta"))
    for w in _lusolve(P, b, cuda, reps=2):
        assert np.array_equal(w, oracle.lusolve(oracle.ilu0(A), b))
