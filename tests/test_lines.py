"""Line schedule of the exact triangular solves (host analysis, no GPU).

The line schedule replaces row-per-thread dependency flags
(hip/Precond/gpuparilu.cpp:257-364) on stencil patterns.  Every index the
kernel uses follows from a few integers: the step of a row, its ring slot,
the ring slot of each dependency, the exchange slot a halo value is read
from.  These tests run the schedule with exactly that arithmetic, patch by
patch in ticket order, and require that every dependency is found where the
kernel looks for it and that the solution equals the oracle's LUsolve bit
for bit (the sums keep its order and operations)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from xsolver_b200 import CSRMatrix
from xsolver_b200 import stencils as st

_ip = C.POINTER(C.c_int)
NAMES = ("fits nx ny nz c al be L ty tz ry rz py npad npy npz npatch nsteps D E nh maxd").split()


def lines(n, rp, ci, upper):
    from xsolver_b200 import _lib

    info = np.zeros(24, np.int32)
    t = dict(delta=np.zeros(32, np.int32), shift=np.zeros(32, np.int32), offq=np.zeros(32, np.int32),
             patch=np.zeros(2 * n + 2, np.int32), rank_of=np.zeros(4 * n + 64, np.int32), halo=np.zeros(256, np.int32),
             exp_of=np.zeros(128, np.int32))
    p = lambda a: np.ascontiguousarray(a).ctypes.data_as(_ip)  # noqa: E731
    rp, ci = np.ascontiguousarray(rp, np.int32), np.ascontiguousarray(ci, np.int32)
    assert _lib.lib().xs_tri_lines(n, p(rp), p(ci), int(upper), p(info), *(p(v) for v in t.values())) == 0
    if not info[0]:
        return None
    g = dict(zip(NAMES, map(int, info)), **t)
    return g


def solve(n, rp, ci, v, rhs, dinv, upper, g):
    """The kernel's schedule, sequentially, with a NaN for every value that
    is not there yet.  A ring of 64 steps; a slot keeps (step, value)."""
    RL = 64
    L, ty, nst, E = g["L"], g["ty"], g["nsteps"], g["E"]
    assert nst % 8 == 0 and g["maxd"] <= 32 and g["nh"] <= 64 and L <= 128 and g["D"] <= 32

    def q0(pY, pZ, Yl, Zl):
        Z = pZ * g["tz"] + Zl
        y = pY * ty + Yl - g["c"] * Z
        return -1 if Z < 0 or Z >= g["nz"] or y < 0 or y >= g["ny"] else (Z * g["ny"] + y) * g["nx"]

    xb = np.full((g["npatch"], nst * E), np.nan)
    out = np.full(n, np.nan)
    for rank in range(g["npatch"]):
        pY, pZ = (int(w) for w in g["patch"][2 * rank:2 * rank + 2])
        ring = np.full((RL, g["npad"]), np.nan)
        own = [(q0(pY, pZ, l % ty, l // ty), g["al"] * (l % ty) + g["be"] * (l // ty),
                (l // ty + g["rz"]) * g["py"] + l % ty + g["ry"], int(g["exp_of"][l])) for l in range(L)]
        halo = []
        for h in range(g["nh"]):
            Yl, Zl = int(g["halo"][2 * h]), int(g["halo"][2 * h + 1])
            if q0(pY, pZ, Yl, Zl) < 0:
                continue
            dY, dZ = -(Yl < 0), -(Zl < 0)
            Yo, Zo = Yl - dY * ty, Zl - dZ * g["tz"]
            ro = int(g["rank_of"][(pZ + dZ) * g["npy"] + pY + dY])
            assert 0 <= ro < rank  # taken by an earlier ticket
            eo = int(g["exp_of"][Zo * ty + Yo])
            assert eo >= 0
            oh = g["al"] * Yl + g["be"] * Zl
            halo.append((ro, eo, oh, g["al"] * Yo + g["be"] * Zo - oh, (Zl + g["rz"]) * g["py"] + Yl + g["ry"]))
        for t in range(-g["maxd"], nst):
            for ro, eo, oh, d, col in halo:  # the pollers' values of step t
                if oh <= t < oh + g["nx"]:
                    assert 0 <= t + d < nst
                    ring[t % RL, col] = xb[ro, (t + d) * E + eo]
            if t < 0:
                continue
            new = []
            for q, off, pad, e in own:
                x = t - off
                if q < 0 or not 0 <= x < g["nx"]:
                    continue
                r = n - 1 - (q + x) if upper else q + x
                acc = rhs[r] * dinv[r] if upper else rhs[r]
                es = range(rp[r], rp[r + 1]) if not upper else range(rp[r + 1] - 1, rp[r] - 1, -1)
                k = -1
                for en in es:
                    o = r - ci[en] if upper else ci[en] - r
                    kk = [j for j in range(g["D"]) if g["offq"][j] == o]
                    assert len(kk) == 1 and kk[0] > k  # diagonals in the order of the sum
                    k = kk[0]
                    dl = int(g["delta"][k])
                    assert 1 <= dl <= g["maxd"] and 0 <= pad - int(g["shift"][k]) < g["npad"]
                    y = ring[(t - dl) % RL, pad - int(g["shift"][k])]
                    assert not np.isnan(y)
                    acc = acc - y * v[en]
                new.append((pad, acc, e, r))
            for pad, acc, e, r in new:
                assert np.isnan(out[r])
                ring[t % RL, pad] = out[r] = acc
                if e >= 0:
                    xb[rank, t * E + e] = acc
            if t - g["maxd"] >= 0:  # no step reads further back
                ring[(t - g["maxd"]) % RL, :] = np.nan
    return out


def _stencil(shape, offs, seed=0):
    """Diagonally dominant matrix with the given offsets (z, y, x) on an nz x ny x nx grid."""
    offs = sorted(offs)
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    coef = -rng.uniform(0.5, 1.5, (n, len(offs)))
    coef[:, offs.index((0,) * len(shape))] = 2.0 * len(offs)
    n, rp, ci, v = st._assemble(shape, offs, coef)
    return CSRMatrix(n, rp, ci, v)


P7 = [(0, 0, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0)]
P27 = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
P5 = [(0, 0), (0, 1), (0, -1), (1, 0), (-1, 0)]
P9 = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]


def _check(n, F, upper):
    rp, ci, v = (F.urp, F.uci, F.uv) if upper else (F.lrp, F.lci, F.lv)
    g = lines(n, rp, ci, upper)
    assert g is not None
    rhs = np.random.default_rng(3).uniform(-1, 1, n)
    x = solve(n, rp, ci, v, rhs, F.dinv, upper, g)
    ref = np.zeros(n)
    for q in range(n):
        r = n - 1 - q if upper else q
        acc = rhs[r] * F.dinv[r] if upper else rhs[r]
        for e in (range(rp[r + 1] - 1, rp[r] - 1, -1) if upper else range(rp[r], rp[r + 1])):
            acc = acc - ref[ci[e]] * v[e]
        ref[r] = acc
    assert np.array_equal(x, ref)
    return g


@pytest.mark.parametrize("shape,offs", [((9, 11, 10), P7), ((6, 20, 17), P7), ((34, 7, 8), P7), ((12, 13, 14), P27),
                                        ((11, 30, 12), P27), ((40, 37), P5), ((7, 150), P5), ((150, 8), P9),
                                        ((11, 12, 13), [o for o in P27 if sum(map(abs, o)) <= 2])])
def test_schedule_solves_ilu0_factors(shape, offs):
    A = _stencil(shape, offs)
    F = oracle.ilu0(A)
    for upper in (False, True):
        _check(A.n, F, upper)


def test_schedule_solves_parilut_fill():
    A = st.convdiff3d_27pt(24)
    F = oracle.parilut(A, fill=2.0, sweeps=5, droptol=1e-4)
    for upper in (False, True):
        _check(A.n, F, upper)


def test_one_sided_and_absent_diagonals():
    """Triangles whose rows miss entries that their diagonal has elsewhere, and one-directional couplings."""
    A = _stencil((12, 13, 14), P7, 4)
    rows = np.repeat(np.arange(A.n), np.diff(A.rowptr))
    keep = (A.colidx == rows) | (np.random.default_rng(1).random(A.nnz) < 0.95)
    rp = np.zeros(A.n + 1, np.int64)
    np.cumsum(np.bincount(rows[keep], minlength=A.n), out=rp[1:])
    B = CSRMatrix(A.n, rp, A.colidx[keep], A.val[keep])
    F = oracle.ilu0(B)
    for upper in (False, True):
        _check(A.n, F, upper)


def test_patterns_that_do_not_qualify():
    """No grid behind the pattern, too many diagonals, or mostly padding: the other schedules keep them."""
    rng = np.random.default_rng(0)
    n = 900
    rp, ci = [0], []
    for r in range(n):
        c = np.unique(rng.integers(0, max(r, 1), 3)) if r else np.array([], int)
        ci += list(c[c < r])
        rp.append(len(ci))
    assert lines(n, np.array(rp), np.array(ci), False) is None
    F = oracle.ilu0(_stencil((10, 10, 10), P7))
    rp, ci = F.lrp, F.lci
    keep = rng.random(len(ci)) < 0.5  # under 80 percent of the diagonals' slots
    rows = np.repeat(np.arange(1000), np.diff(rp))
    rp2 = np.zeros(1001, np.int64)
    np.cumsum(np.bincount(rows[keep], minlength=1000), out=rp2[1:])
    assert lines(1000, rp2, ci[keep], False) is None


def test_equal_slots_of_different_stencils():
    """A 5-point and a 7-point schedule of as many slots, whose value streams
    (slots times diagonals) are of different sizes: what a handle keeps for
    one pattern cannot be told by the slot count to fit the other."""
    sizes = []
    for shape, offs in (((96, 96), P5), ((16, 25, 25), P7), ((80, 80), P5), ((25, 16, 16), P7)):
        A = _stencil(shape, offs)
        low = A.colidx < np.repeat(np.arange(A.n), np.diff(A.rowptr))
        rp = np.concatenate([[0], np.cumsum(low)])[A.rowptr]
        g = lines(A.n, rp, A.colidx[low], False)
        sizes.append((g["npatch"] * g["nsteps"] * g["L"], g["D"]))
    for (sa, da), (sb, db) in (sizes[:2], sizes[2:]):
        assert sa == sb and (da, db) == (2, 3)
