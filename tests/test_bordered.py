"""The bordered layout (bordered.cuh): its lists on the CPU, its factor and
solves on the GPU at the sizes where tiles, panels and blocks end."""
import numpy as np
import pytest

import helpers as H
import hykkt_gb300 as hk

CASES = ["grid150", "grid1500", "grid400_identity", "a200_AC_10", "a2000_AC_09"]


def _system(case):
    if case == "grid400_identity":
        return H.small_grid_system(n_bus=60, seed=2), hk.ORDER_IDENTITY
    if case.startswith("grid"):
        return H.small_grid_system(n_bus=int(case[4:]), seed=3), hk.ORDER_BUILTIN
    return H.load_system(case), hk.ORDER_BUILTIN


@pytest.mark.parametrize("case", CASES)
def test_bordered_lists(case, monkeypatch):
    """Block fronts, border assembly and update lists, walked with numpy, solve
    a random SPD matrix on the permuted pattern as a dense solve does."""
    monkeypatch.setenv("HYKKT_BORDERED", "1")
    s, ordering = _system(case)
    sym = hk.Symbolic(s, ordering=ordering)
    n = s.n_x
    bcol = sym["bd_col"]
    k = len(bcol)
    assert k > 0
    cp, row = sym["lp_cp"], sym["lp_row"]
    rng = np.random.default_rng(0)
    col = np.repeat(np.arange(n), np.diff(cp))
    val = rng.uniform(-1, 1, len(row))
    A = np.zeros((n, n))
    A[row, col] = val
    A[col, row] = val
    A[np.arange(n), np.arange(n)] = np.abs(A).sum(axis=1) + 1.0
    val = A[row, col]
    rp, cols, rrp, rows = (sym["bd_blk_" + w] for w in ("rp", "col", "rrp", "row"))
    ent_rp, ent_q, ent_pos = (sym["bd_ent_" + w] for w in ("rp", "q", "pos"))
    assert np.array_equal(np.sort(np.concatenate([bcol, cols])), np.arange(n))
    size = np.diff(rp) + np.diff(rrp)
    assert np.all(np.diff(size) <= 0) and (len(size) == 0 or size[0] <= 232)
    upd, E, X, b = [], [], [], rng.standard_normal(n)
    for i in range(len(size)):
        nt, N = rp[i + 1] - rp[i], size[i]
        F = np.zeros((N, N))
        r, c = np.tril_indices(N)
        flat = np.zeros(len(r))
        e = slice(ent_rp[i], ent_rp[i + 1])
        assert len(set(ent_pos[e].tolist())) == ent_rp[i + 1] - ent_rp[i]
        flat[ent_pos[e]] = val[ent_q[e]]
        F[r, c] = flat
        F = F + np.tril(F, -1).T
        X.append(np.linalg.inv(np.linalg.cholesky(F[:nt, :nt])))
        E.append(F[nt:, :nt] @ X[i].T @ X[i])
        up = -E[i] @ F[:nt, nt:]
        upd.append(up[np.tril_indices(N - nt)])
    upd = np.concatenate(upd) if upd else np.zeros(0)
    ar, ac, src, arp, apos = (sym["bd_asm_" + w] for w in ("row", "col", "src", "rp", "pos"))
    assert np.array_equal(np.sort(apos), np.arange(len(upd)))  # every update once
    S = np.zeros((k, k))
    for t in range(len(ar)):
        assert S[ar[t], ac[t]] == 0 and ar[t] >= ac[t]
        S[ar[t], ac[t]] = (val[src[t]] if src[t] >= 0 else 0.0) + upd[apos[arp[t]:arp[t + 1]]].sum()
    used = np.concatenate([ent_q, src[src >= 0]])
    assert np.array_equal(np.sort(used), np.arange(len(row)))  # every entry once
    S = S + np.tril(S, -1).T
    u = np.concatenate([E[i] @ b[cols[rp[i]:rp[i + 1]]] for i in range(len(size))]) if len(size) else np.zeros(0)
    ug_rp, ug_pos = sym["bd_ug_rp"], sym["bd_ug_pos"]
    assert np.array_equal(rows[ug_pos], np.repeat(np.arange(k), np.diff(ug_rp)))
    bs = b[bcol] - np.array([u[ug_pos[ug_rp[j]:ug_rp[j + 1]]].sum() for j in range(k)])
    x = np.zeros(n)
    x[bcol] = np.linalg.solve(S, bs)
    for i in range(len(size)):
        c = cols[rp[i]:rp[i + 1]]
        x[c] = X[i].T @ (X[i] @ b[c]) - E[i].T @ x[bcol[rows[rrp[i]:rrp[i + 1]]]]
    assert np.allclose(x, np.linalg.solve(A, b), rtol=1e-10, atol=1e-12)


def _spd(shape, rng):
    """A dense matrix of n columns, or nb blocks of bs columns tied to a border."""
    if isinstance(shape, int):
        G = rng.uniform(-1, 1, (shape, shape))
        return G @ G.T / shape + 0.5 * np.eye(shape)
    nb, bs, border = shape
    n = nb * bs + border
    A = np.zeros((n, n))
    for k in range(nb):
        sl = slice(k * bs, (k + 1) * bs)
        G = rng.uniform(-1, 1, (bs, bs))
        A[sl, sl] = G @ G.T / bs + np.eye(bs)
        touch = rng.choice(border, min(border, 40), replace=False) + nb * bs
        A[np.ix_(touch, np.arange(sl.start, sl.stop))] = rng.uniform(-0.05, 0.05, (len(touch), bs))
    G = rng.uniform(-1, 1, (border, border))
    A[nb * bs:, nb * bs:] = G @ G.T / border + 4 * np.eye(border)
    return np.tril(A) + np.tril(A, -1).T


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 1535, 1537, 2047,
                                   2049, (3, 7, 40), (30, 20, 300), (9, 25, 700), (12, 90, 260), (70, 33, 1600)])
@pytest.mark.parametrize("scale", [1.0, 1e-140, 1e140])
def test_cholesky_sizes(shape, scale):
    """Factor and solve against numpy: the error of a backward stable solve is
    at most a small multiple of n eps cond(A) (cond <= 20 here); rows and
    columns scaled by powers of two apart change nothing but the exponents.
    The same factor and right-hand side give the same bits."""
    rng = np.random.default_rng(11)
    A = _spd(shape, rng)
    n = len(A)
    d = 2.0 ** rng.integers(-8, 9, n)
    A = A * d[:, None] * d[None, :] * scale
    r, c = np.nonzero(np.tril(A))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    ch = hk.Chol(n, rp, c.astype(np.int32))
    b = rng.standard_normal(n)
    if scale < 1e-100:
        # pivots below the reference's absolute tolerance (1e-12) are reported
        assert ch.factor(A[r, c]) == hk.NOT_SPD
        return
    assert ch.factor(A[r, c]) == hk.OK
    x = ch.solve(b * d * scale) * d
    want = np.linalg.solve(A / scale / d[:, None] / d[None, :], b)
    bound = 40 * n * np.finfo(float).eps
    assert np.linalg.norm(x - want) <= max(bound, 1e-14) * np.linalg.norm(want)
    assert np.array_equal(x, ch.solve(b * d * scale) * d)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [65, 257, 700])
@pytest.mark.parametrize("scale", [2.0 ** 300, 2.0 ** 964])
def test_cholesky_near_overflow(n, scale):
    """The update's sums are rounded with integers, beyond 2^900 by FP64: a
    power of two through the matrix changes no bit of the solution."""
    rng = np.random.default_rng(12)
    A = _spd(n, rng)
    r, c = np.nonzero(np.tril(A))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    ch = hk.Chol(n, rp, c.astype(np.int32))
    b = rng.standard_normal(n)
    assert ch.factor(A[r, c]) == hk.OK
    x = ch.solve(b)
    assert ch.factor(A[r, c] * scale) == hk.OK
    assert np.array_equal(ch.solve(b * 2.0 ** 20) * (scale / 2.0 ** 20), x)


@pytest.mark.gpu
def test_not_finite_and_not_spd_are_reported():
    rng = np.random.default_rng(5)
    for shape in (200, (30, 20, 300)):
        A = _spd(shape, rng)
        r, c = np.nonzero(np.tril(A))
        n = len(A)
        rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
        ch = hk.Chol(n, rp, c.astype(np.int32))
        for at, bad in ((0, -1.0), (n // 2, 0.0), (n - 1, -3.0), (n // 3, np.nan), (n - 1, np.inf)):
            v = A[r, c].copy()
            v[(r == at) & (c == at)] = bad
            assert ch.factor(v) == hk.NOT_SPD
        assert ch.factor(A[r, c]) == hk.OK  # the handle stays usable


@pytest.mark.gpu
@pytest.mark.parametrize("n_bus", [40, 700, 2500])
def test_bordered_matches_task_queues(n_bus, monkeypatch):
    """The same system through both layouts: refined to the FP64 floor of the
    solution, so the two agree to rounding; repeated solves are bit-identical."""
    s = H.small_grid_system(n_bus=n_bus, seed=4)
    sols = []
    for v in ("0", "1"):
        monkeypatch.setenv("HYKKT_BORDERED", v)
        p = hk.Plan(s)
        assert (len(p.symbolic("bd_col")) > 0) == (v == "1")
        p.set_accuracy(3000, 1e-12, 4, 1e-13)
        p.solve(s)
        sols.append(p.solution())
        p.solve(s)
        assert all(np.array_equal(a, b) for a, b in zip(sols[-1], p.solution()))
        p.set_concurrency(8)
        p.solve(s)
        assert all(np.array_equal(a, b) for a, b in zip(sols[-1], p.solution()))
    for a, b in zip(*sols):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(a)


@pytest.mark.gpu
@pytest.mark.parametrize("n_bus", [6, 16, 320, 321, 460])
@pytest.mark.parametrize("start", [False, True])
def test_schur_plan_matches_task_queues(n_bus, start, monkeypatch):
    """Small systems form S itself (four rows a task up to 640 constraints,
    eight above): the same solution as the task queues, from a zero and from a
    given start vector, as many CG iterations up to a few of rounding."""
    s = H.small_grid_system(n_bus=n_bus, seed=6)
    y0 = np.random.default_rng(1).uniform(-1, 1, s.m_c) if start else None
    sols, its = [], []
    for v in ("0", "1"):
        monkeypatch.setenv("HYKKT_BORDERED", v)
        p = hk.Plan(s)
        p.set_accuracy(2000, 1e-11, 0, 1e-10)
        assert p.solve(s, y0=y0) == hk.OK
        its.append(p.info()["cg_iterations"])
        p.set_accuracy(2000, 1e-12, 4, 1e-13)
        p.solve(s, y0=y0)
        sols.append(p.solution())
    assert abs(its[0] - its[1]) <= 2
    for a, b in zip(*sols):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(a)


@pytest.mark.gpu
def test_wide_border_on_shares_of_the_gpu():
    """A border wide enough for product panels of eight rows: tasks of one bin
    and of several, the same bits from each, refined to the residual target."""
    s = H.small_grid_system(n_bus=10000, seed=4)
    p = hk.Plan(s)
    assert len(p.symbolic("bd_col")) > 6600
    p.set_accuracy(3000, 1e-11, 4, 1e-11)
    sols = []
    for share in (1, 3, 40):
        p.set_concurrency(share)
        assert p.solve(s) == hk.OK
        sols.append(p.solution())
    for other in sols[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(sols[0], other))
