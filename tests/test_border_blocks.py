"""Blocks of the bordered layout at the sizes where their kernels' launches,
panels and warps end, and pivots that fail inside them."""
import numpy as np
import pytest

import hykkt_gb300 as hk
from hykkt_gb300 import gridgen as gg

# (columns, border rows) of each block: fronts of 1, 32, 33, 64, 65, 128, 129
# and 232 rows, blocks that touch no border row, one column of its own
BLOCKS = [(1, 0), (1, 31), (10, 0), (20, 12), (21, 12), (33, 0), (40, 24), (41, 24), (64, 64), (65, 64), (88, 41),
          (150, 82), (231, 1), (232, 0)]
BORDER = 1601


def _matrix(rng):
    """Dense blocks, each tied to border rows of its own, and a dense border."""
    at = np.cumsum([0] + [c for c, _ in BLOCKS])
    n = at[-1] + BORDER
    A = np.zeros((n, n))
    for (nt, R), a in zip(BLOCKS, at):
        G = rng.uniform(-1, 1, (nt, nt))
        A[a:a + nt, a:a + nt] = G @ G.T / nt + np.eye(nt)
        rows = at[-1] + np.sort(rng.choice(BORDER, R, replace=False))
        A[np.ix_(rows, np.arange(a, a + nt))] = rng.uniform(-0.05, 0.05, (R, nt))
    G = rng.uniform(-1, 1, (BORDER, BORDER))
    A[at[-1]:, at[-1]:] = G @ G.T / BORDER + 4 * np.eye(BORDER)
    A = np.tril(A) + np.tril(A, -1).T
    r, c = np.nonzero(np.tril(A))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    return A, at, r, rp, c.astype(np.int32)


def test_the_layout_has_these_blocks(monkeypatch):
    monkeypatch.setenv("HYKKT_BORDERED", "1")
    A, at, _, _, _ = _matrix(np.random.default_rng(2))
    n = len(A)
    r, c = np.nonzero(A)
    none = np.zeros(0)
    empty = [gg.CSR(0, m, np.zeros(1, np.int32), np.zeros(0, np.int32), none) for m in (0, n, n)]
    H = gg.coo_to_csr(n, n, r, c, A[r, c])
    sym = hk.Symbolic(gg.KKTSystem(H, *empty, np.zeros(n), none, none, none, 0.0), ordering=hk.ORDER_IDENTITY)
    assert len(sym["bd_col"]) == BORDER
    fronts = sorted(zip(np.diff(sym["bd_blk_rp"]).tolist(), np.diff(sym["bd_blk_rrp"]).tolist()))
    assert fronts == sorted(BLOCKS)


@pytest.mark.gpu
def test_factor_and_solve():
    """Backward stable solves of a matrix of condition <= 20 (as in the other
    size tests), the same bits again."""
    rng = np.random.default_rng(2)
    A, _, r, rp, c = _matrix(rng)
    n = len(A)
    ch = hk.Chol(n, rp, c, ordering=hk.ORDER_IDENTITY)
    assert ch.factor(A[r, c]) == hk.OK
    b = rng.standard_normal(n)
    want = np.linalg.solve(A, b)
    x = ch.solve(b)
    assert np.linalg.norm(x - want) <= 40 * n * np.finfo(float).eps * np.linalg.norm(want)
    assert np.array_equal(x, ch.solve(b))


@pytest.mark.gpu
def test_pivots_that_fail_inside_blocks():
    """The first, a middle and the last column of every block, and the border's
    first: a pivot that is not positive or not finite is reported; the
    handle stays usable."""
    rng = np.random.default_rng(2)
    A, at, r, rp, c = _matrix(rng)
    n = len(A)
    ch = hk.Chol(n, rp, c, ordering=hk.ORDER_IDENTITY)
    cols = {int(a + k) for (nt, _), a in zip(BLOCKS, at) for k in (0, nt // 2, nt - 1)} | {int(at[-1])}
    for col, bad in zip(sorted(cols), np.tile([-1.0, 0.0, np.nan, -np.inf, np.inf], len(cols))):
        v = A[r, c].copy()
        v[(r == col) & (c == col)] = bad
        assert ch.factor(v) == hk.NOT_SPD, (col, bad)
    assert ch.factor(A[r, c]) == hk.OK
    b = rng.standard_normal(n)
    want = np.linalg.solve(A, b)
    assert np.linalg.norm(ch.solve(b) - want) <= 40 * n * np.finfo(float).eps * np.linalg.norm(want)
