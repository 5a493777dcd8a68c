"""The Cholesky component's own inputs: its entry map and the caller's array."""
import numpy as np
import pytest

import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu


def _lower(n, rng):
    """A dense SPD matrix and its lower triangle as a CSR list of entries."""
    G = rng.uniform(-1, 1, (n, n))
    A = G @ G.T / n + np.eye(n)
    A = np.tril(A) + np.tril(A, -1).T
    r, c = np.nonzero(np.tril(A))
    return A, np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32), c.astype(np.int32), r


@pytest.mark.parametrize("n", [3, 200, 700])
def test_first_factor_reads_the_whole_entry_map(n):
    """A factorization right after the handle's creation takes every value from
    its place (cond <= 5: the error of a backward stable solve is far below the
    1e-12 asked for)."""
    rng = np.random.default_rng(n)
    A, rp, ci, r = _lower(n, rng)
    b = rng.standard_normal(n)
    want = np.linalg.solve(A, b)
    for _ in range(8):
        ch = hk.Chol(n, rp, ci)
        assert ch.factor(A[r, ci]) == hk.OK
        assert np.linalg.norm(ch.solve(b) - want) <= 1e-12 * np.linalg.norm(want)
        ch.close()


@pytest.mark.parametrize("n", [33, 400])
def test_unaligned_values(n):
    """A view into a byte buffer, whatever its offset, gives the same bits as an
    aligned array."""
    rng = np.random.default_rng(n)
    A, rp, ci, r = _lower(n, rng)
    v = np.ascontiguousarray(A[r, ci])
    b = rng.standard_normal(n)
    ch = hk.Chol(n, rp, ci)
    assert ch.factor(v) == hk.OK
    x = ch.solve(b)
    for off in (1, 4, 7, 8):
        buf = np.zeros(v.nbytes + 16, np.uint8)
        at = (off - buf.ctypes.data) % 8 + (8 if off == 8 else 0)
        u = buf[at:at + v.nbytes].view(np.float64)
        assert u.ctypes.data % 8 == off % 8
        u[:] = v
        assert ch.factor(u) == hk.OK
        assert np.array_equal(ch.solve(b), x)


def test_missing_values_are_refused():
    rng = np.random.default_rng(1)
    A, rp, ci, r = _lower(50, rng)
    ch = hk.Chol(50, rp, ci)
    assert hk.lib().hykkt_chol_factor(ch.h, None) == hk.INVALID
    with pytest.raises(hk.HykktError):
        ch.factor(A[r, ci][:-1])
    assert ch.factor(A[r, ci]) == hk.OK
