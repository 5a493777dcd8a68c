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
