"""Which layout matrices without constraints take (no GPU)."""
import numpy as np
import pytest
import scipy.sparse as sp

import hykkt_gb300 as hk
from hykkt_gb300 import gridgen as gg


def _grid2d(k):
    T = sum(sp.eye(k, k=j) for j in (-1, 0, 1))
    return sp.kron(T, sp.eye(k)) + sp.kron(sp.eye(k), T)


def _band(n, w):
    return sum(sp.eye(n, k=j) for j in range(-w, w + 1))


@pytest.mark.parametrize("name, M, ordering, bordered", [
    # a shallow tree of small fronts: a factorization and a solve or two are
    # faster on the queues
    ("grid 28 x 28", _grid2d(28), hk.ORDER_BUILTIN, False),
    ("grid 26 x 26", _grid2d(26), hk.ORDER_BUILTIN, False),
    # small systems, deep trees, wide fronts
    ("grid 18 x 18", _grid2d(18), hk.ORDER_BUILTIN, True),
    ("grid 22 x 22 as given", _grid2d(22), hk.ORDER_IDENTITY, True),
    ("band", _band(1400, 5), hk.ORDER_BUILTIN, True),
    ("dense", sp.csr_matrix(np.ones((400, 400))), hk.ORDER_IDENTITY, True)])
def test_layout_without_constraints(name, M, ordering, bordered, monkeypatch):
    monkeypatch.setenv("HYKKT_BORDERED", "1")
    M = sp.csr_matrix(M)
    M.sort_indices()
    n = M.shape[0]
    z = np.zeros(0)
    empty = [gg.CSR(0, m, np.zeros(1, np.int32), np.zeros(0, np.int32), z) for m in (0, n, n)]
    s = gg.KKTSystem(gg.CSR(n, n, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data), *empty, np.zeros(n), z,
                     z, z, 0.0)
    assert (len(hk.Symbolic(s, ordering=ordering)["bd_col"]) > 0) == bordered
