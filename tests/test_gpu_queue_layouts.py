"""The task-queue layout on whole supernodes and on wide pieces, which plans
take with HYKKT_BORDERED=0."""
import numpy as np
import pytest

import helpers as H
import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("piece", [0, 512, 600, 1024])
def test_wide_pieces_on_the_queues(piece, monkeypatch):
    """Refined to the FP64 floor, a plan on the queues and the bordered one agree
    to rounding; repeated solves and shares give the same bits."""
    s = H.small_grid_system(n_bus=4000, seed=4)
    ref = hk.Plan(s)
    ref.set_accuracy(3000, 1e-12, 4, 1e-13)
    ref.solve(s)
    want = ref.solution()
    assert len(ref.symbolic("bd_col")) > 0
    monkeypatch.setenv("HYKKT_BORDERED", "0")
    p = hk.Plan(s, solve_piece=piece)
    assert len(p.symbolic("bd_col")) == 0
    width = (p.symbolic("sq_c1") - p.symbolic("sq_c0")).max()
    assert width > 1024 if piece == 0 else width <= piece
    p.set_accuracy(3000, 1e-12, 4, 1e-13)
    p.solve(s)
    sol = p.solution()
    for a, b in zip(sol, want):
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
    for share in (1, 4):
        p.set_concurrency(share)
        p.solve(s)
        assert all(np.array_equal(a, b) for a, b in zip(sol, p.solution()))
