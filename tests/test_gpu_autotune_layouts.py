"""The autotuner's candidates are different layouts, and its choice is the
layout that the plan then has, also from the cache file."""
import numpy as np
import pytest

import helpers as H
import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu


def _plan(s):
    p = hk.Plan(s)
    p.set_accuracy(2000, 1e-11, 3, 1e-9)
    return p


def _bordered(p):
    return len(p.symbolic("bd_col")) > 0


@pytest.mark.parametrize("share", [1, 3])
def test_candidates_are_distinct_layouts(tmp_path, share):
    s = H.small_grid_system(n_bus=500, seed=3)
    cache = str(tmp_path / "tune.txt")
    p = _plan(s)
    t = p.autotune(s, share=share, cache=cache)
    kinds = [(c["solve_piece"], c["warp_subtree"], c["chunk_fma"]) for c in t["timed"]]
    assert len(set(kinds)) == len(kinds)
    assert kinds[0] == (0, 0, 0)  # the bordered layout
    assert (0, 16, 4096) in kinds and all(k[2] > 0 for k in kinds[1:])  # the task queues
    assert all(c["solves_per_s"] > 0 for c in t["timed"])
    assert _bordered(p) == (t["chunk_fma"] == 0)
    # the same choice from the file, for a plan that was made as either layout
    for piece in (0, 256):
        q = hk.Plan(s, solve_piece=piece)
        u = q.autotune(s, share=share, cache=cache)
        assert u["from_cache"] and u["chunk_fma"] == t["chunk_fma"]
        assert _bordered(q) == _bordered(p)


def test_cached_layouts(tmp_path, monkeypatch):
    """Entries that name the queues give them; entries without a layout give what
    a plan of that piece takes."""
    s = H.small_grid_system(n_bus=500, seed=3)
    cache = tmp_path / "tune.txt"
    p = _plan(s)
    p.autotune(s, share=1, cache=str(cache))
    f = cache.read_text().split()
    assert p.solve(s) == hk.OK
    x = p.solution()
    for words, bordered in ((["0", "16", "4096", "9.9", "queues"], False), (["0", "16", "4096", "9.9"], True),
                            (["256", "0", "4096", "9.9"], False), (["0", "16", "4096", "9.9", "bordered"], True)):
        cache.write_text(" ".join(f[:2] + words) + "\n")
        q = _plan(s)
        t = q.autotune(s, share=1, cache=str(cache))
        assert t["from_cache"] and _bordered(q) == bordered, words
        assert q.solve(s) == hk.OK
        for a, b in zip(q.solution(), x):
            assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
    monkeypatch.setenv("HYKKT_BORDERED", "0")
    q = _plan(s)
    t = q.autotune(s, share=1)
    assert not _bordered(q) and all(c["chunk_fma"] > 0 for c in t["timed"])
