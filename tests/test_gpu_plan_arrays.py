"""The arrays of a plan's analysis, whatever the layout its solves take."""
import numpy as np
import pytest

import helpers as H
import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu

ARRAYS = ["etree", "colcount", "hg_rp", "lp_row", "L_ri", "sn_first", "sn_parent", "sn_nrows", "sn_rows", "sn_rp",
          "sn_children", "sq_sn", "sq_c0", "sq_c1", "sq_level", "tf_kind", "tb_item", "bd_need", "unit_cols"]


@pytest.mark.parametrize("n_bus", [60, 700])
@pytest.mark.parametrize("piece", [0, 1024, 256])
def test_plan_arrays_of_every_layout(n_bus, piece):
    """Plans with and without the bordered layout answer as the host analysis
    does for their ordering; another request gives the same."""
    s = H.small_grid_system(n_bus=n_bus, seed=3)
    p = hk.Plan(s, solve_piece=piece)
    assert (len(p.symbolic("bd_col")) > 0) == (piece != 256)
    sym = hk.Symbolic(s, perm=p.perm(), solve_piece=piece)
    assert np.array_equal(sym["perm"], p.perm())
    for _ in range(2):
        for what in ARRAYS:
            assert np.array_equal(p.symbolic(what), sym[what]), what
    with pytest.raises(KeyError):
        p.symbolic("no_such_array")
