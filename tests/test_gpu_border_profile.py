"""The profile's work of the border updates: on the variant that did it, and
all of it."""
import pytest

import helpers as H
import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_bus", [200, 460, 900, 5000])
def test_update_work_is_booked_where_it_ran(n_bus):
    s = H.small_grid_system(n_bus=n_bus, seed=5)
    p = hk.Plan(s)
    k = len(p.symbolic("bd_col"))
    assert k > 0
    assert p.solve(s) in (hk.OK, hk.CG_NOT_CONVERGED)
    prof = p.profile()
    mc = s.m_c if any(n.startswith("k_schur_cg") for n in prof) else 0
    assert (mc > 0) == (n_bus < 800)
    upd = {n: v for n, v in prof.items() if n.startswith("k_border_update")}
    panels = -(-k // 32)
    assert sum(v[0] for v in upd.values()) == panels - (0 if mc else 1)
    entries = sum(sum(i + 1 - 32 for i in range(32 * (q + 1), k)) + mc * max(0, k - 32 * (q + 1)) + mc * (mc + 1) // 2
                  for q in range(panels))
    assert all(v[2] > 0 and v[3] > 0 for v in upd.values())
    assert sum(v[2] for v in upd.values()) == pytest.approx(64.0 * entries, rel=1e-5)
    assert sum(v[3] for v in upd.values()) == pytest.approx(16.0 * entries, rel=1e-5)
