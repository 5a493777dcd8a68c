"""Several plans of the bordered layout in flight at the default share: each of
their launches asks for the whole GPU, so most CTAs of a launch start while
other CTAs of it are already at work, or have ended its CG loop."""
import numpy as np
import pytest

import helpers as H
import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu

# buses, seed: Schur plans (to about 600 buses), plans with blocks and plans
# that are all border, with CG runs of different lengths
SIZES = [(40, 1), (230, 2), (330, 3), (460, 4), (700, 5), (1000, 6), (1500, 7), (2500, 8)]


@pytest.mark.parametrize("rtol", [1e-3, 1e-11])
def test_plans_in_flight_at_default_share(rtol):
    """Short CG runs (many loops that end) and long ones: every solution is the
    lone solve's, bit for bit, with as many iterations."""
    systems = [H.small_grid_system(n_bus=n, seed=seed) for n, seed in SIZES]
    plans = [hk.Plan(s) for s in systems]
    assert all(len(p.symbolic("bd_col")) > 0 for p in plans)
    alone = []
    for p, s in zip(plans, systems):
        p.set_accuracy(3000, rtol, 3, 1e-9)
        st = p.solve(s)
        assert st in (hk.OK, hk.ACCURACY_NOT_MET)
        alone.append((st, p.info()["cg_iterations_total"], p.solution()))
    for _ in range(12):
        for p, s in zip(plans, systems):
            p.solve(s, sync=False)
        for p, (st, its, sol) in zip(plans, alone):
            assert p.wait() == st
            assert p.info()["cg_iterations_total"] == its
            assert all(np.array_equal(a, b) for a, b in zip(sol, p.solution()))


@pytest.mark.parametrize("n_bus", [60, 460, 900])
def test_cg_hand_over_beside_factorizations(n_bus):
    """The CTA that takes an iteration's last step, held up by another plan's
    factorizations, hands its state to the next one's last step: the iterates
    stay those of the lone run at every share of the GPU."""
    s = H.small_grid_system(n_bus=n_bus, seed=9, dx=(1e-8, 1e4), ds=(1e-8, 1e8))
    big = H.small_grid_system(n_bus=3000, seed=10)
    p, q = hk.Plan(s), hk.Plan(big)
    p.set_accuracy(2000, 1e-11, 0, 1e-10)
    q.set_accuracy(1, 1e-1, 0, 1e-10)
    st = p.solve(s)
    its, sol = p.info()["cg_iterations_total"], p.solution()
    for share in (1, 3, 40):
        p.set_concurrency(share)
        for _ in range(4):
            q.solve(big, sync=False)
            assert p.solve(s) == st
            assert p.info()["cg_iterations_total"] == its
            assert all(np.array_equal(a, b) for a, b in zip(sol, p.solution()))
            q.wait()
