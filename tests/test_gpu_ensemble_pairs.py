"""Members stepped two at a time (ensembles of 60,000 cells and more, at most a
third of them alone) against single runs: the packed arithmetic rounds each
half as the single operation, so the same bits; the depths differ between the
members of a pair, an odd member is alone, and a fault in one member of a pair
leaves the other's numbers as they are."""
import numpy as np
import pytest

from imodel_gb300 import swm
from imodel_gb300.swm import SWM, Ensemble

pytestmark = pytest.mark.gpu


def _state(g, seed):
    rng = np.random.default_rng(seed)
    h, u = swm.initialize_fields_tc2(g)
    return h + rng.normal(0, 5.0, g.nv), u + rng.normal(0, 0.5, g.ne)


# levels and members: two grids, one with an odd member; one grid, one tile
# size; more tiles than blocks; as 4, but below the line of 60,000 cells
@pytest.mark.parametrize("grids", [((4, 25), (3, 4)), ((5, 6),), ((6, 2), (5, 5)), ((2, 371),),
                                   ((4, 23),)])
def test_paired_members_equal_single_runs(grid_at, grids):
    gs = [grid_at(lv) for lv, _ in grids]
    ens = Ensemble(gs, [n for _, n in grids])
    states = [[_state(g, 1000 * k + j) for j in range(n)]
              for k, (g, (_, n)) in enumerate(zip(gs, grids))]
    for k, mem in enumerate(states):
        for j, (h, u) in enumerate(mem):
            ens.set_state(k, j, h, u)
    dts = [900.0 * 2.0 ** min(0, 5 - lv) for lv, _ in grids]
    steps = [4, 7][:len(grids)]
    ens.advance(dts, steps)
    for k, (g, mem) in enumerate(zip(gs, states)):
        # the grid's h_ref: its first member's mean (sequential sums)
        s = a = 0.0
        for ai, hi in zip(g.hx_areag.tolist(), mem[0][0].tolist()):
            a += ai
            s += ai * hi
        single = SWM(g, "fp32", h_ref=float(np.float32(s / a)))
        for j in sorted({0, 1, len(mem) // 2, len(mem) - 2, len(mem) - 1}):
            hs, us = single.ode_rk4(*mem[j], dts[k], steps[k])
            he, ue = ens.get_state(k, j)
            assert np.array_equal(he, hs) and np.array_equal(ue, us), (k, j)
        single.close()
    ens.close()


def test_a_fault_in_one_member_of_a_pair(grid_at):
    g = grid_at(5)
    ens = Ensemble([g], [6])
    states = [_state(g, j) for j in range(6)]
    for j, (h, u) in enumerate(states):
        ens.set_state(0, j, h, u)
    h, u = states[3]
    u = u.copy()
    u[11] = np.inf
    ens.set_state(0, 3, h, u)
    ens.advance([900.0], [1])
    with pytest.raises(swm.SWMError) as ei:
        ens.get_state(0, 3)
    assert ei.value.code == 3
    good = ens.get_state(0, 2)
    ens.set_state(0, 2, *states[2])
    ens.set_state(0, 3, *states[3])
    ens.advance([900.0], [1])
    again = ens.get_state(0, 2)
    assert np.array_equal(good[0], again[0]) and np.array_equal(good[1], again[1])
    ens.close()
