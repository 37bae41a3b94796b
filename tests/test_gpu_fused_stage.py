"""The fused FP32 stage (variant 1 without options: one kernel per RK stage
over tiles) against the separate triangle, cell and edge kernels (variant 2):
the same arithmetic, so the same bits, from one tile on the whole sphere to
tiles cut off by the end of a curve segment."""
import numpy as np
import pytest

from imodel_gb300 import swm
from imodel_gb300.swm import SWM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [0, 1, 2, 3, 4, 6, 7])
def test_fused_stage_equals_the_separate_kernels(grid_at, level):
    g = grid_at(level)
    rng = np.random.default_rng(level)
    h, u = swm.initialize_fields_tc2(g)
    h = h + rng.normal(0, 5.0, g.nv)
    u = u + rng.normal(0, 0.5, g.ne)
    bt = 50.0 * (1.0 + g.v_p[:, 0])
    dt = 900.0 * 2.0 ** min(0, 5 - level)
    out = []
    for v in (1, 2):
        m = SWM(g, "fp32", bt=bt, h_ref=2900.0)
        m.set_tuning(variant=v)
        assert m.launch_count(1) == (4 if v == 1 else 12)
        out.append(m.tendency(h, u) + m.ode_rk4(h, u, dt, 5))
        # pole to pole the options take the separate kernels, then go back
        m.set_apvm(0.5, dt)
        assert m.launch_count(1) == 20
        m.set_apvm(0.0, dt)
        out[-1] += m.ode_rk4(h, u, dt, 1)
        m.close()
    for a, b in zip(*out):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


def test_fused_stage_reports_a_vanishing_depth(grid_at):
    """The PV division's guard and the NaN scan raise the same statuses."""
    g = grid_at(3)
    m = SWM(g, "fp32", h_ref=1.0)
    m.set_tuning(variant=1)
    with pytest.raises(swm.SWMError) as ei:
        m.tendency(np.zeros(g.nv), np.zeros(g.ne))
    assert ei.value.code == 4
    h, u = swm.initialize_fields_tc2(g)
    u[3] = np.nan
    with pytest.raises(swm.SWMError) as ei:
        m.ode_rk4(h, u, 600.0, 1)
    assert ei.value.code == 3
    m.close()


@pytest.mark.parametrize("advection", ["trsk", "upw1"])
@pytest.mark.parametrize("level,case", [(2, 2), (4, 3), (6, 2), (7, 3)])
def test_fused_moist_stage_close_to_fp64(grid_at, level, case, advection):
    """The fused FP32 moist stage at each tile size against the FP64 handle.
    Four steps are sixteen evaluations of a few hundred FP32 roundings (6e-8
    each), so 1e-5 of each field's norm bounds them; the cloud and rain water
    begin at zero and are measured against the vapour they come from."""
    from imodel_gb300.moist import FIELDS, Moist, moist_fields
    g = grid_at(level)
    f = moist_fields(g, case)
    dt = min(900.0, 110.0 * 2.0 ** (8 - level))
    out = []
    for prec in ("fp64", "fp32"):
        m = Moist(g, case, f, advection=advection, precision=prec)
        m.set_state(f)
        m.advance(dt, 4)
        out.append(m.get_state())
        m.close()
    norm = {k: np.linalg.norm(out[0][k]) for k in FIELDS}
    norm["hqc"] = norm["hqr"] = norm["hqv"]
    for k in FIELDS:
        assert np.linalg.norm(out[1][k] - out[0][k]) <= 1e-5 * norm[k], k
