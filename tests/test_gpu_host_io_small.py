"""Host arrays on both sides of the size up to which a state passes through the
handle's page-locked area (levels 2 and 5; level 6 goes through pageable
copies): every call that shares the area, one after the other, gives what the
same calls give on their own, in place too."""
import numpy as np
import pytest

from imodel_gb300 import _capi, swm
from imodel_gb300.swm import SWM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("level", [2, 5, 6])
def test_calls_that_share_the_area(grid_at, precision, level):
    g = grid_at(level)
    h, u = swm.initialize_fields_tc2(g)
    rng = np.random.default_rng(level)
    h2, u2 = h + rng.normal(0, 5.0, g.nv), u + rng.normal(0, 0.5, g.ne)
    dt = 200.0
    kw = {} if precision == "fp64" else {"h_ref": 2900.0}
    a = SWM(g, precision, **kw)
    t2 = a.tendency(h2, u2)
    t1 = a.tendency(h, u)
    s1 = a.ode_rk4(h, u, dt, 2)
    b = SWM(g, precision, **kw)
    b.set_state(h2, u2)
    b.set_state(h, u)
    # a tendency of another state leaves the handle's state alone
    for x, y in zip(b.tendency(h2, u2), t2):
        assert np.array_equal(x, y)
    b.advance(dt, 1)
    b.advance(dt, 1)
    for x, y in zip(b.get_state(), s1):
        assert np.array_equal(x, y)
    # in place: the outputs are the inputs' arrays
    hi, ui = h.copy(), u.copy()
    p = _capi.as_f64p
    assert b.lib.imodel_swm_tendency(b.handle, p(hi), p(ui), p(hi), p(ui)) == 0
    assert np.array_equal(hi, t1[0]) and np.array_equal(ui, t1[1])
    # a NaN is reported and written back all the same, and is gone afterwards
    bad = h.copy()
    bad[1] = np.nan
    b.set_state(bad, u)
    ho, uo = np.zeros(g.nv), np.zeros(g.ne)
    assert b.lib.imodel_swm_get_state(b.handle, p(ho), p(uo)) == 3
    assert np.isnan(ho[1]) and np.array_equal(uo, _stored(u, precision))
    b.set_state(h, u)
    ho, uo = b.get_state()
    assert np.array_equal(uo, _stored(u, precision))
    a.close()
    b.close()


def _stored(u, precision):
    return u if precision == "fp64" else u.astype(np.float32).astype(np.float64)
