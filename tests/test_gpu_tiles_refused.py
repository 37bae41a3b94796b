"""Handles that get no memory for the fused stage's tiles step with the separate
kernels, which need none: the same bits, and for the moist model the same up
to rounding."""
import numpy as np
import pytest

from imodel_gb300 import _capi, swm
from imodel_gb300.swm import SWM

pytestmark = pytest.mark.gpu


def without_tiles(make, has_tiles):
    """The handle that make() gives when one device allocation fails and the
    create succeeds all the same: that allocation was the tiles'."""
    lib = _capi.swm_lib()
    for after in range(1, 200):
        assert lib.imodel_swm_test_fail_alloc(after) == 0
        try:
            m = make()
        except swm.SWMError as e:
            assert e.code == _capi.ENOMEM
            continue
        finally:
            lib.imodel_swm_test_fail_alloc(0)
        assert not has_tiles(m), "no allocation of a create can be refused"
        return m
    raise AssertionError("no create succeeded")


@pytest.mark.parametrize("weights", [False, True])
def test_separate_kernels_without_memory_for_tiles(grid_at, weights):
    from imodel_gb300 import learned_weights
    g = grid_at(3)
    kw = {"h_ref": 2900.0}
    if weights:
        kw["learned_weights"] = learned_weights.trained_params()
    h, u = swm.initialize_fields_tc2(g)
    a = SWM(g, "fp32", **kw)
    assert a.launch_count(1) == 4
    b = without_tiles(lambda: SWM(g, "fp32", **kw), lambda m: m.launch_count(1) == 4)
    assert b.launch_count(1) == 12
    out = []
    for m in (a, b):
        out.append(m.tendency(h, u) + m.ode_rk4(h, u, 600.0, 4))
        m.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("advection", ["trsk", "upw1"])
@pytest.mark.parametrize("level,case", [(2, 2), (4, 3), (6, 2), (7, 3)])
def test_fused_moist_stage_against_the_separate_kernels(grid_at, level, case, advection):
    """Two steps of the fused moist stage, at each tile size, against the
    separate kernels, element by element.  The shallow-water terms have the same
    bits; the moist terms' products may be fused differently: a rounding (2^-24)
    of every term, about six of them in each of eight evaluations."""
    from imodel_gb300.moist import FIELDS, Moist, moist_fields
    g = grid_at(level)
    f = moist_fields(g, case)
    dt = min(900.0, 110.0 * 2.0 ** (8 - level))

    def make():
        return Moist(g, case, f, advection=advection, precision="fp32")

    out = []
    for m in (make(), without_tiles(make, lambda m: False)):
        m.set_state(f)
        m.advance(dt, 1)
        m.advance(dt, 1)
        out.append(m.get_state())
        m.close()
    eps = 48 * 2.0 ** -24
    s = {k: np.abs(f[k]).max() for k in FIELDS}
    tol = {"htheta": s["htheta"] + 10.0 * s["hqv"], "htracer": s["htracer"]}
    # condensation and rain move what they move with the vapour's rounding
    tol["hqv"] = tol["hqc"] = tol["hqr"] = s["hqv"]
    # the thermal source: g/2 grad(h h theta) / h_e and g theta_e grad(b)
    a, b = g.ed_v0().T
    dx = g.ed_leng * swm.ERAD
    h, q = f["h"], f["htheta"]
    hm = h[a] + h[b]
    force = (np.abs(h[b] - h[a]) * (q[a] + q[b]) / (2.0 * hm) + np.abs(q[b] - q[a]) / 2.0
             + np.abs(f["theta"][a] * (f["bt"][b] - f["bt"][a]))) * swm.GRAV / dx
    tol["u"] = s["u"] + 2.0 * dt * force.max()
    tol["h"] = np.abs(f["h"] - f["h"].mean()).max() + 2.0 * dt * 6.0 * s["h"] * tol["u"] / dx.min()
    for k in FIELDS:
        d = np.abs(out[0][k] - out[1][k])
        assert np.all(np.isfinite(out[0][k])) and d.max() <= eps * tol[k], (k, d.max(), eps * tol[k])
