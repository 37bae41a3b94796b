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
