"""Calls that fail, and the calls after them: an error that something else has
left in the thread is the failure, as the runtime reports it once to the next
check."""
import ctypes

import numpy as np
import pytest

from imodel_gb300 import _capi, swm
from imodel_gb300.swm import SWM

pytestmark = pytest.mark.gpu


def _leave_an_error():
    """A failed allocation of the program's own, whose status stays with the
    thread (the library's runtime is this one)."""
    rt = ctypes.CDLL("libcudart.so.13")
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(1 << 62)) == 2
    assert rt.cudaPeekAtLastError() == 2


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("call", ["get_state", "step", "tendency"])
def test_a_failed_call_keeps_no_address_of_the_caller(grid_at, precision, call):
    g = grid_at(3)  # small: the results pass through the handle's area
    h, u = swm.initialize_fields_tc2(g)
    m = SWM(g, precision)
    m.set_state(h, u)
    m.advance(300.0, 1)
    ho, uo = h.copy(), u.copy()
    p = _capi.as_f64p
    _leave_an_error()
    if call == "get_state":
        rc = m.lib.imodel_swm_get_state(m.handle, p(ho), p(uo))
    elif call == "step":
        rc = m.lib.imodel_swm_step(m.handle, p(ho), p(uo), 300.0, 1)
    else:
        rc = m.lib.imodel_swm_tendency(m.handle, p(h), p(u), p(ho), p(uo))
    assert rc == _capi.ECUDA or rc == _capi.ENOMEM
    # the arrays are the program's again: no later call writes to them
    ho[:], uo[:] = -1.0, -2.0
    m.advance(300.0, 1)
    assert np.all(ho == -1.0) and np.all(uo == -2.0)
    m.set_state(h, u)
    m.advance(300.0, 1)
    m.diagnostics()
    m.get_state()
    assert np.all(ho == -1.0) and np.all(uo == -2.0)
    m.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_steps_do_not_fail_on_an_error_of_something_else(grid_at, precision):
    """advance checks its own launches: another part of the program that ran
    out of memory does not make it fail."""
    g = grid_at(3)
    h, u = swm.initialize_fields_tc2(g)
    out = []
    for leave in (False, True):
        m = SWM(g, precision)
        m.set_state(h, u)
        if leave:
            _leave_an_error()
        m.advance(300.0, 3)
        if leave:
            ctypes.CDLL("libcudart.so.13").cudaGetLastError()
        out.append(m.get_state())
        m.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
