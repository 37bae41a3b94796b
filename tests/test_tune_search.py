"""The autotuner's search, with given times in place of measured ones (no GPU):
configurations whose kernels are the same are timed once, and the block sizes
kept are sizes that were timed on kernels which use them."""
import ctypes

import pytest

from imodel_gb300 import _capi

TRIAL = ctypes.CFUNCTYPE(ctypes.c_float, ctypes.POINTER(ctypes.c_int32))


def search(space, time):
    lib = _capi.swm_lib()
    seen = []

    def trial(c):
        t = tuple(c[:6])
        seen.append(t)
        return time(t, len(seen))

    choice = (ctypes.c_int32 * 6)()
    lib.imodel_swm_test_tune_search.argtypes = [ctypes.POINTER(ctypes.c_int32), TRIAL,
                                                ctypes.POINTER(ctypes.c_int32)]
    assert lib.imodel_swm_test_tune_search((ctypes.c_int32 * 4)(*space), TRIAL(trial), choice) == 0
    return tuple(choice), seen


def separate(t, base, best):
    """Separate kernels: 1 ms more for every block size that is not the best."""
    return base + sum(1.0 for a, b in zip(t[1:5], best) if a != b)


def test_fused_stage_is_timed_once_and_keeps_measured_sizes():
    best = (128, 256, 512, 256)

    def time(t, k):
        # what the fused stage's time varies by from trial to trial
        if t[0] == 1:
            return 10.0 - 0.01 * k
        return separate(t, {0: 50.0, 2: 20.0}[t[0]], best)

    choice, seen = search((1, 1, 1, 0), time)
    assert len([t for t in seen if t[0] == 1]) == 1
    assert choice[0] == 1
    # (the pre-pass, which variant 2 runs with options only, is not refined)
    assert (choice[1], choice[3], choice[4]) == (128, 512, 256)


def test_same_kernels_are_timed_once():
    best = (512, 128, 128, 512)
    choice, seen = search((1, 1, 0, 0), lambda t, k: separate(t, 30.0 if t[0] == 0 else 20.0, best))
    assert {t[0] for t in seen} == {0, 1}
    assert len(set(seen)) == len(seen)
    assert choice[0] == 1 and (choice[1], choice[3], choice[4]) == (512, 128, 512)


@pytest.mark.parametrize("space,fast", [((1, 1, 1, 0), 0), ((1, 1, 1, 0), 2), ((1, 0, 0, 0), 0)])
def test_the_fastest_separate_variant(space, fast):
    best = (256, 512, 128, 512)
    choice, seen = search(
        space, lambda t, k: 90.0 if t[0] == 1 else separate(t, 20.0 if t[0] == fast else 40.0, best))
    assert choice[0] == fast
    assert (choice[1], choice[3], choice[4]) == (256, 128, 512)
    assert fast != 0 or choice[2] == 512
    assert len(set(seen)) == len(seen)
    assert space[1] or {t[0] for t in seen} == {0}


def test_network_split():
    choice, seen = search((0, 1, 0, 1), lambda t, k: separate(t, 20.0, (256,) * 4) + (5 - t[5]))
    assert choice == (1, 256, 256, 256, 256, 4)
    assert {t[0] for t in seen} == {1}


def test_no_configuration_runs():
    """Every trial fails: a variant that the handle may run, whatever its sizes."""
    for space, variant in (((1, 0, 0, 0), 0), ((1, 1, 0, 0), 1), ((1, 1, 1, 0), 1)):
        assert search(space, lambda t, k: 1e30)[0][0] == variant
