"""Host code of the GPU drivers, run without a GPU (see _hostlib.py)."""
import ctypes as C

import _hostlib
import numpy as np
import pytest


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return _hostlib.load(tmp_path_factory.mktemp("host"))


def test_exchange_words_hold_tags_of_one_form(lib):
    assert lib.check_exchange_roles() == 0


@pytest.mark.parametrize("stops", [[0], [511], [512], [1600], [0, 1, 1023, 1024], [700, 100], [1600, 0]])
def test_start_state_does_not_depend_on_when_it_is_read(lib, stops):
    assert lib.check_start_state((C.c_int * len(stops))(*stops), len(stops)) == 0


@pytest.mark.parametrize("check_every", [0, 1])
@pytest.mark.parametrize("volume", [0.0, 1e-300, 3.7e-3, 2.5e6])
@pytest.mark.parametrize("tol", [-np.inf, -400.0, -17.5, -16.0, -15.5, -14.9, -10.0, 0.0, 3.0, 154.5, 200.0, np.inf,
                                 np.nan])
def test_stop_test_follows_the_plain_rule(lib, tol, volume, check_every):
    """Sums on both sides of the tolerance, and those a volume without points
    (integration radius below the first cell) or a diverged run gives."""
    near = volume * 10.0 ** (2.0 * min(max(tol, -30.0), 150.0)) if np.isfinite(tol) else 1.0
    sums = np.array([0.0, np.inf, np.nan, 1e-320, 1e-30, 1.0, 1e300]
                    + [near * f for f in (0.5, 1 - 1e-6, 1 - 1e-8, 1 + 1e-8, 1 + 1e-6, 2.0)])
    assert lib.check_stop_rule(C.c_double(tol), C.c_double(volume), check_every,
                               sums.ctypes.data_as(C.POINTER(C.c_double)), len(sums)) == 0
