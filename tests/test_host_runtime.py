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
