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
