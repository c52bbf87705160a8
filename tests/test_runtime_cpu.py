"""Per-device set-up: run once when it succeeds, and again after a failure (the
upload of tables can fail for want of memory that is there later)."""
import ctypes

import pytest

from pentago_b200 import capi


@pytest.mark.parametrize("failures", [0, 1, 3])
def test_a_setup_that_failed_is_tried_again(failures):
    runs = ctypes.c_int(-1)
    assert capi.lib().pg_selftest_once(failures, ctypes.byref(runs)) == 0
    assert runs.value == failures + 1
