"""The clock of the attention's wait for a unit's first piece (WaitClock, host only): it ends a wait 50 ms after its start, and no single reading
of the timer that is off ends one, whichever it is."""
import ctypes

import pytest

import renderformer_cuda_b200 as pkg  # noqa: F401
from renderformer_cuda_b200 import _abi

LIMIT = 50 * 10 ** 6


def _ended(readings):
    words = [r % 2 ** 64 for r in readings]
    return _abi.load("rfk.h").rfk_wait_clock((ctypes.c_ulonglong * len(words))(*words), len(words))


@pytest.mark.parametrize("start", [1, 5 * LIMIT, 2 ** 63 - LIMIT // 2, 2 ** 64 - LIMIT // 2])
def test_a_wait_ends_after_its_limit(start):
    readings = [start + i * LIMIT // 100 for i in range(300)]
    assert 100 < _ended(readings) <= 104
    assert _ended(readings[:100]) == 0


@pytest.mark.parametrize("off", [-10 ** 15, -3 * LIMIT, 3 * LIMIT, 10 ** 15, 2 ** 62])
@pytest.mark.parametrize("bad", [0, 1, 2, 17, 49])
def test_one_reading_that_is_off_ends_no_wait(bad, off):
    readings = [10 ** 16 + i * LIMIT // 100 for i in range(300)]
    readings[bad] += off
    assert _ended(readings[:50]) == 0                 # half the limit has passed
    assert _ended(readings) > 100 or bad < 2          # a start that is off into the future keeps the wait to the other limit


def test_bad_arguments():
    assert _abi.load("rfk.h").rfk_wait_clock(None, 1) == -1 and _ended([]) == -1
