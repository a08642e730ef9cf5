"""The word of a handed-over attention unit (handover.cuh) in every order of its two parties' steps, on the host: the second piece takes up
a state only if the first has left it and takes all of the unit otherwise, and the word is zero again for the next launch whatever
becomes of either - a first piece that gives up, a second one that stops waiting, a first one that comes after that."""
import ctypes

import pytest

import renderformer_cuda_b200 as pkg  # noqa: F401
from renderformer_cuda_b200 import _abi

DONE, FAILED, LOOK, SETTLE = range(4)
GO, WAIT, WHOLE = range(3)


def _step(word, event):
    nxt = ctypes.c_int(-1)
    act = _abi.load("rfk.h").rfk_handover_step(word, event, ctypes.byref(nxt))
    assert act >= 0
    return nxt.value, act


@pytest.mark.parametrize("first", [DONE, FAILED])
@pytest.mark.parametrize("patience", range(5))
@pytest.mark.parametrize("late_step", [False, True])
def test_every_order_of_the_steps(first, patience, late_step):
    """`patience`: looks after which the second piece stops waiting; the first piece's step falls before, between or after the looks, or
    (late_step) between the look that ended the wait and the step that follows it."""
    for at in range(patience + 3):
        word, act, gave, settled = 0, None, False, False
        for now in range(patience + 3):
            if now == at and not late_step:
                word, gave = _step(word, first)[0], True
            if not settled:
                same, seen = _step(word, LOOK)
                assert same == word and (seen != WAIT) == gave      # looking changes nothing
                if seen != WAIT or now == patience:
                    if now == at and late_step:
                        word, gave = _step(word, first)[0], True
                    word, act = _step(word, SETTLE)
                    settled = True
                    assert act == (GO if gave and first == DONE else WHOLE)
            if now == at and not gave:
                word, gave = _step(word, first)[0], True
        assert gave and settled and word == 0


def test_bad_arguments():
    step = _abi.load("rfk.h").rfk_handover_step
    assert step(0, LOOK, None) == -1 and step(99, LOOK, ctypes.byref(ctypes.c_int())) == -1


@pytest.mark.parametrize("pieces", range(1, 9))
def test_the_counter_of_a_cut_unit_is_zero_after_its_last_piece(pieces):
    """Whichever pieces give up, in whichever places: the counter is zero behind the last, and a unit is merged once if all arrived."""
    arrives = _abi.load("rfk.h").rfk_piece_arrives
    for failures in range(2 ** pieces):
        counter, merges = ctypes.c_int(0), []
        for i in range(pieces):
            assert counter.value != 0 or i == 0
            merges.append(arrives(ctypes.byref(counter), failures >> i & 1, pieces))
        assert counter.value == 0
        assert merges == [0] * (pieces - 1) + [int(failures == 0)]
