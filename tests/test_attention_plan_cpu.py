"""CPU tests of the attention launcher's work planning (rfk_flash_attention_plan, host only): which grids are cut
along the keys, and that a cut covers every key tile of every unit exactly once with consistent slot bookkeeping."""
import ctypes
import heapq

import pytest

import renderformer_cuda_b200 as pkg  # noqa: F401
from renderformer_cuda_b200 import _abi


def _plan(units, n_tiles, sms=148):
    lib = _abi.load("rfk.h")
    whole, n = ctypes.c_int(-1), ctypes.c_int(-1)
    buf = (ctypes.c_ushort * (6 * 320))()
    rc = lib.rfk_flash_attention_plan(units, n_tiles, sms, ctypes.byref(whole), ctypes.byref(n), ctypes.cast(buf, ctypes.c_void_p), 320)
    assert rc == 0
    pieces = [tuple(buf[6 * i + k] for k in range(6)) for i in range(n.value)]
    return whole.value, pieces


@pytest.mark.parametrize("units,n_tiles,sms", [(64, 89, 148), (12, 32, 148), (1, 64, 148), (7, 500, 132), (100, 200, 148),
                                               (3, 9, 148), (147, 1000, 148), (40, 89, 16)])
def test_cut_grids_cover_every_tile_once(units, n_tiles, sms):
    whole, pieces = _plan(units, n_tiles, sms)
    if not pieces:
        assert whole == units
        return
    assert whole == 0 and units < sms                                   # only grids that leave SMs idle are cut
    assert len(pieces) <= 320 and len(pieces) <= 2 * min(sms, 160)
    covered = {u: [0] * n_tiles for u in range(units)}
    by_unit = {}
    for unit, t0, nt, first, count, slot in pieces:
        assert nt >= 1 and t0 + nt <= n_tiles
        for t in range(t0, t0 + nt):
            covered[unit][t] += 1
        by_unit.setdefault(unit, []).append((first, count, slot))
    assert all(c == 1 for u in covered.values() for c in u), "a key tile is missed or taken twice"
    slots = sorted(s for v in by_unit.values() for _, _, s in v)
    assert slots == list(range(len(pieces)))                            # one workspace slot per piece
    for unit, recs in by_unit.items():
        first, count = recs[0][0], recs[0][1]
        assert all(r[0] == first and r[1] == count for r in recs) and count == len(recs) and count <= 9
        assert sorted(r[2] for r in recs) == list(range(first, first + count))   # the unit's slots are consecutive
    sizes = [p[2] for p in pieces]
    assert sizes == sorted(sizes, reverse=True)                         # longest first
    share = -(-units * n_tiles // min(sms, 160, units * 8))
    assert max(sizes) <= share


@pytest.mark.parametrize("units,n_tiles", [(256, 89), (148, 89), (108, 25), (4, 1), (64, 10), (300, 40), (0, 5)])
def test_grids_left_whole(units, n_tiles):
    """A grid of one round or more, or pieces so short that their fixed cost (about twelve tile times) eats the gain."""
    whole, pieces = _plan(units, n_tiles)
    assert whole == units and pieces == []


def test_plan_rejects_bad_arguments():
    lib = _abi.load("rfk.h")
    w, n = ctypes.c_int(), ctypes.c_int()
    assert lib.rfk_flash_attention_plan(4, 0, 148, ctypes.byref(w), ctypes.byref(n), None, 0) == -1
    assert lib.rfk_flash_attention_plan(4, 8, 0, ctypes.byref(w), ctypes.byref(n), None, 0) == -1
    assert lib.rfk_flash_attention_plan(4, 8, 148, None, ctypes.byref(n), None, 0) == -1
    assert lib.rfk_flash_attention_plan(64, 89, 148, ctypes.byref(w), ctypes.byref(n), None, 0) == 0 and n.value > 0   # count only


@pytest.mark.parametrize("units,n_tiles,sms", [(184, 89, 148), (208, 89, 148), (149, 200, 148), (301, 500, 148), (20, 64, 16)])
def test_last_round_is_cut_behind_whole_rounds(units, n_tiles, sms):
    whole, pieces = _plan(units, n_tiles, sms)
    assert whole == units // sms * sms and pieces
    seen = [[0] * n_tiles for _ in range(units)]
    for unit, t0, nt, first, count, slot in pieces:
        assert unit >= whole and first <= slot < first + count <= len(pieces)
        for t in range(t0, t0 + nt):
            seen[unit][t] += 1
    assert all(c == 1 for u in seen[whole:] for c in u)


@pytest.mark.parametrize("units,n_tiles", [(368, 89), (464, 113), (224, 55), (232, 113)])
def test_last_round_that_saves_less_than_a_fifth_stays_whole(units, n_tiles):
    """The line that the header states. The encoder of a scene of 5633 triangles and 16 heads is 368 units of 89 tiles, where a cut is
    estimated to save 12 %: its sums, and with them the K/V cache and the views, keep their order."""
    assert _plan(units, n_tiles) == (units, [])


def _handover(units, n_tiles, sms=148):
    fn = _abi.load("rfk.h").rfk_flash_attention_handover_plan
    fn.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int),
                   ctypes.c_void_p, ctypes.c_int]
    fn.restype = ctypes.c_int
    whole, n = ctypes.c_int(-1), ctypes.c_int(-1)
    buf = (ctypes.c_ushort * (3 * 160))()
    assert fn(units, n_tiles, sms, ctypes.byref(whole), ctypes.byref(n), ctypes.cast(buf, ctypes.c_void_p), 160) == 0
    return whole.value, [tuple(buf[3 * i + k] for k in range(3)) for i in range(n.value)]


@pytest.mark.parametrize("sms", [148, 132, 16, 160])
def test_handed_over_units_fill_the_last_round(sms):
    """Every unit is taken once; the first pieces are launched together and wait for nothing, so that a second piece always waits for
    a block ahead of it; blocks handed out in order finish sooner than whole units by what the plan asks for, and no second piece
    starts before its first one is done."""
    cta, give, take = 5, 2, 2
    planned = 0
    for units in range(1, 4 * sms, max(1, sms // 12)):
        for n_tiles in (3, 15, 16, 33, 89, 700):
            whole, handed = _handover(units, n_tiles, sms)
            rounds = -(-units // sms) * (n_tiles + cta)
            if not handed:
                assert whole == units
                continue
            planned += 1
            assert units > sms and len(handed) < sms
            assert sorted(u for u, _, _ in handed) == list(range(whole, units)) and sorted(s for _, _, s in handed) == list(range(len(handed)))
            assert all(4 <= first <= n_tiles - 4 for _, first, _ in handed)
            free, ready = [0] * sms, {}
            heapq.heapify(free)
            for u, first, _ in handed:
                ready[u] = heapq.heappop(free) + first + cta + give
                heapq.heappush(free, ready[u])
            for _ in range(whole):
                heapq.heappush(free, heapq.heappop(free) + n_tiles + cta)
            for u, first, _ in sorted(handed, key=lambda h: h[1]):
                start = heapq.heappop(free)
                assert start >= ready[u]
                heapq.heappush(free, start + n_tiles - first + cta + take)
            assert max(free) <= 0.96 * rounds
    assert planned > 10
    assert _handover(sms, 89, sms) == (sms, []) and _handover(2 * sms, 89, sms) == (2 * sms, []) and _handover(70000, 89, sms) == (70000, [])
    assert _handover(200, 89, 161) == (200, [])          # more SMs than slots
