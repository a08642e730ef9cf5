"""Units that one CTA begins and another finishes (plan_handover): the bits of whole units, whatever the state that changes hands -
a reference that moves in the second piece's first tile, rows without a finite score yet, a padded last tile -, launch after launch."""
import ctypes

import pytest
import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def tc_path():
    pkg.ops.flash_attention_error(clear=True)
    pkg.ops.flash_attention_set_path(2)      # the tcgen05 kernel or an error
    yield
    pkg.ops.flash_attention_set_path(0)
    _abi.load("rfk.h").rfk_flash_attention_set_split(1)
    torch.cuda.synchronize()
    assert pkg.ops.flash_attention_error(clear=True) == 0


def _call(form, q, k, v, o, B, Hh, Sq, Sk, n_keys, D, ws, ss=None, tiles=0, dim=0, v_shared=False):
    lib = _abi.load("rfk.h")
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if form == "ordered":
        fn = lib.rfk_flash_attention_ordered_ws
        fn.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_size_t] + [ctypes.c_int] * 7 + [ctypes.c_float, ctypes.c_void_p]
        fn.restype = ctypes.c_int
        rc = fn(p(q), p(k), p(v), p(o), p(ws), ws.numel(), B, Hh, Sq, Sk, n_keys, D, 0, D ** -0.5, stream)
    else:
        fn = lib.rfk_flash_attention_ex_wide
        fn.argtypes, fn.restype = lib.rfk_flash_attention_ex.argtypes, ctypes.c_int
        rc = fn(p(q), p(k), p(v), p(o), p(ss), tiles, dim, pkg.ops.K_EPS_FP16, p(ws), ws.numel(), int(v_shared), B, Hh, Sq, Sk, n_keys, D,
                0, D ** -0.5, stream)
    assert rc == 0, rc


def _handed(units, n_tiles):
    """The units that the launcher hands over on this device, none where it cuts the last round along the keys instead."""
    lib = _abi.load("rfk.h")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    whole, n = ctypes.c_int(), ctypes.c_int()
    assert lib.rfk_flash_attention_plan(units, n_tiles, sms, ctypes.byref(whole), ctypes.byref(n), None, 0) == 0
    cut = n.value
    assert lib.rfk_flash_attention_handover_plan(ctypes.c_longlong(units), n_tiles, sms, ctypes.byref(whole), ctypes.byref(n), None, 0) == 0
    return n.value, cut


# units of 256 queries and tiles of 64 keys on 148 SMs: little more than one round, little more than two, of few tiles and of many
@pytest.mark.parametrize("form,D,B,Hh,Sq,Sk,n_keys,scores", [
    ("split", 64, 1, 50, 700, 1024, 1024, "rising"), ("split", 64, 2, 80, 257, 1536, 1530, "random"),
    ("split", 64, 1, 64, 1024, 4104, 4099, "rising"), ("split", 64, 3, 41, 600, 1400, 1399, "empty"),
    ("split", 128, 1, 58, 900, 1604, 1601, "random"), ("split", 128, 1, 50, 700, 1024, 1024, "rising"),
    ("ordered", 128, 1, 38, 1000, 1536, 1529, "rising"), ("ordered", 128, 2, 23, 1024, 5672, 5665, "random"),
    ("ordered", 128, 1, 80, 300, 2000, 1990, "empty")])
def test_handed_over_units_have_the_bits_of_whole_ones(form, D, B, Hh, Sq, Sk, n_keys, scores):
    units, n_tiles = B * Hh * -(-Sq // 256), -(-n_keys // 64)
    handed, cut = _handed(units, n_tiles)
    assert handed > 0 and (form == "ordered" or cut == 0), (units, n_tiles, handed, cut)
    g = torch.Generator(device="cuda").manual_seed(units)
    Q, K, V = (torch.randn(B, Hh, n, D, device="cuda", generator=g).half() for n in (Sq, Sk, Sk))
    if scores != "random":    # every tile's maximum above the one before: the reference moves all along the keys
        d = torch.nn.functional.normalize(Q.float().mean(2, keepdim=True), dim=-1)
        K = (K.float() + 40.0 * torch.linspace(0.0, 1.0, Sk, device="cuda").view(1, 1, Sk, 1) * d).half()
    if scores == "empty":     # rows whose first finite score comes late, or never
        Q[:, :, ::7] = Q[:, :, ::7].abs() + 0.01
        Q[:, :, 3] = float("inf")
        K[:, :, : Sk * 3 // 4, 0] = -float("inf")
        Q[:, :, :, 0] = Q[:, :, :, 0].abs() + 0.01
    ws = pkg.ops.flash_attention_workspace()
    lib = _abi.load("rfk.h")
    outs = []
    for split in (0, 1, 1):
        lib.rfk_flash_attention_set_split(split)
        outs.append(torch.full_like(Q, 7.0))
        _call(form, Q, K, V, outs[-1], B, Hh, Sq, Sk, n_keys, D, ws)
    words = [o.view(torch.int16) for o in outs]      # NaN included
    assert torch.equal(words[0], words[1]) and torch.equal(words[0], words[2]) and not ws[:1024].any()
    if scores == "random":
        want = torch.nn.functional.scaled_dot_product_attention(Q.float(), K[:, :, :n_keys].float(), V[:, :, :n_keys].float())
        assert (outs[1].float() - want).abs().max() < 4e-3 + 4e-3 * want.abs().max()


def test_handed_over_units_with_row_statistics_and_shared_values():
    B, Hh, Sq, Sk, D = 2, 16, 1300, 2000, 64       # 192 units of 32 tiles
    assert _handed(192, 32)[0] > 0 and _handed(192, 32)[1] == 0
    g = torch.Generator(device="cuda").manual_seed(5)
    Q, K = (torch.randn(B, Hh, n, D, device="cuda", generator=g).half() for n in (Sq, Sk))
    V = torch.randn(Hh, Sk, D, device="cuda", generator=g).half()
    ss = 64 + 900 * torch.rand(B * Sq, 4, device="cuda", generator=g)
    ws = pkg.ops.flash_attention_workspace()
    outs = []
    for split in (0, 1):
        _abi.load("rfk.h").rfk_flash_attention_set_split(split)
        outs.append(torch.full_like(Q, 7.0))
        _call("split", Q, K, V, outs[-1], B, Hh, Sq, Sk, Sk, D, ws, ss=ss, tiles=4, dim=Hh * D, v_shared=True)
    assert torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0].float()).all()


@pytest.mark.parametrize("form,D,B,Hh,Sq,Sk", [("split", 64, 1, 50, 700, 1024), ("ordered", 128, 1, 38, 1000, 1536)])
def test_a_second_piece_without_a_state_takes_the_unit(form, D, B, Hh, Sq, Sk):
    """The first pieces find that their units have been taken (3) and leave no state, so that each second piece runs into the limit of its
    wait, 50 ms, and computes all of its unit: the same bits, and no error."""
    handed, cut = _handed(B * Hh * -(-Sq // 256), -(-Sk // 64))
    assert handed > 0 and (form == "ordered" or cut == 0)
    g = torch.Generator(device="cuda").manual_seed(9)
    Q, K, V = (torch.randn(B, Hh, n, D, device="cuda", generator=g).half() for n in (Sq, Sk, Sk))
    ws, outs = pkg.ops.flash_attention_workspace(), []
    for taken in (False, True):
        ws[:1024].view(torch.int32)[:handed] = 3 if taken else 0
        outs.append(torch.full_like(Q, 7.0))
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        _call(form, Q, K, V, outs[-1], B, Hh, Sq, Sk, Sk, D, ws)
        end.record()
        end.synchronize()
        assert (start.elapsed_time(end) > 40) == taken
    assert torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0].float()).all()


def test_two_launches_in_flight_on_two_streams():
    """Handed-over launches of two streams share the SMs, each with a workspace of its own: the bits of each alone, time after time."""
    B, Hh, Sq, Sk, D = 1, 50, 700, 1024, 64          # 150 units of 16 tiles
    assert _handed(150, 16)[0] > 0 and _handed(150, 16)[1] == 0
    g = torch.Generator(device="cuda").manual_seed(11)
    sides = []
    for _ in range(2):
        q, k, v = (torch.randn(B, Hh, n, D, device="cuda", generator=g).half() for n in (Sq, Sk, Sk))
        want = torch.empty_like(q)
        ws = pkg.ops.flash_attention_workspace()
        _call("split", q, k, v, want, B, Hh, Sq, Sk, Sk, D, ws)
        sides.append((q, k, v, want, ws, torch.cuda.Stream(), [torch.full_like(q, 7.0) for _ in range(20)]))
    torch.cuda.synchronize()
    for i in range(20):
        for q, k, v, _, ws, stream, outs in sides:
            with torch.cuda.stream(stream):
                _call("split", q, k, v, outs[i], B, Hh, Sq, Sk, Sk, D, ws)
    torch.cuda.synchronize()
    for _, _, _, want, ws, _, outs in sides:
        assert all(torch.equal(o, want) for o in outs) and not ws[:1024].any()
