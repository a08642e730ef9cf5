"""Every tile of the DPT head's 3x3 convolution at the edges of its pixel boxes (16 x 8 and 8 x 8) and channel blocks: fewer pixels than a box, odd
numbers of boxes, several tiles a pair, 32 and 96 output channels in tiles of 64, both orders of the sums, every epilogue. Oracles: torch in fp64
(one fp16 rounding, 2^-11 relative, and the fp32 sum of products of magnitude 1 / sqrt(9 C), 1e-4), the widest tile that takes the shape for
the order of the sums (bit for bit; the order itself is pinned against the projection kernel elsewhere), and the separate element-wise operators on
the kernel's own plain output, bit for bit."""
import ctypes

import pytest
import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p
RULE, T128x128, T64x128, T64x64, T32x128 = range(5)


def _lib():
    L = _abi.load("rfk.h")
    L.rfk_conv3x3_nhwc_tiled.argtypes, L.rfk_conv3x3_nhwc_tiled.restype = [VP] * 6 + [ctypes.c_int] * 8 + [VP], ctypes.c_int
    L.rfk_conv_error.argtypes, L.rfk_conv_error.restype = [ctypes.POINTER(ctypes.c_int), ctypes.c_int], ctypes.c_int
    return L


def _p(t):
    return VP(0 if t is None else t.data_ptr())


@pytest.fixture(autouse=True)
def _no_time_out():
    L, code = _lib(), ctypes.c_int()
    L.rfk_conv_error(ctypes.byref(code), 1)
    yield
    torch.cuda.synchronize()
    assert L.rfk_conv_error(ctypes.byref(code), 1) == 0 and code.value == 0


def _operands(N, H, W, C, K):
    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W + C)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    return rnd(N, H, W, C).half(), (rnd(K, 3, 3, C) / (9 * C) ** 0.5).half(), rnd(K).half(), rnd(N, H, W, K).half()


def _conv(x, w, bias, res, silu, rows_outside, tile, second=False):
    (N, H, W, C), K = x.shape, w.shape[0]
    out = torch.full((N, H, W, K), 7.0, device="cuda", dtype=torch.float16)
    out2 = torch.full_like(out, 7.0) if second else None
    rc = _lib().rfk_conv3x3_nhwc_tiled(_p(x), _p(w), _p(bias), _p(res), _p(out), _p(out2), N, H, W, C, K, int(silu), int(rows_outside), tile,
                                       VP(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, rc
    return (out, out2) if second else out


# small and ragged maps, an odd number of boxes, several tiles a pair of SMs (of a single channel block each, for 32 channels), several images
CASES = [(t, *s) for t in (T128x128, T64x128, T64x64, RULE) for s in [(1, 1, 1, 64, 128), (1, 8, 16, 64, 128), (1, 9, 17, 192, 256), (3, 20, 20, 128, 128),
                                                                     (1, 200, 210, 64, 128)]]
CASES += [(t, *s) for t in (T64x128, T64x64, RULE) for s in [(1, 5, 7, 64, 32), (1, 17, 33, 128, 96), (2, 9, 50, 192, 64), (1, 150, 130, 64, 96)]]
CASES += [(T32x128, *s) for s in [(1, 1, 1, 64, 32), (1, 7, 18, 128, 32), (2, 30, 33, 128, 32), (1, 200, 210, 64, 32)]]


@pytest.mark.parametrize("tile,N,H,W,C,K", CASES)
def test_plain_convolution_and_order_of_the_sums(tile, N, H, W, C, K):
    x, w, _, _ = _operands(N, H, W, C, K)
    want = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), w.permute(0, 3, 1, 2).double(), padding=1).permute(0, 2, 3, 1)
    for rows_outside in (False, True):
        got = _conv(x, w, None, None, False, rows_outside, tile)
        assert ((got.double() - want).abs() <= 1e-4 + 1e-3 * want.abs()).all()
        assert torch.equal(got, _conv(x, w, None, None, False, rows_outside, T64x128 if K % 128 else T128x128))


@pytest.mark.parametrize("tile,N,H,W,C,K", CASES)
def test_epilogues_equal_the_separate_operators(tile, N, H, W, C, K):
    x, w, bias, residual = _operands(N, H, W, C, K)
    plain = _conv(x, w, None, None, False, False, tile)
    for b, r, silu in [(bias, None, True), (bias, residual, False), (None, residual, True), (None, None, False), (bias, residual, True)]:
        want = plain.clone()
        if b is not None or r is not None or silu:
            pkg.ops.bias_act_residual_nhwc(want, b, r, N * H * W, K, silu)
        act = torch.empty_like(want)
        pkg.ops.silu(want, act, want.numel())
        assert torch.equal(_conv(x, w, b, r, silu, False, tile), want)
        got, got_act = _conv(x, w, b, r, silu, False, tile, second=True)
        assert torch.equal(got, want) and torch.equal(got_act, act)


@pytest.mark.parametrize("tile,N,H,W,C,K", [c for c in CASES if c[0] != T32x128 and not (c[4] <= 128 and c[5] == 32)])
def test_sum_into_the_path_equals_the_separate_operators(tile, N, H, W, C, K):
    L = _lib()
    L.rfk_conv3x3_nhwc_add.argtypes, L.rfk_conv3x3_nhwc_add.restype = [VP] * 6 + [ctypes.c_int] * 7 + [VP], ctypes.c_int
    L.rfk_residual_add_silu_nhwc.argtypes, L.rfk_residual_add_silu_nhwc.restype = [VP] * 3 + [ctypes.c_longlong, VP], ctypes.c_int
    x, w, bias, residual = _operands(N, H, W, C, K)
    st = VP(torch.cuda.current_stream().cuda_stream)
    path = torch.randn(N, H, W, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(H)).half()
    for b, r in [(bias, residual), (None, None)]:
        unit, want, want_silu = _conv(x, w, b, r, False, False, tile), path.clone(), torch.empty_like(path)
        assert L.rfk_residual_add_silu_nhwc(_p(want), _p(unit), _p(want_silu), want.numel(), st) == 0
        got, got_silu = path.clone(), torch.full_like(path, 7.0)
        assert L.rfk_conv3x3_nhwc_add(_p(x), _p(w), _p(b), _p(r), _p(got), _p(got_silu), N, H, W, C, K, 0, tile, st) == 0
        assert torch.equal(got, want) and torch.equal(got_silu, want_silu)
    assert L.rfk_conv3x3_nhwc_add(_p(x), _p(w), None, _p(got), _p(got), _p(got_silu), N, H, W, C, K, 0, tile, st) == -1


def test_refuses_tiles_that_do_not_take_the_shape():
    x, w, _, _ = _operands(1, 8, 8, 64, 96)
    out = torch.full((1, 8, 8, 96), 7.0, device="cuda", dtype=torch.float16)
    call = lambda C, K, tile: _lib().rfk_conv3x3_nhwc_tiled(_p(x), _p(w), None, None, _p(out), None, 1, 8, 8, C, K, 0, 0, tile, None)
    assert call(64, 96, T128x128) == call(64, 96, T32x128) == call(192, 32, T32x128) == call(64, 96, 5) == call(64, 96, -1) == -1   # RFK_EINVAL
    assert call(64, 40, RULE) == call(32, 96, RULE) == -2                                                                         # RFK_EUNSUPPORTED
    torch.cuda.synchronize()
    assert (out == 7).all()
