"""The DPT head's 3x3 convolution on CTA pairs: edges of its 16 x 8 pixel boxes, odd numbers of boxes, one and several images, both
tile widths, both orders of the sums, every epilogue. Oracle: torch fp64 for the convolution (one fp16 rounding, 2^-11 relative, and
the fp32 sum of at most 9 * 192 products of magnitude 1 / sqrt(9 C), 1e-4), and the separate element-wise operators on the
kernel's own plain output for the epilogues, bit for bit - each intermediate is rounded to fp16."""
import ctypes

import pytest
import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p


def _lib():
    L = _abi.load("rfk.h")
    L.rfk_conv3x3_nhwc.argtypes, L.rfk_conv3x3_nhwc.restype = [VP] * 6 + [ctypes.c_int] * 7 + [VP], ctypes.c_int
    L.rfk_conv_error.argtypes, L.rfk_conv_error.restype = [ctypes.POINTER(ctypes.c_int), ctypes.c_int], ctypes.c_int
    L.rfk_residual_add_silu_nhwc.argtypes, L.rfk_residual_add_silu_nhwc.restype = [VP] * 3 + [ctypes.c_longlong, VP], ctypes.c_int
    return L


def _p(t):
    return VP(0 if t is None else t.data_ptr())


def _stream():
    return VP(torch.cuda.current_stream().cuda_stream)


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


def _conv(x, w, bias, res, silu, rows_outside, second=False):
    (N, H, W, C), K = x.shape, w.shape[0]
    out = torch.full((N, H, W, K), 7.0, device="cuda", dtype=torch.float16)
    out2 = torch.full_like(out, 7.0) if second else None
    rc = _lib().rfk_conv3x3_nhwc(_p(x), _p(w), _p(bias), _p(res), _p(out), _p(out2), N, H, W, C, K, int(silu), int(rows_outside), _stream())
    assert rc == 0, rc
    return (out, out2) if second else out


SIZES = [(1, 8, 16, 64, 128), (1, 1, 1, 64, 256), (1, 5, 7, 64, 128), (1, 17, 33, 128, 256), (3, 20, 20, 192, 256), (2, 9, 50, 64, 384),
         (1, 200, 210, 64, 256), (1, 250, 250, 64, 128), (1, 135, 203, 128, 768)]   # several tiles a pair, an odd number of boxes


@pytest.mark.parametrize("rows_outside", [False, True])
@pytest.mark.parametrize("N,H,W,C,K", SIZES)
def test_plain_convolution(N, H, W, C, K, rows_outside):
    x, w, _, _ = _operands(N, H, W, C, K)
    got = _conv(x, w, None, None, False, rows_outside)
    want = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), w.permute(0, 3, 1, 2).double(), padding=1).permute(0, 2, 3, 1)
    assert ((got.double() - want).abs() <= 1e-4 + 1e-3 * want.abs()).all()


@pytest.mark.parametrize("bias,silu,res", [(b, s, r) for b in (0, 1) for s in (0, 1) for r in (0, 1)])
@pytest.mark.parametrize("N,H,W,C,K", SIZES)
def test_epilogues_equal_the_separate_operators(N, H, W, C, K, bias, silu, res):
    x, w, b, r = _operands(N, H, W, C, K)
    b, r = (b if bias else None), (r if res else None)
    want = _conv(x, w, None, None, False, False)
    if bias or silu or res:
        pkg.ops.bias_act_residual_nhwc(want, b, r, N * H * W, K, bool(silu))
    act = torch.empty_like(want)
    pkg.ops.silu(want, act, want.numel())
    assert torch.equal(_conv(x, w, b, r, silu, False), want)
    got, got_act = _conv(x, w, b, r, silu, False, second=True)
    assert torch.equal(got, want) and torch.equal(got_act, act)


@pytest.mark.parametrize("rows_outside", [False, True])
@pytest.mark.parametrize("C,K", [(64, 128), (192, 256)])
def test_order_of_the_sums(C, K, rows_outside):
    """The bits of the projection kernel over the patches laid out in the named order: 64-channel blocks of one tap each."""
    N, H, W = 1, 11, 19
    x, w, _, _ = _operands(N, H, W, C, K)
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    taps = [(r, s) for r in range(3) for s in range(3)]
    blocks = ([(r, s, c) for r in range(3) for c in range(0, C, 64) for s in range(3)] if rows_outside
              else [(r, s, c) for c in range(0, C, 64) for r, s in taps])
    a = torch.cat([xp[0, r:r + H, s:s + W, c:c + 64].reshape(H * W, 64) for r, s, c in blocks], 1).contiguous()
    b = torch.cat([w[:, r, s, c:c + 64] for r, s, c in blocks], 1).contiguous()
    want = torch.empty(H * W, K, device="cuda", dtype=torch.float16)
    pkg.ops.gemm_f16(a, b, want, H * W, K, 9 * C)
    assert torch.equal(_conv(x, w, None, None, False, rows_outside).view(H * W, K), want)


def test_refuses_what_it_does_not_take():
    L = _lib()
    x, w, _, _ = _operands(1, 8, 8, 64, 128)
    out = torch.empty(1, 8, 8, 128, device="cuda", dtype=torch.float16)
    call = lambda C, K, o=out, src=x: L.rfk_conv3x3_nhwc(_p(src), _p(w), None, None, _p(o), None, 1, 8, 8, C, K, 0, 0, _stream())
    assert call(32, 128) == call(64, 64) == -2 and call(64, 128, x) == -1 and call(0, 128) == -1


@pytest.mark.parametrize("n", [8, 2048, 8 * 4097])
def test_sum_and_its_silu_equal_the_separate_operators(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    y, r = (torch.randn(n, device="cuda", generator=g).half() for _ in range(2))
    want, act, got, s = y.clone(), torch.empty_like(y), y.clone(), torch.empty_like(y)
    pkg.ops.residual_add(want, r, n)
    pkg.ops.silu(want, act, n)
    assert _lib().rfk_residual_add_silu_nhwc(_p(got), _p(r), _p(s), n, _stream()) == 0
    assert torch.equal(got, want) and torch.equal(s, act)


def _plan(L, ctx, model, B, pH, pW, library_only):
    dpt, own = VP(), ctypes.c_int(-1)
    L.rfk_dpt_create_from.argtypes = [VP] * 2 + [ctypes.c_int] * 6 + [VP, VP]
    assert L.rfk_dpt_create_from(ctx.h, ctypes.byref(model.dpt_c), B, model.dim, pH, pW, 8, library_only, ctypes.byref(own), ctypes.byref(dpt)) == 0
    return dpt, own.value


@pytest.mark.parametrize("pH,pW,F,B", [(48, 48, 256, 1), (52, 52, 256, 1), (64, 64, 256, 1), (72, 72, 256, 1), (33, 128, 256, 1), (40, 40, 512, 1),
                                       (52, 52, 256, 2), (16, 16, 256, 1)])
def test_heads_have_the_bits_of_the_library_convolutions(pH, pW, F, B):
    """Whole heads, the convolutions of a view on the kernel and all of them with the library: maps whose order of sums the
    library changes from one size to the next, oblong ones, more features, images above 512 pixels, small ones. Several views
    stay with the library."""
    from renderformer_cuda_b200 import session
    L = _abi.load("rfk_layers.h")
    model = session.Model.random(seed=3, dim=256, num_heads=4, ffn_hidden=256, enc_layers=0, dec_layers=1, with_dpt=True, dpt_features=F,
                                 dpt_out_channels=(256, 512, 1024, 1024))
    g = torch.Generator(device="cuda").manual_seed(pH)
    feats = [torch.randn(B, pH * pW, 256, device="cuda", generator=g).half() for _ in range(4)]
    taps, ctx = (VP * 4)(*[f.data_ptr() for f in feats]), session.Ctx()
    images = []
    for library_only in (0, 1):
        dpt, own = _plan(L, ctx, model, B, pH, pW, library_only)
        assert (own > 0) == (not library_only and B == 1)
        image = torch.full((B, 3, pH * 8, pW * 8), 7.0, device="cuda", dtype=torch.float16)
        for _ in range(2):   # the buffers of the first pass are those of the second
            assert L.rfk_dpt_forward(dpt, taps, VP(image.data_ptr()), _stream()) == 0
        torch.cuda.synchronize()
        images.append(image)
        L.rfk_dpt_destroy(dpt)
    assert torch.isfinite(images[0].float()).all() and torch.equal(*images)
    ctx.close()


@pytest.mark.parametrize("p", [8, 24, 40, 48, 52, 64, 72])
def test_convolutions_that_leave_the_library(p):
    """All 3 x 3 convolutions of one view but the one of stride 2: four in front of the fusion blocks, two a residual unit of which three blocks have two
    and one has one, two at full resolution. At 24 x 24 tokens the library adds one of them in an order that the kernel does not have."""
    from renderformer_cuda_b200 import session
    model = session.Model.random(seed=3, dim=64, num_heads=1, ffn_hidden=64, enc_layers=0, dec_layers=1, with_dpt=True, dpt_features=256,
                                 dpt_out_channels=(256, 512, 1024, 1024))
    L, ctx = _abi.load("rfk_layers.h"), session.Ctx()
    dpt, n = _plan(L, ctx, model, 1, p, p, 0)
    left = L.rfk_dpt_num_library_convolutions(dpt)
    L.rfk_dpt_destroy(dpt)
    ctx.close()
    assert n + left == 4 + 2 * (3 * 2 + 1) + 2 + 1 and left == (2 if p == 24 else 1)


def test_a_head_holds_no_copies_beside_its_maps():
    """Device memory of a planned head of a 512 x 512 view: the SiLU copies that producers leave are the buffers in which the residual
    units then build their results, so there is one map per unit beside them. The rounding of allocations to 2 MB and the library's
    handle and workspace are 18 MB more; copies beside the maps would be 132."""
    from renderformer_cuda_b200 import session
    p, F, ch = 64, 256, (256, 512, 1024, 1024)
    model = session.Model.random(seed=3, dim=64, num_heads=1, ffn_hidden=64, enc_layers=0, dec_layers=1, with_dpt=True, dpt_features=F, dpt_out_channels=ch)
    L, ctx = _abi.load("rfk_layers.h"), session.Ctx()
    rn = [(s * p) ** 2 * F for s in (4, 2, 1)] + [(p // 2) ** 2 * F]
    maps = sum(c * p * p for c in ch) + 2 * sum((c * f * f * p * p) for c, f in ((ch[0], 4), (ch[1], 2))) + ch[3] * (p // 2) ** 2
    maps += 2 * sum(rn) + 2 * sum(rn[:3]) + rn[3]                                # layer_rn and its SiLU, one more per residual unit
    maps += 2 * (64 * p * p * F + sum(rn[:3]))                                   # resampled and projected fusion outputs
    maps += (8 * p) ** 2 * (2 * (F // 2) + 32 + 3 + 3)
    filters = sum(c * c * f * f for c, f in ((ch[0], 4), (ch[1], 2))) + 9 * (ch[3] ** 2 + sum(ch) * F + 14 * F * F + F * F // 2 + 32 * F // 2)
    held = []
    for _ in range(2):   # the first plan of a process also loads the library
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        dpt, _ = _plan(L, ctx, model, 1, p, p, 0)
        held.append(before - torch.cuda.mem_get_info()[0])
        L.rfk_dpt_destroy(dpt)
    ctx.close()
    print(f"held {held[1] / 1e6:.1f} MB, maps and filters {2 * (maps + filters) / 1e6:.1f} MB")
    assert held[1] <= 2 * (maps + filters) + (60 << 20)
