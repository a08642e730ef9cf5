"""The rotation kernels at the edges of their forms: batches of one tensor that share a table (the cached keys of several layers), odd numbers of
heads, grids of more heads or batches than a grid dimension has blocks, rows that are copied, results longer than half of the L2."""
import ctypes

import pytest
import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu
ops = pkg.ops


def _rotated(x, cos, sin):
    half = x.shape[-1] // 2
    x = x.float()
    return x * cos.float() + torch.cat([-x[..., half:], x[..., :half]], -1) * sin.float()


def _near(got, want):
    # one rounding to fp16 (spacing 2^-10 of the value at most), beside fp32 products of values of order one that may cancel
    assert ((got.float() - want).abs() <= want.abs() * 2.0 ** -10 + 1e-6).all()


@pytest.mark.parametrize("layers,heads,rows,hd", [(1, 2, 33, 64), (2, 3, 33, 64), (3, 2, 1, 16), (12, 16, 127, 64), (12, 8, 65, 128),
                                                  (5, 4, 129, 48), (12, 16, 3000, 64)])
@pytest.mark.parametrize("scaled", [False, True])
def test_layers_that_share_a_table(layers, heads, rows, hd, scaled):
    g = torch.Generator(device="cuda").manual_seed(layers * 1000 + rows)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    src = rnd(layers, 2, heads, rows, hd).half()     # a K and a V slab a layer
    cos, sin = rnd(rows, hd).half(), rnd(rows, hd).half()
    scale = rnd(layers, heads * hd) if scaled else None
    dst = torch.full((layers, heads, rows, hd), float("nan"), device="cuda", dtype=torch.half)
    fn = _abi.load("rfk.h").rfk_rope_one_oop_strided
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())
    slab = heads * rows * hd
    assert fn(p(src), p(dst), p(cos), p(sin), layers, 2 * slab, slab, 0, heads, rows, hd, rows, rows, p(scale), heads * hd if scaled else 0,
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = _rotated(src[:, 0], cos, sin)
    if scaled:
        want = want * scale.view(layers, heads, 1, hd)
    _near(dst, want)


@pytest.mark.parametrize("batch,heads,rows,hd", [(1, 70000, 1, 16), (70000, 1, 1, 16), (2, 3, 43, 48), (1, 1, 1, 64), (3, 16, 129, 128)])
def test_two_tensors_in_place(batch, heads, rows, hd):
    g = torch.Generator(device="cuda").manual_seed(batch + heads)
    q, k = (torch.randn(batch, heads, rows, hd, device="cuda", generator=g).half() for _ in range(2))
    cos, sin = (torch.randn(batch, rows, hd, device="cuda", generator=g).half() for _ in range(2))
    want = [_rotated(t, cos[:, None], sin[:, None]) for t in (q, k)]
    ops.apply_rope(q, k, cos, sin, batch, heads, rows, hd)
    _near(q, want[0])
    _near(k, want[1])


def test_rows_behind_the_sequence_are_copied():
    g = torch.Generator(device="cuda").manual_seed(3)
    src = torch.randn(2, 4, 40, 64, device="cuda", generator=g).half()
    cos, sin = (torch.randn(2, 33, 64, device="cuda", generator=g).half() for _ in range(2))
    dst = torch.empty_like(src)
    ops.rope_one_oop(src, dst, cos, sin, 2, 4, 33, 64, 40, 40, True)
    _near(dst[:, :, :33], _rotated(src[:, :, :33], cos[:, None], sin[:, None]))
    assert torch.equal(dst[:, :, 33:], src[:, :, 33:])


@pytest.mark.parametrize("hd", [24, 64])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_one_tensor_given_twice_is_rotated_twice(hd, dtype):
    g = torch.Generator(device="cuda").manual_seed(hd)
    x = torch.randn(2, 3, 70, hd, device="cuda", generator=g).to(dtype)
    cos, sin = (torch.randn(2, 70, hd, device="cuda", generator=g).half() for _ in range(2))
    both, one = (ops.apply_rope, ops.apply_rope_one) if dtype == torch.float16 else (ops.apply_rope_f32, ops.apply_rope_one_f32)
    got, want = x.clone(), x.clone()
    both(got, got, cos, sin, 2, 3, 70, hd)
    for _ in range(2):
        one(want, cos, sin, 2, 3, 70, hd)
    assert torch.equal(got, want)
