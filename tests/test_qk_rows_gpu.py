"""Norm and rotation of head-split q and k in place (qk_rows_kernel and the form for other widths): the bits of
rfk_qkv_norm_rope_transpose on the same rows, whose own tests compare it with the oracle. One row, fewer rows than blocks, odd
counts that leave half a block without a row, rows of one, two and four warps, an output pitch of more rows than there are."""
import ctypes

import pytest
import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p


@pytest.mark.parametrize("S,heads,hd", [(1, 16, 64), (2, 8, 128), (333, 16, 64), (899, 8, 64), (1777, 16, 128), (5665, 8, 128), (50, 5, 64)])
@pytest.mark.parametrize("parts,rope", [(2, True), (2, False), (1, False)])
def test_rows_in_place_have_the_bits_of_the_transposing_kernel(S, heads, hd, parts, rope):
    dim, pitch = heads * hd, S + 7
    g = torch.Generator(device="cuda").manual_seed(S + heads)
    x = (torch.randn(S, parts * dim, device="cuda", generator=g) * 3).half()
    gamma = [1 + 0.1 * torch.randn(dim, device="cuda", generator=g) for _ in range(parts)]
    cos, sin = (torch.randn(S, hd, device="cuda", generator=g).half() for _ in "cs")
    want = [torch.full((heads, pitch, hd), 7.0, device="cuda", dtype=torch.float16) for _ in range(parts)]
    L = _abi.load("rfk.h")
    p = lambda t: VP(0 if t is None else t.data_ptr())
    stream = VP(torch.cuda.current_stream().cuda_stream)
    arr = lambda ts: (VP * parts)(*[t.data_ptr() for t in ts])
    assert L.rfk_qkv_norm_rope_transpose(p(x), parts * dim, parts, arr(gamma), arr(want), (ctypes.c_int * parts)(*[int(rope)] * parts), p(cos),
                                         p(sin), 1, S, heads, hd, pkg.ops.K_EPS_FP16, pitch, stream) == 0
    got = [torch.full_like(w, 7.0) for w in want]
    for i, o in enumerate(got):
        o[:, :S] = x[:, i * dim:(i + 1) * dim].view(S, heads, hd).transpose(0, 1)
    fn = L.rfk_qk_norm_rope_heads
    fn.argtypes, fn.restype = [VP] * 6 + [ctypes.c_int] * 4 + [ctypes.c_float, VP], ctypes.c_int
    assert fn(p(got[0]), p(got[1] if parts == 2 else None), p(gamma[0]), p(gamma[1] if parts == 2 else None), p(cos if rope else None),
              p(sin if rope else None), S, pitch, heads, hd, pkg.ops.K_EPS_FP16, stream) == 0
    for w, o in zip(want, got):
        assert torch.equal(w, o)
