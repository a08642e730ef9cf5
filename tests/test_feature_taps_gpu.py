"""The feature taps of a view: a tapped layer writes its tap itself and the next layer goes on from there. A tap is what a shorter
network's token map is; the last layer may be tapped (its map is copied) or not (it writes the token map itself)."""
import ctypes

import pytest
import torch

from renderformer_cuda_b200 import _abi, session

pytestmark = pytest.mark.gpu


class _Span:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f2", "data": (ptr, False), "version": 3}


def _frames(model, layers, scene, cams):
    """Per camera the token map and the four taps of a session with the model's first `layers` decoder layers."""
    model.c.dec_layers = layers
    s = session.RenderSession(model, scene[0].shape[0], 128)
    s.encode_scene(*scene)
    s.finalize()
    out = []
    for cam in cams:
        s.render_frame(cam, 0.7)
        tokens = s.download().clone().flatten().cuda()
        ptr = (ctypes.c_void_p * 4)()
        assert _abi.load("rfk_layers.h").rfk_session_feature_taps(s.h, ptr) == 0
        out.append((tokens, [torch.as_tensor(_Span(p, tokens.numel()), device="cuda") for p in ptr]))
    torch.cuda.synchronize()
    out = [(t, [x.clone() for x in taps]) for t, taps in out]     # after the last frame: the one before keeps its own
    torch.cuda.synchronize()
    s.close()
    return out


@pytest.mark.parametrize("heads", [4, 2])
def test_taps_are_the_token_maps_of_shorter_networks(heads):
    model = session.Model.random(seed=6, dim=256, num_heads=heads, ffn_hidden=512, enc_layers=1, dec_layers=20, num_register_tokens=5)
    g = torch.Generator(device="cuda").manual_seed(6)
    tri = torch.rand(50, 3, 3, device="cuda", generator=g) * 2 - 1
    vn = torch.nn.functional.normalize(torch.randn(50, 3, 3, device="cuda", generator=g), dim=-1)
    scene = (tri.contiguous(), vn.contiguous(), torch.rand(50, 13, device="cuda", generator=g).half())
    cams = [torch.eye(4), torch.eye(4)]
    cams[0][2, 3], cams[1][2, 3] = 3.0, 4.0
    long = _frames(model, 20, scene, cams)                                 # taps behind layers 5, 10, 15 and 20
    shorter = {n: _frames(model, n, scene, cams) for n in (5, 10, 15)}     # the first has its own taps behind 1 to 4
    for v in range(2):
        tokens, taps = long[v]
        assert torch.isfinite(tokens.float()).all() and torch.equal(taps[3], tokens)
        for i, n in enumerate((5, 10, 15)):
            assert torch.equal(taps[i], shorter[n][v][0]), n
        assert not torch.equal(taps[0], taps[1])
    assert not torch.equal(long[0][1][0], long[1][1][0])
