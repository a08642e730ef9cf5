"""Sessions with 128-wide heads end to end: scene in, token map out, with and without an image head (which keeps the mma.sync
attention, the library's window products and the separate query norm), and on every path a program can set. Oracle: the fp64
torch evaluation of the decoder layers on the session's own K/V cache and tables. Bound: that of the layers' tests, four
layers here as there (fp16 rounding between the steps, 9.6e-4 mean and 1.6e-2 largest), with one more rounded step ahead."""
import numpy as np
import pytest
import torch

import renderformer_cuda_b200 as pkg
import torch_layers as TL
from oracle import ref_pipeline as RP

pytestmark = pytest.mark.gpu
ops, H16 = pkg.ops, torch.float16
N, RES, DIM, HEADS, HD = 300, 128, 256, 2, 128


@pytest.fixture(autouse=True)
def _paths():
    yield
    ops.gemm_set_path(0)
    ops.flash_attention_set_path(0)
    torch.cuda.synchronize()
    assert ops.gemm_error() == 0 and ops.flash_attention_error() == 0 and ops.conv_error() == 0


def _render(with_dpt):
    """(token map, the same in fp64 from this session's scene state)"""
    from renderformer_cuda_b200 import session
    import cases
    m = session.Model.random(seed=6, dim=DIM, num_heads=HEADS, ffn_hidden=1024, enc_layers=1, dec_layers=4, num_register_tokens=5,
                             with_dpt=with_dpt, dpt_features=64, dpt_out_channels=(32, 64, 128, 128))
    g = torch.Generator(device="cuda").manual_seed(8)
    tri = (torch.rand(N, 3, 3, device="cuda", generator=g) * 2 - 1).contiguous()
    vn = torch.nn.functional.normalize(torch.randn(N, 3, 3, device="cuda", generator=g), dim=-1).contiguous()
    tex = torch.rand(N, 13, device="cuda", generator=g).half()
    c2w, fov = cases.look_at_c2w(np.random.default_rng(2), 1)
    s = session.RenderSession(m, N, RES)
    s.encode_scene(tri, vn, tex)
    s.finalize()
    s.render_frame(c2w[0], float(fov[0]))
    got = s.download().clone().cuda()
    lay, state = RP.state_layout(m, N), s.scene_state
    Se, pad, P = lay["Se"], lay["Se_pad"], RES // 8
    kv = state[:2 * m.dec_layers * lay["kv_layer"]].view(H16).view(m.dec_layers, 2, HEADS, pad, HD)
    tri16, vn16 = (state[lay[k]:lay[k] + N * 18].view(H16) for k in ("tri_off", "vn_off"))
    vtri, vvn = torch.empty(N * 9, device="cuda", dtype=H16), torch.empty(N * 9, device="cuda", dtype=H16)
    vpos, kc = torch.empty(pad * 9, device="cuda", dtype=H16), torch.empty(pad, HD, device="cuda", dtype=H16)
    ks = torch.empty_like(kc)
    ops.view_geometry(torch.from_numpy(np.asarray(c2w[0], dtype=np.float32)).reshape(16).cuda(), tri16, vn16,
                      state[lay["c_off"]:lay["c_off"] + 12].view(torch.float32), m.t["vt_rope_freqs"], vtri, vvn, vpos, kc, ks, N,
                      m.num_register_tokens, pad, m.rope_num_freqs, HD)
    pat = torch.empty(P * P, 192, device="cuda", dtype=H16)
    ops.ray_gen_patchify(torch.eye(4, device="cuda").reshape(16).contiguous(), torch.tensor([float(fov[0])], device="cuda"), None,
                         pat, 1, RES, 8)
    x = pat.double() @ m.t["ray_enc_w"].double().t() + m.t["ray_enc_b"].double()
    x = TL.rms(x, m.t["ray_enc_norm"].double()) + m.t["ray_map_patch_token"].double()
    for i in range(m.dec_layers):
        x = TL.decoder_layer(x, TL.layer_weights(m, i), kv[i, 0, :, :Se], kv[i, 1, :, :Se], kc[:Se], ks[:Se], RP.shift_mask(P, 8, 4),
                             4 if i % 2 else 0, HEADS, P, P, 8, dtype=torch.float64)
    s.close()
    return got.view_as(x), x


@pytest.mark.parametrize("gemm_path,attention_path", [(0, 0), (2, 0), (1, 0), (3, 0), (0, 1), (0, 2)])
@pytest.mark.parametrize("with_dpt", [False, True], ids=["token_map", "image"])
def test_token_map_against_fp64(with_dpt, gemm_path, attention_path):
    ops.gemm_set_path(gemm_path)
    ops.flash_attention_set_path(attention_path)
    mean, largest = TL.err_stats(*_render(with_dpt))
    print(f"mean {mean:.2e} largest {largest:.2e}")
    assert mean < 9.6e-4 and largest < 1.6e-2, (mean, largest)


def test_images_keep_the_mma_attention():
    """The token map under an image head has the bits of the mma.sync kernel whatever is set; without one it has not."""
    image, tokens = _render(True)[0], _render(False)[0]
    ops.flash_attention_set_path(1)
    assert torch.equal(image, _render(True)[0])
    assert not torch.equal(image, tokens)
