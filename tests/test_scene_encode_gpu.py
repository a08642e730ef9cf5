"""Scene encoding: the geometry kernels (fp16 copies, centre) at sizes around a thread's stride, and a session that encodes
several scenes with its one block of work buffers. Oracle: fp16 casts and a double-precision mean on the host, exact - every
partial sum of the fp16 vertices is exact in double precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scene(n, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    tri = ((torch.rand(n, 3, 3, device="cuda", generator=g) * 2 - 1) * scale).contiguous()
    vn = torch.nn.functional.normalize(torch.randn(n, 3, 3, device="cuda", generator=g), dim=-1).contiguous()
    return tri, vn, torch.rand(n, 13, device="cuda", generator=g).half().contiguous()


def _session(n, heads=4, dim=256):
    import renderformer_cuda_b200  # noqa: F401
    from renderformer_cuda_b200 import session
    model = session.Model.random(seed=2, dim=dim, num_heads=heads, ffn_hidden=2 * dim, enc_layers=1, dec_layers=1,
                                 num_register_tokens=5)
    return session.RenderSession(model, n, 64)


def _geometry(s, n):
    """(fp16 triangles, fp16 normals, fp32 centre): the last three pieces of the scene state, 256-byte aligned each."""
    up = lambda v: (v + 255) // 256 * 256
    raw = s.scene_state.cpu().numpy().view(np.uint8)
    size = up(n * 18)
    start = raw.size - 256 - 2 * size
    f16 = lambda o: raw[o:o + n * 18].view(np.float16).reshape(n * 3, 3)
    return f16(start), f16(start + size), raw[start + 2 * size:start + 2 * size + 12].view(np.float32)


@pytest.mark.parametrize("n,scale", [(1, 1.0), (113, 1.0), (114, 300.0), (341, 1.0), (1365, 0.01), (5633, 20.0)])
def test_geometry_of_the_scene_state(n, scale):
    s = _session(n)
    tri, vn, tex = _scene(n, n, scale)
    s.encode_scene(tri, vn, tex)
    t16, v16, centre = _geometry(s, n)
    want = tri.half().cpu().numpy().reshape(n * 3, 3)
    assert np.array_equal(t16.view(np.uint16), want.view(np.uint16))
    assert np.array_equal(v16.view(np.uint16), vn.half().cpu().numpy().reshape(n * 3, 3).view(np.uint16))
    assert np.array_equal(centre, (want.astype(np.float64).sum(0) / (3.0 * n)).astype(np.float32))
    s.close()


@pytest.mark.parametrize("heads", [4, 2, 8])
def test_a_session_encodes_scene_after_scene(heads):
    """64-, 128- and 32-wide heads (the last with a materialised score matrix among the work buffers)."""
    n = 61
    a, b = _session(n, heads), _session(n, heads)
    first, second = _scene(n, 1), _scene(n, 2)
    a.encode_scene(*first)
    one = a.scene_state.clone()
    a.encode_scene(*second)
    assert not torch.equal(a.scene_state, one)
    b.encode_scene(*second)
    assert torch.equal(a.scene_state, b.scene_state)
    a.encode_scene(*first)
    assert torch.equal(a.scene_state, one)
    kv = one[:2 * 72 * 256 * 2].view(torch.float16).view(2, heads, 72, 256 // heads)
    assert torch.isfinite(kv).all() and (kv[:, :, 66:] == 0).all() and (kv[:, :, :66] != 0).any(-1).all()
    a.close(); b.close()


@pytest.mark.parametrize("Sk,heads,hd,kv_dim", [(1, 4, 64, 256), (33, 2, 128, 256), (120, 4, 64, 72), (333, 16, 64, 1024), (4700, 4, 64, 256)])
def test_values_of_the_cache_are_the_plain_projection_head_split(Sk, heads, hd, kv_dim):
    """V stored head-split by its projection, with pad rows behind each head: the plain product transposed, bit for bit,
    on small and on large tiles, and zeros behind it."""
    import ctypes
    import renderformer_cuda_b200 as pkg
    from renderformer_cuda_b200 import _abi, session
    L, VP = _abi.load("rfk_layers.h"), ctypes.c_void_p
    dim, pad = heads * hd, (Sk + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(Sk)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
    model = session.Model.random(seed=1, dim=dim, num_heads=heads, ffn_hidden=256, enc_layers=0, dec_layers=1)
    w = model.decoder_record(0).cross_attn
    x, wv, wk = rnd(Sk, kv_dim), rnd(dim, kv_dim), rnd(dim, kv_dim)
    w.v_proj_w, w.k_proj_w = wv.data_ptr(), wk.data_ptr()
    K, V = (torch.full((heads, pad, hd), 7.0, device="cuda", dtype=torch.float16) for _ in range(2))
    proj, want = torch.empty(2 * Sk, dim, device="cuda", dtype=torch.float16), torch.empty(Sk, dim, device="cuda", dtype=torch.float16)
    ctx = session.Ctx()
    rc = L.rfk_precompute_cross_kv(ctx.h, ctypes.byref(w), VP(x.data_ptr()), VP(K.data_ptr()), VP(V.data_ptr()), VP(proj.data_ptr()),
                                   1, Sk, pad, kv_dim, dim, heads, VP(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, rc
    pkg.ops.gemm_f16(x, wv, want, Sk, dim, kv_dim)
    torch.cuda.synchronize()
    assert torch.equal(V[:, :Sk], want.view(Sk, heads, hd).permute(1, 0, 2))
    assert (V[:, Sk:] == 0).all() and (K[:, Sk:] == 0).all() and torch.isfinite(K.float()).all()
    ctx.close()


@pytest.mark.parametrize("with_dpt", [True, False])
def test_cut_of_the_last_round_and_images(with_dpt):
    """2500 triangles and 16 heads are 160 units of attention work on 148 SMs: a session that ends at the token map cuts the
    last round's along the keys, one with an image head does not, so that its images stay what they were."""
    import renderformer_cuda_b200 as pkg
    from renderformer_cuda_b200 import session
    n = 2500
    model = session.Model.random(seed=2, dim=1024, num_heads=16, ffn_hidden=256, enc_layers=1, dec_layers=1, with_dpt=with_dpt,
                                 dpt_features=64, dpt_out_channels=(32, 64, 128, 128))
    s = session.RenderSession(model, n, 64)
    states = []
    try:
        for split in (1, 0):
            pkg.ops.flash_attention_set_split(split)
            s.encode_scene(*_scene(n, 3))
            states.append(s.scene_state.clone())
    finally:
        pkg.ops.flash_attention_set_split(1)
    assert torch.equal(*states) == with_dpt
    s.close()


@pytest.mark.parametrize("S,heads,hd", [(1, 4, 64), (33, 4, 64), (300, 2, 128), (1100, 16, 64), (4700, 4, 64), (333, 16, 64), (1, 8, 128),
                                        (77, 16, 128), (512, 20, 64), pytest.param(64, 8, 32, id="packed_both_times-64-8-32")])
@pytest.mark.parametrize("rope", [True, False])
def test_head_split_projection_has_the_bits_of_the_separate_epilogue(S, heads, hd, rope):
    """Self-attention of one batch element: q, k, v stored head-split by their projection, q and k normalised and rotated in
    place, against the packed projection and its epilogue kernel, which a projection with a bias (here of zeros) takes."""
    import ctypes
    from renderformer_cuda_b200 import _abi, session
    L, VP = _abi.load("rfk_layers.h"), ctypes.c_void_p
    dim = heads * hd
    g = torch.Generator(device="cuda").manual_seed(S + hd)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, wi, wo = rnd(S, dim).half(), (rnd(3 * dim, dim) / dim ** 0.5).half(), (rnd(dim, dim) / dim ** 0.5).half()
    gq, gk = 1 + 0.1 * rnd(dim), 1 + 0.1 * rnd(dim)
    ang = rnd(S, hd // 2)
    cos, sin = (torch.cat([f(ang)] * 2, -1).half().contiguous() for f in (torch.cos, torch.sin))
    zero = torch.zeros(3 * dim, device="cuda", dtype=torch.float16)
    ctx, outs = session.Ctx(), []
    score = torch.empty(heads * S * ((S + 7) // 8 * 8), device="cuda") if hd == 32 else None
    for bias in (None, zero):
        w = session.MhaW(wi.data_ptr(), None if bias is None else bias.data_ptr(), wo.data_ptr(), None, gq.data_ptr(), gk.data_ptr())
        out = torch.full((S, dim), 7.0, device="cuda", dtype=torch.float16)
        buf = torch.full((6 * S * dim,), 7.0, device="cuda", dtype=torch.float16)
        rc = L.rfk_self_attention(ctx.h, ctypes.byref(w), VP(x.data_ptr()), VP(out.data_ptr()), VP(buf.data_ptr()),
                                  VP(score.data_ptr() if score is not None else 0), 1, S, dim, heads,
                                  VP(cos.data_ptr() if rope else 0), VP(sin.data_ptr() if rope else 0),
                                  VP(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, rc
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.isfinite(outs[0].float()).all() and torch.equal(*outs)
    ctx.close()


@pytest.mark.parametrize("dim", [8, 256, 264, 512, 768, 1024])
@pytest.mark.parametrize("rows", [1, 5, 300])
def test_embedding_norms_and_sum_have_the_bits_of_the_separate_steps(rows, dim):
    import ctypes
    import renderformer_cuda_b200 as pkg
    from renderformer_cuda_b200 import _abi
    ops, VP = pkg.ops, ctypes.c_void_p
    g = torch.Generator(device="cuda").manual_seed(rows + dim)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, b, c, ga, gb = rnd(rows, dim).half(), rnd(rows, dim).half(), rnd(dim).half(), 1 + 0.1 * rnd(dim), 1 + 0.1 * rnd(dim)
    norms = []
    for x, gamma in ((a, ga), (b, gb)):
        f = torch.empty(rows, dim, device="cuda")
        ops.cast_fp16_to_fp32(x, f, rows * dim)
        ops.rmsnorm_f32(f, gamma, f, rows, dim, ops.K_EPS_FP16)
        norms.append(f)
    want, got = (norms[0] + norms[1]) + c.float(), torch.empty(rows, dim, device="cuda")
    fn = _abi.load("rfk.h").rfk_norm_pair_add
    fn.argtypes, fn.restype = [VP] * 6 + [ctypes.c_int] * 2 + [ctypes.c_float, VP], ctypes.c_int
    assert fn(*(VP(t.data_ptr()) for t in (a, ga, b, gb, c, got)), rows, dim, ops.K_EPS_FP16,
              VP(torch.cuda.current_stream().cuda_stream)) == 0
    assert torch.equal(got, want)


# on CTA pairs with tiles of 192 columns: 1.2 and 1.9 rounds of 74 pairs, and less than one, with rows that fill neither a tile nor a store box
@pytest.mark.parametrize("Sk,heads,hd,pad", [(5665, 8, 128, 5672), (5665, 16, 64, 5672), (2501, 8, 128, 2504), (2501, 8, 128, 2600), (4100, 8, 64, 4104)])
def test_cache_of_large_scenes_has_the_bits_of_the_separate_epilogue(Sk, heads, hd, pad):
    """V stored head-split by its projection against the plain projection and its epilogue kernel, which a projection with a bias (here of
    zeros) takes; K's norm with and without one."""
    import ctypes
    from renderformer_cuda_b200 import _abi, session
    L, VP = _abi.load("rfk_layers.h"), ctypes.c_void_p
    dim = heads * hd
    g = torch.Generator(device="cuda").manual_seed(Sk + hd)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, wk, wv = rnd(Sk, dim).half(), (rnd(dim, dim) / dim ** 0.5).half(), (rnd(dim, dim) / dim ** 0.5).half()
    zero = torch.zeros(dim, device="cuda", dtype=torch.float16)
    model = session.Model.random(seed=1, dim=dim, num_heads=heads, ffn_hidden=256, enc_layers=0, dec_layers=1)
    w = model.decoder_record(0).cross_attn
    w.k_proj_w, w.v_proj_w = wk.data_ptr(), wv.data_ptr()
    ctx, outs = session.Ctx(), []
    for bias in (None, zero):
        w.k_proj_b = w.v_proj_b = None if bias is None else bias.data_ptr()
        K, V = (torch.full((heads, pad, hd), 7.0, device="cuda", dtype=torch.float16) for _ in range(2))
        proj = torch.full((2 * Sk, dim), 7.0, device="cuda", dtype=torch.float16)
        rc = L.rfk_precompute_cross_kv(ctx.h, ctypes.byref(w), VP(x.data_ptr()), VP(K.data_ptr()), VP(V.data_ptr()), VP(proj.data_ptr()),
                                       1, Sk, pad, dim, dim, heads, VP(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, rc
        torch.cuda.synchronize()
        outs.append((K, V, bool((proj[Sk:] != 7.0).any())))
    assert not outs[0][2] and outs[1][2]                # V's two routes
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert (outs[0][0][:, Sk:] == 0).all() and torch.isfinite(outs[0][0].float()).all() and (outs[0][0][:, :Sk] != 0).any(-1).all()
    ctx.close()
