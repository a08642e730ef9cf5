"""Products whose norms are folded into them: rows scaled by their sums of squares, sums written beside the output, rows put in the order of
another shift or in raster order - on small tiles and CTA pairs, against fp32 torch on the same fp16 operands."""
import ctypes

import pytest
import torch

from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -10


class Product(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("A", "W", "W_up", "R", "C", "raster")] + [(n, ctypes.c_int) for n in ("M", "N", "K")] + [
        ("in_ss", ctypes.c_void_p), ("in_tiles", ctypes.c_int), ("in_mul", ctypes.c_float), ("eps", ctypes.c_float), ("out_ss", ctypes.c_void_p),
        ("ss_mask", ctypes.c_int), ("part_stride", ctypes.c_longlong)] + [
        (n, ctypes.c_int) for n in ("seq", "num_heads", "head_dim", "out_seq", "blocks_across", "blocks_down", "shift_from", "shift_to", "quarters")]


class More(ctypes.Structure):
    _fields_ = [("pairs", ctypes.c_int), ("w_mul", ctypes.c_void_p), ("w_up_mul", ctypes.c_void_p)]


def _run(path=0, w_mul=None, **kw):
    lib = _abi.load("rfk.h")
    f, more = Product(), More(w_mul=w_mul.data_ptr() if w_mul is not None else None)
    f.eps = EPS
    for k, v in kw.items():
        setattr(f, k, v.data_ptr() if torch.is_tensor(v) else v)
    tiles = ctypes.c_int()
    assert lib.rfk_gemm_set_path(path) == 0
    try:
        rc = lib.rfk_gemm_folded_more(ctypes.byref(f), ctypes.byref(more), ctypes.byref(tiles), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    finally:
        lib.rfk_gemm_set_path(0)
    assert rc == 0
    code = ctypes.c_int()
    assert lib.rfk_gemm_error(ctypes.byref(code), 0) == 0 and code.value == 0
    return tiles.value


def _gen(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).half()


def _near(got, want, terms):
    # the output's rounding (2^-11 of the value), and fp32 sums of `terms` products in another order
    tol = want.abs() * 2.0 ** -10 + 2.0 ** -24 * 8 * terms ** 0.5 * want.square().mean().sqrt() + 1e-6
    assert ((got.float() - want).abs() <= tol).all(), float(((got.float() - want).abs() / tol).max())


def _factor(x, mul):
    return mul * torch.rsqrt(x.float().square().mean(-1, keepdim=True) + EPS)


def _check_sums(ss, tiles, x, parts=1):
    """ss [parts][M][tiles] against the squares of x [M, parts * dim]."""
    dim = x.shape[1] // parts
    got = ss.flatten()[: parts * x.shape[0] * tiles].view(parts, x.shape[0], tiles)
    assert tiles in (dim // 256, dim // 32)
    want = x.float().square().view(x.shape[0], parts, tiles, -1).sum(-1).permute(1, 0, 2)
    assert torch.allclose(got, want, rtol=2e-5, atol=1e-6)


# 64 rows: 64 x 32 tiles; 1024: 128 x 64; 2304: 128 x 128; 3136 and 5632: pairs of 192 and 256 columns; 4160: a tail of rows
@pytest.mark.parametrize("M", [64, 256, 1024, 2304, 3136, 4096, 4160, 5632])
@pytest.mark.parametrize("groups", [1, 8])
def test_gate_of_scaled_rows(M, groups):
    rnd = _gen(M)
    K, N = 256, 512
    x, w, u = rnd(M, K), rnd(N, K, scale=K ** -0.5), rnd(N, K, scale=K ** -0.5)
    tiles = K // 256 if groups == 1 else K // 32
    ss = x.float().square().view(M, tiles, -1).sum(-1).contiguous()
    out = torch.empty(M, N, device="cuda", dtype=torch.half)
    _run(A=x, W=w, W_up=u, C=out, M=M, N=N, K=K, in_ss=ss, in_tiles=tiles, in_mul=2.0)
    f = _factor(x, 2.0)
    a, b = (x.float() @ w.float().t()) * f, (x.float() @ u.float().t()) * f
    want = torch.nn.functional.silu(a) * b
    # the gate's exponential and reciprocal are approximate (2^-22 each), so is the factor's square root; a and b are fp32 sums whose rounding
    # (some 1e-6 of their terms) the other one multiplies
    tol = want.abs() * 2.0 ** -10 + 1e-5 * (1 + a.abs()) * (1 + b.abs())
    assert ((out.float() - want).abs() <= tol).all()


@pytest.mark.parametrize("M,seq,parts,hd", [(64, 64, 1, 64), (256, 256, 1, 64), (256, 64, 3, 64), (1024, 512, 1, 128), (2304, 64, 3, 128), (3136, 3136, 1, 64),
                                            (4096, 4096, 1, 128), (4160, 64, 3, 64)])
@pytest.mark.parametrize("path", [0, 2])
def test_heads_of_scaled_rows_with_sums(M, seq, parts, hd, path):
    rnd = _gen(M + parts)
    K, dim = 512, 512
    heads, N = dim // hd, parts * dim
    x, w = rnd(M, K), rnd(N, K, scale=K ** -0.5)
    ss = x.float().square().view(M, K // 256, -1).sum(-1).contiguous()
    out = torch.full((parts, M // seq, heads, seq, hd), float("nan"), device="cuda", dtype=torch.half)
    sums = torch.full((parts * M * dim // 32,), float("nan"), device="cuda")
    tiles = _run(path, A=x, W=w, C=out, M=M, N=N, K=K, in_ss=ss, in_tiles=K // 256, in_mul=1.0, out_ss=sums, ss_mask=(1 << parts) - 1,
                 part_stride=M * dim, seq=seq, num_heads=heads, head_dim=hd)
    got = out.permute(1, 3, 0, 2, 4).reshape(M, N)
    _near(got, (x.float() @ w.float().t()) * _factor(x, 1.0), K)
    _check_sums(sums, tiles, got, parts)


def _to_blocks(grid, shift):
    """[views, H, W, dim] -> rows: the 4 x 4 blocks in window order of the grid shifted by `shift` tokens."""
    v, h, w, d = grid.shape
    g = torch.roll(grid, (shift, shift), (1, 2)).view(v, h // 8, 2, 4, w // 8, 2, 4, d)
    return g.permute(0, 1, 4, 2, 5, 3, 6, 7).reshape(v * h * w, d).contiguous()


@pytest.mark.parametrize("views,h,w", [(1, 8, 8), (1, 16, 16), (2, 24, 16), (1, 40, 48), (1, 64, 64), (4, 32, 40)])
@pytest.mark.parametrize("src,dst", [(0, 4), (4, 0), (0, 0)])
@pytest.mark.parametrize("path", [0, 2])
def test_residual_rows_go_to_another_shift_and_to_raster(views, h, w, src, dst, path):
    rnd = _gen(h * w + src)
    N, K = 256, 512
    grid = rnd(views, h, w, N)
    M = views * h * w
    r, a, wt = _to_blocks(grid, src), rnd(M, K), rnd(N, K, scale=K ** -0.5)
    out, raster = (torch.full((M, N), float("nan"), device="cuda", dtype=torch.half) for _ in range(2))
    sums = torch.full((M * N // 32,), float("nan"), device="cuda")
    args = dict(A=a, W=wt, R=r, M=M, N=N, K=K, blocks_across=w // 4, blocks_down=h // 4, shift_from=src // 4, shift_to=dst // 4)
    tiles = _run(path, C=out, raster=raster, out_ss=sums, **args)
    plain = torch.empty(M, N, device="cuda", dtype=torch.half)
    _run(path, A=a, W=wt, R=r, C=plain, M=M, N=N, K=K)
    _near(plain, r.float() + a.float() @ wt.float().t(), K)
    # the same bits, elsewhere
    back = _to_blocks(torch.arange(M, device="cuda", dtype=torch.float32).view(views, h, w, 1), src).long().flatten()   # raster row of each row
    assert torch.equal(raster[back], plain)
    assert torch.equal(out, _to_blocks(raster.view(views, h, w, N), dst))
    _check_sums(sums, tiles, out)
    alone = torch.empty_like(raster)
    _run(path, C=None, raster=alone, **args)
    assert torch.equal(alone, raster)


def test_sums_have_the_same_bits_from_small_tiles_and_pairs():
    rnd = _gen(5)
    M, N, K = 1024, 1024, 512
    a, w, r = rnd(M, K), rnd(N, K, scale=K ** -0.5), rnd(M, N)
    res = []
    for path in (0, 2):
        out, sums = torch.empty(M, N, device="cuda", dtype=torch.half), torch.empty(M * N // 32, device="cuda")
        tiles = _run(path, A=a, W=w, R=r, C=out, M=M, N=N, K=K, out_ss=sums)
        s = sums[: M * tiles].view(M, tiles)
        if tiles == N // 32:      # eight in order make 256 columns
            t = s.view(M, N // 256, 8)
            s = t[..., 0].clone()
            for i in range(1, 8):
                s += t[..., i]
        res.append((out, s))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("views,h,w", [(1, 8, 8), (2, 24, 16), (1, 40, 48), (4, 64, 64)])
def test_tokens_that_enter_folded_layers(views, h, w):
    from renderformer_cuda_b200 import ops
    rnd = _gen(h + w)
    M, N = views * h * w, 1024
    rows, norm, token = rnd(M, N), 1 + 0.1 * rnd(N).float(), rnd(N)
    x, ss = torch.empty(M, N, device="cuda", dtype=torch.half), torch.empty(M, 4, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert _abi.load("rfk.h").rfk_embed_tokens(p(rows), p(norm), p(token), p(x), p(ss), M, N, ctypes.c_float(EPS), w // 4, h // 4,
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = rows.clone()
    ops.rmsnorm(want, norm, want, M, N)
    ops.broadcast_add(want, token, want.numel(), N)
    assert torch.equal(x, _to_blocks(want.view(views, h, w, N), 0))
    _check_sums(ss, 4, x)


def _fold(weights, gammas):
    """rfk_fold_weights of matrices [rows][1024]: the folded rows and what each 64 of them were divided by."""
    n, rows = len(weights), sum(w.shape[0] for w in weights)
    out, mul = torch.empty(rows, 1024, device="cuda", dtype=torch.half), torch.full((rows // 64,), float("nan"), device="cuda")
    table = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])
    rc = _abi.load("rfk.h").rfk_fold_weights(table(weights), table(gammas), (ctypes.c_int * n)(*[w.shape[0] for w in weights]), n, 1024,
                                             ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(mul.data_ptr()),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return out, mul


@pytest.mark.parametrize("rows", [(64,), (1024, 3072, 256, 256), (64, 192) * 32])
def test_folded_weights(rows):
    rnd = _gen(len(rows))
    w = [rnd(r, 1024) for r in rows]
    gamma = [rnd(1024).float() * 2.0 ** (3 * (i % 9) - 12) for i in range(len(rows))]
    out, mul = _fold(w, gamma)
    assert (mul.log2() == mul.log2().round()).all()
    product = torch.cat([a.float() * g for a, g in zip(w, gamma)])
    largest = (product.abs().view(-1, 64 * 1024).amax(1) / mul).log2()
    assert (largest >= 13).all() and (largest <= 14).all()
    assert torch.equal(out, (product / mul.repeat_interleave(64)[:, None]).half())


@pytest.mark.parametrize("spread", [0.0, 1.0, 1.5, 2.0, "half"])
@pytest.mark.parametrize("M", [64, 512, 4096])
def test_norm_weights_that_hold_down_large_channels(M, spread):
    """Weight x norm weight keeps the bits of an fp16 value however far norm weights lie apart. Each product has one operand rounded (2^-11 of it at most,
    2^-11 / sqrt 3 in the mean of squares, for a mantissa anywhere in its binade less), and so has the result: 4e-4 of the result's norm."""
    g = torch.Generator(device="cuda").manual_seed(M)
    n = lambda *s: torch.randn(*s, device="cuda", generator=g)
    N = K = 1024
    gamma = torch.where(torch.arange(K, device="cuda") % 2 == 0, 1.0, 0.001) if spread == "half" else torch.exp(spread * n(K))
    w, x = (0.02 * n(N, K)).half(), (n(M, K) / gamma).half()
    f, mul = _fold([w], [gamma])
    ss = x.float().square().view(M, 4, -1).sum(-1).contiguous()
    out = torch.empty(1, 16, M, 64, device="cuda", dtype=torch.half)
    _run(A=x, W=f, C=out, M=M, N=N, K=K, in_ss=ss, in_tiles=4, in_mul=1.0, part_stride=M * N, seq=M, num_heads=16, head_dim=64, w_mul=mul)
    xd = x.double()
    want = (xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + EPS) * gamma.double()) @ w.double().t()
    got = out[0].permute(1, 0, 2).reshape(M, N).double()
    assert (got - want).norm() <= 4e-4 * want.norm()


def _scene(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    tri = (torch.rand(n, 3, 3, device="cuda", generator=g) * 2 - 1).contiguous()
    vn = torch.nn.functional.normalize(torch.randn(n, 3, 3, device="cuda", generator=g), dim=-1).contiguous()
    return tri, vn, torch.rand(n, 13, device="cuda", generator=g).half()


def _view(model, scene, res, path=0, **kw):
    from renderformer_cuda_b200 import session
    c2w = torch.eye(4)
    c2w[2, 3] = 3.0
    s = session.RenderSession(model, scene[0].shape[0], res, **kw)
    s.encode_scene(*scene)
    lib = _abi.load("rfk.h")
    try:
        lib.rfk_gemm_set_path(path)
        s.finalize()
        s.render_frame(c2w, 0.7)
        return s, s.download()
    finally:
        lib.rfk_gemm_set_path(0)


@pytest.mark.parametrize("heads,res", [(16, 64), (8, 128), (16, 192)])
@pytest.mark.parametrize("weights", [1.0, 2.0 ** -6, 37.0])
def test_views_of_folded_and_separate_norms_agree(heads, res, weights):
    """1024-wide rows, norm weights of several magnitudes: the folded layers, and with them switched off (the library's products). Twelve roundings
    of 2^-11 and sums in other orders a layer apart."""
    from renderformer_cuda_b200 import session
    model = session.Model.random(seed=3, dim=1024, num_heads=heads, ffn_hidden=512, enc_layers=1, dec_layers=4)
    for i in range(4):
        for k in ("query_norm", "self_attn_norm", "ffn_norm"):
            model.t[f"dec{i}.{k}"].mul_(weights)
    scene = _scene(60, res)
    s, got = _view(model, scene, res)
    few = s.kernels_per_view
    s.close()
    s, want = _view(model, scene, res, path=1)
    assert s.kernels_per_view != few
    s.close()
    assert torch.isfinite(got.float()).all()
    assert (got.float() - want.float()).norm() <= 3e-3 * want.float().norm()


def test_weights_changed_in_place_count_from_the_next_encoding():
    from renderformer_cuda_b200 import session
    model = session.Model.random(seed=3, dim=1024, num_heads=16, ffn_hidden=512, enc_layers=1, dec_layers=2)
    scene = _scene(60, 1)
    s, before = _view(model, scene, 64)
    other = session.Model.random(seed=4, dim=1024, num_heads=16, ffn_hidden=512, enc_layers=1, dec_layers=2)
    for k, t in model.t.items():   # all but the query norms of the cross-attention, which a session takes over when it is made
        if k.endswith("cq_norm"):
            other.t[k].copy_(t)
        else:
            t.copy_(other.t[k])
    s.encode_scene(*scene)
    c2w = torch.eye(4)
    c2w[2, 3] = 3.0
    s.render_frame(c2w, 0.7)
    got = s.download().clone()
    s.close()
    f, want = _view(other, scene, 64)
    f.close()
    assert not torch.equal(before, want) and torch.equal(got, want)


@pytest.mark.parametrize("heads,res,use_graph", [(16, 64, True), (8, 128, True), (16, 192, True), (16, 64, False)])
def test_norm_weights_changed_across_powers_of_two(heads, res, use_graph):
    """The scales that are taken out of the weights are not part of a captured view: norm weights 8, 1/16 and 37 times as large."""
    from renderformer_cuda_b200 import session
    model = session.Model.random(seed=3, dim=1024, num_heads=heads, ffn_hidden=512, enc_layers=1, dec_layers=2)
    scene = _scene(60, 1)
    s, before = _view(model, scene, res, use_graph=use_graph)
    before = before.clone()
    for i in range(2):
        for k, by in (("query_norm", 8.0), ("self_attn_norm", 1 / 16), ("ffn_norm", 37.0)):
            model.t[f"dec{i}.{k}"].mul_(by)
    s.encode_scene(*scene)
    c2w = torch.eye(4)
    c2w[2, 3] = 3.0
    s.render_frame(c2w, 0.7)
    got = s.download().clone()
    s.close()
    f, want = _view(model, scene, res, use_graph=use_graph)
    f.close()
    assert not torch.equal(before, want) and torch.equal(got, want)


def test_sessions_fit_where_they_fit_without_folded_weights():
    """150 MB less than a session takes are left, of which 302 MB are folded weights: it keeps separate norms, and renders."""
    from renderformer_cuda_b200 import session
    model = session.Model.random(seed=3, dim=1024, num_heads=16, ffn_hidden=4096, enc_layers=1, dec_layers=12)
    scene, mb = _scene(60, 1), 1 << 20
    free = lambda: torch.cuda.mem_get_info()[0]
    torch.cuda.empty_cache()
    s, want = _view(model, scene, 64)     # whatever is loaded and kept once, and how much a session takes
    few, want = s.kernels_per_view, want.clone()
    with_all = free()
    s.close()
    took = free() - with_all
    assert took > 450 * mb
    taken = torch.empty(free() - took + 150 * mb, dtype=torch.uint8, device="cuda")
    s, got = _view(model, scene, 64)
    assert s.kernels_per_view > few
    s.close()
    del taken
    torch.cuda.empty_cache()
    assert (got.float() - want.float()).norm() <= 3e-3 * want.float().norm()


@pytest.mark.parametrize("views_per_frame", [1, 2])
def test_every_session_of_a_scheduler_takes_changed_weights(views_per_frame):
    """Two sessions share the scene state that one of them encodes; after load_scene both render with the weights as they are then."""
    from renderformer_cuda_b200 import session
    dims = dict(dim=1024, num_heads=16, ffn_hidden=512, enc_layers=1, dec_layers=2)
    model, other = (session.Model.random(seed=k, **dims) for k in (3, 4))
    scene, n = _scene(60, 1), 4 * views_per_frame
    c2w = torch.eye(4).repeat(n, 1, 1)
    c2w[:, 2, 3] = 3.0 + 0.1 * torch.arange(n)
    fov, out = torch.full((n,), 0.7), torch.empty(n, 64, 1024, dtype=torch.half).pin_memory()
    def render(s):
        assert s.render(c2w, fov, out) == list(range(n))
        return out.clone()
    new = lambda m: session.ViewScheduler(m, 60, 64, streams_per_gpu=2, views_per_frame=views_per_frame)
    s = new(model)
    s.load_scene(*scene)
    before = render(s)
    for k, t in model.t.items():   # all but the query norms of the cross-attention, which a session takes over when it is made
        if k.endswith("cq_norm"):
            other.t[k].copy_(t)
        else:
            t.copy_(other.t[k])
    s.load_scene(*scene)
    got = render(s)
    s.close()
    f = new(other)
    f.load_scene(*scene)
    want = render(f)
    f.close()
    for v in range(n):
        assert not torch.equal(before[v], want[v]) and torch.equal(got[v], want[v]), v


@pytest.mark.parametrize("M,pad,parts,hd", [(1, 8, 4, 64), (333, 336, 24, 128), (777, 784, 6, 64), (2665, 2672, 8, 64)])
@pytest.mark.parametrize("path", [0, 2])
def test_parts_with_factors_of_their_own_and_room_behind_the_rows(M, pad, parts, hd, path):
    """The keys and values of several layers: any number of rows, heads with room for more, each part its own factor, sums for every other one."""
    rnd = _gen(M)
    K = dim = 1024
    heads, N = dim // hd, parts * dim
    x, w = rnd(M, K), rnd(N, K, scale=K ** -0.5)
    ss = x.float().square().view(M, 4, -1).sum(-1).contiguous()
    mul = 2.0 ** -(torch.arange(parts, device="cuda") % 5).float()
    out = torch.full((parts, heads, pad, hd), 7.0, device="cuda", dtype=torch.half)
    sums = torch.full((parts * M * dim // 32,), float("nan"), device="cuda")
    tiles = _run(path, A=x, W=w, C=out, M=M, N=N, K=K, in_ss=ss, in_tiles=4, in_mul=1.0, out_ss=sums, ss_mask=0x55555555, part_stride=dim * pad, seq=M,
                 num_heads=heads, head_dim=hd, out_seq=pad, w_mul=mul.repeat_interleave(dim // 64))
    assert (out[:, :, M:] == 7.0).all()
    got = out[:, :, :M].permute(2, 0, 1, 3).reshape(M, N)
    factor = _factor(x, 1.0)
    for i in range(parts):
        cols = slice(i * dim, (i + 1) * dim)
        _near(got[:, cols], (x.float() @ w[cols].float().t()) * factor * mul[i], K)
    s = sums[: parts * M * tiles].view(parts, M, tiles)
    assert s[1::2].isnan().all()
    want = got.float().square().view(M, parts, tiles, -1).sum(-1).permute(1, 0, 2)
    assert torch.allclose(s[0::2], want[0::2], rtol=2e-5, atol=1e-6)


@pytest.mark.parametrize("M,parts", [(256, 3), (3136, 3), (4096, 2)])
def test_factors_of_parts_without_sums(M, parts):
    """3136 rows: pair tiles of 192 columns, which cross from one part of 512 into the next."""
    lib = _abi.load("rfk.h")
    assert M != 3136 or lib.rfk_gemm_pair_tile(M, parts * 512, 74) == 192
    rnd = _gen(M + parts)
    K, dim, hd = 512, 512, 64
    x, w = rnd(M, K), rnd(parts * dim, K, scale=K ** -0.5)
    ss = x.float().square().view(M, K // 256, -1).sum(-1).contiguous()
    mul = 2.0 ** (3 * torch.arange(parts, device="cuda")).float()
    out = torch.full((parts, 1, dim // hd, M, hd), float("nan"), device="cuda", dtype=torch.half)
    _run(A=x, W=w, C=out, M=M, N=parts * dim, K=K, in_ss=ss, in_tiles=K // 256, in_mul=1.0, part_stride=M * dim, seq=M, num_heads=dim // hd, head_dim=hd,
         w_mul=mul.repeat_interleave(dim // 64))
    got, factor = out.permute(1, 3, 0, 2, 4).reshape(M, parts * dim), _factor(x, 1.0)
    for i in range(parts):
        cols = slice(i * dim, (i + 1) * dim)
        _near(got[:, cols], (x.float() @ w[cols].float().t()) * factor * mul[i], K)


# both sides of the line, which is 148 tiles of 128 x 128 on 148 SMs: 1 layer of keys and values, 3, 9 and 12
@pytest.mark.parametrize("M,parts,small", [(92, 6, True), (1152, 2, True), (1153, 2, False), (128, 18, True), (129, 18, False), (33, 24, False)])
def test_sums_of_256_columns_or_nothing(M, parts, small):
    """Whoever has room for one sum each 256 columns asks for pairs: small tiles, which write eight times as many, are refused before anything is written."""
    lib = _abi.load("rfk.h")
    assert lib.rfk_folded_on_pairs(M, parts * 1024) == (not small)
    rnd = _gen(M)
    K = dim = 1024
    x, w = rnd(M, K), rnd(parts * dim, K, scale=K ** -0.5)
    ss = x.float().square().view(M, 4, -1).sum(-1).contiguous()
    out = torch.full((parts, 16, M, 64), 7.0, device="cuda", dtype=torch.half)
    sums, n = torch.full((2 * parts * M * 4,), -1.0, device="cuda"), parts * M * 4
    f, more, tiles = Product(), More(pairs=1), ctypes.c_int()
    for k, v in dict(A=x, W=w, C=out, M=M, N=parts * dim, K=K, in_ss=ss, in_tiles=4, in_mul=1.0, eps=EPS, out_ss=sums, ss_mask=0x55555555,
                     part_stride=dim * M, seq=M, num_heads=16, head_dim=64).items():
        setattr(f, k, v.data_ptr() if torch.is_tensor(v) else v)
    rc = lib.rfk_gemm_folded_more(ctypes.byref(f), ctypes.byref(more), ctypes.byref(tiles), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert (sums[n:] == -1.0).all()
    if small:
        assert rc == -2 and (sums == -1.0).all() and (out == 7.0).all()
        return
    assert rc == 0 and tiles.value == 4
    got = out.permute(2, 0, 1, 3).reshape(M, parts * dim)
    _near(got, (x.float() @ w.float().t()) * _factor(x, 1.0), K)
    want = got.float().square().view(M, parts, 4, -1).sum(-1).permute(1, 0, 2)
    assert torch.allclose(sums[:n].view(parts, M, 4)[0::2], want[0::2], rtol=2e-5, atol=1e-6)


@pytest.mark.parametrize("n,heads,layers", [(1, 16, 1), (60, 16, 3), (333, 8, 12), (1100, 16, 12), (2600, 8, 2)])
def test_cache_of_all_layers_at_once_and_layer_by_layer(n, heads, layers):
    """1024-wide rows: sessions with an image head keep one norm, two products and a transposing norm a layer; sessions without take one product."""
    from renderformer_cuda_b200 import session
    model = lambda dpt: session.Model.random(seed=6, dim=1024, num_heads=heads, ffn_hidden=256, enc_layers=1, dec_layers=layers, with_dpt=dpt,
                                             dpt_features=64, dpt_out_channels=(32, 64, 128, 128))
    scene, keys = _scene(n, n), (32 + n + 7) // 8 * 8
    states = []
    for dpt in (False, True):
        s = session.RenderSession(model(dpt), n, 64)
        for _ in range(2):   # the second time into what the first one left
            s.encode_scene(*scene)
        states.append(s.scene_state[: 2 * layers * keys * 1024 * 2].clone().view(torch.half).view(2 * layers, heads, keys, 1024 // heads))
        s.close()
    got, want = states
    assert (got[:, :, 32 + n:] == 0).all() and torch.isfinite(got).all()
    for i in range(2 * layers):   # (the encoder's attention may be cut along its keys without an image head)
        assert (got[i].float() - want[i].float()).norm() <= 1.5e-3 * want[i].float().norm()


@pytest.mark.parametrize("views,h,w", [(1, 8, 8), (3, 8, 8), (1, 16, 16), (4, 16, 16), (9, 16, 16), (1, 8, 24), (21, 8, 8), (41, 8, 8), (17, 16, 16), (150, 8, 8)])
@pytest.mark.parametrize("N,K", [(1024, 4096), (1024, 512), (256, 1536)])
def test_sums_in_quarters(views, h, w, N, K):
    """A residual product whose sum over K is that of its quarters: by clusters of four for few rows, by single CTAs for more, by pairs for many (41 views of
    64 rows: pair tiles with a tail of rows; 150: several tiles a pair, and pairs with 256 columns too). The sums and the
    order of their addition are the same whoever makes them: a view's rows have the bits of the frame that it shares; and they are those of four
    products of a quarter each, which leave fp32 nowhere, up to the distance of two orders."""
    rnd = _gen(views * 100 + h * w + K)
    M = views * h * w
    a, wt = rnd(M, K), rnd(N, K, scale=K ** -0.5)
    grid = rnd(views, h, w, N)
    r = _to_blocks(grid, 0)
    args = dict(W=wt, N=N, K=K, blocks_across=w // 4, blocks_down=h // 4, shift_from=0, shift_to=1, quarters=1)
    out, raster = (torch.full((M, N), float("nan"), device="cuda", dtype=torch.half) for _ in range(2))
    sums = torch.full((M * N // 32,), float("nan"), device="cuda")
    tiles = _run(0, A=a, R=r, C=out, raster=raster, out_ss=sums, M=M, **args)
    _check_sums(sums, tiles, out)
    back = _to_blocks(torch.arange(M, device="cuda", dtype=torch.float32).view(views, h, w, 1), 0).long().flatten()
    _near(raster[back], r.float() + a.float() @ wt.float().t(), K)
    assert torch.equal(out, _to_blocks(raster.view(views, h, w, N), 4))
    n = h * w
    if (views, h) in ((1, 8), (3, 8), (4, 16)):   # pairs whatever the size
        again, again_raster, again_sums = torch.empty_like(out), torch.empty_like(raster), torch.empty_like(sums)
        assert _run(2, A=a, R=r, C=again, raster=again_raster, out_ss=again_sums, M=M, **args) == tiles
        assert torch.equal(again, out) and torch.equal(again_raster, raster) and torch.equal(again_sums, sums)
        _run(2, A=a, W=wt, R=r, C=again, M=M, N=N, K=K, quarters=1)   # rows where they are, without sums
        assert torch.equal(again, raster[back])
    for v in {0, views // 2, views - 1}:
        alone, alone_raster = torch.full((n, N), float("nan"), device="cuda", dtype=torch.half), torch.full((n, N), float("nan"), device="cuda", dtype=torch.half)
        alone_sums = torch.full((n * N // 32,), float("nan"), device="cuda")
        _run(0, A=a[v * n:(v + 1) * n], R=r[v * n:(v + 1) * n], C=alone, raster=alone_raster, out_ss=alone_sums, M=n, **args)
        assert torch.equal(alone, out[v * n:(v + 1) * n]) and torch.equal(alone_raster, raster[v * n:(v + 1) * n])
        assert torch.equal(alone_sums, sums.view(views, -1)[v])


def test_sums_in_quarters_are_refused_where_they_cannot_be():
    f = Product()
    x = torch.zeros(64, 1024, device="cuda", dtype=torch.half)
    lib, tiles = _abi.load("rfk.h"), ctypes.c_int()
    for n in ("A", "W", "R", "C"):
        setattr(f, n, x.data_ptr())
    f.M, f.N, f.K, f.quarters = 64, 256, 256, 1
    assert lib.rfk_gemm_folded(ctypes.byref(f), ctypes.byref(tiles), None) == -2     # RFK_EUNSUPPORTED: 256 are not four stages
