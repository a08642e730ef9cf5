"""Performance cases: the work a program does through this package's public entry points.

A case is a dict of plain values; `kind` says which path it takes:

  norm, rope, softmax, front   the element-wise and row operators (`ops`), on one scene's or one view's tensors
  encode                       a scene goes in: 12 encoder layers and the cross-attention K/V cache of 12 decoder layers
  view                         one camera in, the decoder's token map of that view out in pinned memory (interactive use:
                               the program waits for each frame)
  image                        the same with the DPT head: a [3, res, res] fp32 image out
  views                        a batch of cameras through the ViewScheduler (offline rendering: frames stay in flight)

The path is inference only, so there is no backward direction; activations and weights are fp16 throughout, the residual
stream of the encoder fp32. The network has the dimensions of renderformer-v1.1-swin-large (dim 1024, 12 + 12 layers, FFN
4096) with random weights, once with 16 heads of 64 (the benchmark's configuration) and once with 8 heads of 128 (the
published checkpoint's head geometry).
"""
import math

import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import session

ops = pkg.ops

DIM, FFN, LAYERS, REGISTERS, PATCH, TEX = 1024, 4096, 12, 32, 8, 13
H, F = torch.float16, torch.float32


def listed():
    return [
        # -- operators ------------------------------------------------------------------------------------------
        # the residual stream of a 5633-triangle scene between two encoder layers
        {"name": "norm_f32_5633", "kind": "norm", "stream": "f32", "rows": 5633, "dim": 1024},
        # triangle rotary tables, rotation of Q and K and the normals' encoding of that scene
        {"name": "rope_5633", "kind": "rope", "tris": 5633, "heads": 16},
        # materialised cross-attention scores of one 512 x 512 view: the largest single tensor an operator is given
        {"name": "softmax_65536x5633", "kind": "softmax", "rows": 65536, "cols": 5633},
        # ray front end and gate of a preview-sized view: nothing here is longer than its launch
        {"name": "front_64", "kind": "front", "res": 64, "tris": 301, "batch": 1},
        # the same for a full view
        {"name": "front_512", "kind": "front", "res": 512, "tris": 5633, "batch": 1},
        # -- scene -----------------------------------------------------------------------------------------------
        {"name": "encode_5633", "kind": "encode", "tris": 5633, "heads": 16},
        # -- views -----------------------------------------------------------------------------------------------
        # moving the camera in a small scene at preview size: 145 short kernels one after the other
        {"name": "view_128_small_scene", "kind": "view", "res": 128, "tris": 301, "heads": 16},
        # the benchmark's view, one at a time
        {"name": "view_512", "kind": "view", "res": 512, "tris": 5633, "heads": 16},
        # the same view with the published checkpoint's heads
        {"name": "view_512_h128", "kind": "view", "res": 512, "tris": 5633, "heads": 8},
        # an image at an in-between size, whose 1600 tokens fill no power of two, with the published heads
        {"name": "image_320_h128", "kind": "image", "res": 320, "tris": 4575, "heads": 8},
        # a full image
        {"name": "image_512", "kind": "image", "res": 512, "tris": 5633, "heads": 16},
        # offline rendering of a camera path: frames of four views, two in flight
        {"name": "views16_512", "kind": "views", "res": 512, "tris": 5633, "heads": 16, "views": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["norm", "rope", "softmax", "front", "encode", "view", "view", "image", "views"])
    tris = _log_int(rng, 60, 7200)
    res = 64 * rng.randint(1, 8)
    heads = rng.choice([8, 16])
    if kind == "norm":
        return {"kind": kind, "stream": rng.choice(["f32", "mixed", "f16"]), "rows": _log_int(rng, 33, 45000),
                "dim": rng.choice([256, 768, 1024])}
    if kind == "rope":
        return {"kind": kind, "tris": tris, "heads": heads}
    if kind == "softmax":
        return {"kind": kind, "rows": 16 * _log_int(rng, 64, 4096), "cols": tris}
    if kind == "front":
        return {"kind": kind, "res": res, "tris": tris, "batch": rng.randint(1, 6)}
    if kind == "encode":
        return {"kind": kind, "tris": tris, "heads": heads}
    if kind == "views":
        return {"kind": kind, "res": res, "tris": min(tris, 5633), "heads": heads,
                "views": rng.randint(2, 16 if heads == 16 else 6)}
    return {"kind": kind, "res": res, "tris": tris, "heads": heads}


# -- inputs -----------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=F):
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


def _scene(g, n):
    """Triangles with vertices in [-1, 1]^3, unit vertex normals, albedo / roughness / emission in [0, 1]."""
    tri = torch.rand(n, 3, 3, device="cuda", generator=g) * 2 - 1
    vn = torch.nn.functional.normalize(_randn(g, n, 3, 3), dim=-1)
    tex = torch.rand(n, TEX, device="cuda", generator=g).half()
    return tri.contiguous(), vn.contiguous(), tex.contiguous()


def _cameras(seed, n):
    """Pinhole cameras on a sphere of radius 2 to 4 that look at the origin, 30 to 60 degrees: [n, 4, 4] and [n], host."""
    g = torch.Generator().manual_seed(int(seed) + 7)
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g), dim=-1)
    pos = d * (2 + 2 * torch.rand(n, 1, generator=g))
    up = torch.tensor([0.0, 0.0, 1.0]).expand(n, 3).clone()
    up[d[:, 2].abs() > 0.95] = torch.tensor([0.0, 1.0, 0.0])
    right = torch.nn.functional.normalize(torch.linalg.cross(up, d), dim=-1)
    c2w = torch.zeros(n, 4, 4)
    c2w[:, :3, 0], c2w[:, :3, 1], c2w[:, :3, 2], c2w[:, :3, 3] = right, torch.linalg.cross(d, right), d, pos
    c2w[:, 3, 3] = 1
    return c2w.contiguous(), (30 + 30 * torch.rand(n, generator=g)) * (math.pi / 180)


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    s = dict(case)
    if kind == "norm":
        rows, dim = case["rows"], case["dim"]
        s["x"] = _randn(g, rows, dim, dtype=H if case["stream"] == "f16" else F)
        s["r"] = _randn(g, rows, dim, dtype=F if case["stream"] == "f32" else H)
        s["gamma"] = 1 + 0.02 * _randn(g, dim)
        s["y"] = torch.empty(rows, dim, device="cuda", dtype=H)
    elif kind == "rope":
        n, hd = case["tris"], DIM // case["heads"]
        nf = min(6, hd // 2 // 9)
        s.update(hd=hd, nf=nf)
        tri, vn, _ = _scene(g, n)
        s["pos"], s["vn"] = tri.reshape(n, 9).half(), vn.reshape(n, 9)
        s["freqs"] = torch.tensor([math.pi * 10000.0 ** (-i / nf) for i in range(nf)], device="cuda", dtype=F)
        s["q"], s["k"] = _randn(g, case["heads"], n, hd, dtype=H), _randn(g, case["heads"], n, hd, dtype=H)
        s["cos"], s["sin"] = torch.empty(n, hd, device="cuda", dtype=H), torch.empty(n, hd, device="cuda", dtype=H)
        s["pe"] = torch.empty(n, 9 * 13, device="cuda", dtype=H)
    elif kind == "softmax":
        pad = (case["cols"] + 7) // 8 * 8
        s["pad"] = pad
        s["scores"] = torch.randn(case["rows"], pad, device="cuda", generator=g)
        s["scores"] *= 3
        s["scores"][:, case["cols"]:] = -math.inf
        s["probs"] = torch.empty(case["rows"], pad, device="cuda", dtype=H)
    elif kind == "front":
        b, res = case["batch"], case["res"]
        tri, vn, _ = _scene(g, case["tris"])
        s["tri_world"] = tri.half().expand(b, -1, -1, -1).contiguous()
        s["vn_world"] = vn.half().expand(b, -1, -1, -1).contiguous()
        s["tri"], s["vn"] = torch.empty_like(s["tri_world"]), torch.empty_like(s["vn_world"])
        c2w, fov = _cameras(seed, b)
        s["c2w"], s["fov"] = c2w.cuda(), fov.cuda()
        s["rays_o"] = torch.empty(b, 3, device="cuda", dtype=F)
        s["rays_d"] = torch.empty(b, res, res, 3, device="cuda", dtype=H)
        s["pe"] = torch.empty(b, res * res, 39, device="cuda", dtype=H)
        n = b * (res // PATCH) ** 2 * FFN
        s["gate"], s["up"], s["act"] = _randn(g, n, dtype=H), _randn(g, n, dtype=H), torch.empty(n, device="cuda", dtype=H)
    else:
        _prepare_session(s, case, seed, g)
    return s


def _prepare_session(s, case, seed, g):
    kind, res = case["kind"], case.get("res", 512)
    s["model"] = model = session.Model.random(seed=int(seed), num_heads=case["heads"], with_dpt=kind == "image")
    s["scene"] = _scene(g, case["tris"])
    if kind == "encode":
        s["session"] = session.RenderSession(model, case["tris"], res)
        return
    s["c2w"], s["fov"] = _cameras(seed, case.get("views", 1))
    if kind == "views":
        # a frame of several views needs heads of 64; other heads go one view per frame
        s["sched"] = session.ViewScheduler(model, case["tris"], res, streams_per_gpu=2,
                                           views_per_frame=4 if case["heads"] == 16 else 1)
        s["sched"].load_scene(*s["scene"])
    else:
        s["fov"] = float(s["fov"][0])
        s["session"] = session.RenderSession(model, case["tris"], res)
        s["session"].encode_scene(*s["scene"])
        s["session"].finalize()
    if kind == "image":
        s["host"] = torch.empty(3, res, res, dtype=F).pin_memory()
    else:
        s["host"] = torch.empty(*([case["views"]] if kind == "views" else []), (res // PATCH) ** 2, DIM, dtype=H).pin_memory()


# -- one pass ---------------------------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "norm":
        if s["stream"] == "f32":
            ops.rmsnorm_residual_f32_cast16(s["x"], s["r"], s["gamma"], s["y"], s["rows"], s["dim"], ops.K_EPS_FP32)
        elif s["stream"] == "mixed":
            ops.rmsnorm_residual_mixed_cast16(s["x"], s["r"], s["gamma"], s["y"], s["rows"], s["dim"], ops.K_EPS_FP32)
        else:
            ops.rmsnorm_residual_f16(s["x"], s["r"], s["gamma"], s["y"], s["rows"], s["dim"])
        return [s["x"], s["y"]]
    if kind == "rope":
        n, heads, hd = s["tris"], s["heads"], s["hd"]
        ops.triangle_rope_freqs(s["pos"], s["freqs"], s["cos"], s["sin"], 1, n, s["nf"], hd)
        ops.apply_rope(s["q"], s["k"], s["cos"], s["sin"], 1, heads, n, hd)
        ops.nerf_pe_f32(s["vn"], s["pe"], 1, n, 9, 6, 0.0, 5.0, True)
        return [s["cos"], s["sin"], s["q"], s["k"], s["pe"]]
    if kind == "softmax":
        ops.softmax_cast_fp16(s["scores"], s["probs"], s["rows"], s["cols"], s["pad"], s["pad"])
        return s["probs"]
    if kind == "front":
        b, res = s["batch"], s["res"]
        s["tri"].copy_(s["tri_world"])
        s["vn"].copy_(s["vn_world"])
        ops.world_to_cam(s["c2w"], s["tri"], s["vn"], b, s["tris"])
        ops.ray_gen(s["c2w"], s["fov"], s["rays_o"], s["rays_d"], b, res)
        ops.nerf_pe(s["rays_d"], s["pe"], b, res * res, 3, 6, 0.0, 5.0, True)
        ops.fused_silu_mul(s["gate"], s["up"], s["act"], s["act"].numel())
        return [s["tri"], s["vn"], s["rays_o"], s["rays_d"], s["pe"], s["act"]]
    if kind == "encode":
        s["session"].encode_scene(*s["scene"])
        state = s["session"].scene_state
        kv = 2 * LAYERS * _keys_padded(s["tris"]) * DIM * 2      # bytes of the K/V cache; geometry and centre follow
        return {"kv": state[:kv].view(H), "geometry": state[kv:]}
    if kind == "views":
        s["sched"].render(s["c2w"], s["fov"], out=s["host"])
        return s["host"]
    s["session"].render_frame(s["c2w"], s["fov"])
    return s["session"].download_image(s["host"]) if kind == "image" else s["session"].download(s["host"])


# -- what a pass cannot do without ------------------------------------------------------------------------------------

def _keys_padded(tris):
    return (tris + REGISTERS + 7) // 8 * 8


def _decoder(tokens, keys, dim=DIM):
    """Operations of 12 decoder layers for `tokens` query rows; bytes of their weights and of the K/V cache."""
    per_layer = 2 * tokens * dim * dim * 6 + 6 * tokens * dim * FFN + 4 * tokens * keys * dim + 4 * tokens * 64 * dim
    return LAYERS * per_layer + 2 * tokens * 192 * dim, 2 * LAYERS * (6 * dim * dim + 3 * dim * FFN + 2 * keys * dim)


def _head(p):
    """Operations and weight bytes of the DPT head on a p x p token grid (features 256, channels 256/512/1024/1024)."""
    fl = wb = 0

    def conv(h, cin, cout, k):
        nonlocal fl, wb
        fl += 2 * h * h * cin * cout * k * k
        wb += 2 * cin * cout * k * k

    chans, sides = (256, 512, 1024, 1024), (4 * p, 2 * p, p, (p + 1) // 2)
    for c in chans:
        conv(p, DIM, c, 1)
    for c, f in ((256, 4), (512, 2)):
        fl += 2 * p * p * c * c * f * f
        wb += 2 * c * c * f * f
    conv(sides[3], 1024, 1024, 3)
    for i, (c, h) in enumerate(zip(chans, sides)):
        conv(h, c, 256, 3)
        for _ in range(2 if i == 3 else 4):
            conv(h, 256, 256, 3)
        # the 1x1 after the resample acts on each pixel alone, so it can be taken before it
        conv(h, 256, 256, 1)
    conv(8 * p, 256, 128, 3)
    conv(8 * p, 128, 32, 3)
    conv(8 * p, 32, 3, 1)
    return fl, wb


def work(case):
    kind = case["kind"]
    if kind == "norm":
        x, r = (2 if case["stream"] == "f16" else 4), (4 if case["stream"] == "f32" else 2)
        n = case["rows"] * case["dim"]
        return {"bytes": n * (2 * x + r + 2) + 4 * case["dim"], "flops": 6 * n}
    if kind == "rope":
        n, hd = case["tris"], DIM // case["heads"]
        # positions and tables, Q and K in and out, normals in and their encoding out
        return {"bytes": n * (18 + 2 * 2 * hd) + 4 * 2 * n * DIM + n * (36 + 2 * 117), "flops": 2 * 3 * n * DIM}
    if kind == "softmax":
        return {"bytes": case["rows"] * (4 * case["cols"] + 2 * ((case["cols"] + 7) // 8 * 8)), "flops": 5 * case["rows"] * case["cols"]}
    if kind == "front":
        b, px = case["batch"], case["batch"] * case["res"] ** 2
        gate = px // PATCH ** 2 * FFN
        # triangles and normals in and out, ray directions out and their encoding out, the gate's two inputs and output
        return {"bytes": 2 * 2 * 2 * 9 * b * case["tris"] + px * (6 + 78) + 3 * 2 * gate, "flops": 40 * px + 5 * gate}
    if kind == "encode":
        s = case["tris"] + REGISTERS
        layer = 2 * s * DIM * DIM * 4 + 6 * s * DIM * FFN + 4 * s * s * DIM
        kv = 2 * s * DIM * DIM * 2
        weights = 2 * LAYERS * (4 * DIM * DIM + 3 * DIM * FFN + 2 * DIM * DIM)
        return {"bytes": weights + case["tris"] * (72 + 2 * TEX) + 2 * 2 * LAYERS * _keys_padded(case["tris"]) * DIM,
                "flops": LAYERS * (layer + kv) + 2 * s * DIM * (TEX + 117)}
    views, tokens = case.get("views", 1), (case["res"] // PATCH) ** 2
    flops, weights = _decoder(tokens, case["tris"] + REGISTERS)
    flops *= views
    out = 2 * views * tokens * DIM
    if kind == "image":
        head, head_weights = _head(case["res"] // PATCH)
        flops, weights, out = flops + head, weights + head_weights, 4 * 3 * case["res"] ** 2
    return {"bytes": weights + out + 36 * case["tris"], "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("norm", "rope", "softmax", "front"):
        # results are rounded to fp16 once (spacing 2^-10 of the value at most): two correct fp32 computations may round
        # to neighbours; probabilities below 2^-14 are subnormal and carry fewer bits
        return {"rel": 1e-3, "max": 2e-3}
    if kind == "encode":
        return {"rel": 3e-3, "max": 3e-2}      # 12 layers of fp16 products on an fp32 stream
    if kind == "image":
        # 12 layers, then a head of 32 fp16 convolutions whose output is an exponent: 10^x magnifies a rounding by 2.3 x
        return {"rel": 1e-2, "max": 1e-1}
    return {"rel": 4e-3, "max": 4e-2}          # 12 layers with an fp16 residual stream
