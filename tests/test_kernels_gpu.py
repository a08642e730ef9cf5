"""GPU parity tests: every kernel, called through the C ABI, against
  (1) the CPU oracle on the same seeded inputs,
  (2) the reference engine's own CUDA kernels run live on the same device, when the
      oracle/_ref libraries travelled with the tree, and
  (3) the committed outputs of those reference kernels (tests/golden/)."""
from pathlib import Path

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden" / "reference_outputs.npz"


@pytest.fixture(scope="module")
def golden():
    return np.load(GOLDEN) if GOLDEN.exists() else None


@pytest.fixture(scope="module", autouse=True)
def _library_is_native():
    import renderformer_cuda_b200 as pkg
    from renderformer_cuda_b200 import _abi
    assert _abi.library_path("rfk.h").exists(), "librfk.so missing: the CUDA path must be the one that runs"
    assert "sm_100a" in pkg.version()


@pytest.mark.parametrize("case", cases.CASES, ids=lambda c: c.name)
def test_kernel_matches_oracle(case):
    i = case.inputs()
    got = case.rfk(i)
    want = case.oracle(i)
    for k, kind in case.kinds.items():
        cases.compare(case.oracle_kinds.get(k, kind), got[k], want[k], f"{case.name}.{k} vs oracle")


@pytest.mark.parametrize("case", [c for c in cases.CASES if c.ref is not None], ids=lambda c: c.name)
def test_kernel_matches_reference_kernels_live(case):
    from oracle import ref
    if not (ref.available() and ref.layers_available()):
        pytest.skip("oracle/_ref libraries not present")
    i = case.inputs()
    got = case.rfk(i)
    want = case.ref(i)
    for k, kind in case.kinds.items():
        cases.compare(kind, got[k], want[k], f"{case.name}.{k} vs reference kernels")


@pytest.mark.parametrize("case", [c for c in cases.CASES if c.ref is not None], ids=lambda c: c.name)
def test_kernel_matches_reference_golden(case, golden):
    if golden is None:
        pytest.skip("golden fixtures not generated yet")
    got = case.rfk(case.inputs())
    for k, kind in case.kinds.items():
        cases.compare(kind, got[k], golden[f"{case.name}::{k}"], f"{case.name}.{k} vs golden")


def test_launch_counter_counts():
    import torch
    import renderformer_cuda_b200 as pkg
    x = torch.randn(8, 1024, device="cuda").half()
    g = torch.ones(1024, device="cuda")
    n0 = pkg.ops.launch_count()
    pkg.ops.rmsnorm(x, g, x, 8, 1024)
    assert pkg.ops.launch_count() == n0 + 1


def test_kernels_run_on_a_side_stream_and_in_a_graph():
    """The entry points neither allocate nor synchronise: they can be captured."""
    import torch
    import renderformer_cuda_b200 as pkg
    x = torch.randn(64, 1024, device="cuda").half(); g = torch.ones(1024, device="cuda")
    y = torch.empty_like(x); pe_in = torch.randn(1, 64, 9, device="cuda")
    pe_out = torch.empty(1, 64, 117, device="cuda", dtype=torch.float16)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        pkg.ops.rmsnorm(x, g, y, 64, 1024)
    s.synchronize()
    want = y.clone()
    y.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.ops.rmsnorm(x, g, y, 64, 1024)
        pkg.ops.nerf_pe_f32(pe_in, pe_out, 1, 64, 9, 6, 0.0, 5.0, True)   # the reference form mallocs here
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert torch.isfinite(pe_out.float()).all()


@pytest.mark.gpu
@pytest.mark.parametrize("B,Hh,W,dim,ws,shift", [(1, 16, 16, 256, 8, 0), (1, 16, 16, 256, 8, 4), (2, 8, 24, 1024, 4, 3),
                                                 (1, 64, 64, 1024, 8, 4), (1, 8, 8, 2048, 8, 1)])
def test_rmsnorm_residual_with_window_ordered_operand_equals_the_separate_kernels(B, Hh, W, dim, ws, shift):
    """The fused norm that writes its output in swin window order (or reads its residual out of it) is bit-identical
    to residual+norm followed by window_gather, and to window_scatter(+residual) followed by the norm."""
    import torch
    import renderformer_cuda_b200 as pkg
    ops = pkg.ops
    rows = B * Hh * W
    g = torch.Generator(device="cuda").manual_seed(rows + dim + shift)
    x0 = torch.randn(rows, dim, device="cuda", generator=g).half()
    r = torch.randn(rows, dim, device="cuda", generator=g).half()
    gamma = torch.rand(dim, device="cuda", generator=g) + 0.5
    # (1) y in window order
    xa, xb = x0.clone(), x0.clone()
    ya, tmp, yb = torch.empty_like(x0), torch.empty_like(x0), torch.empty_like(x0)
    ops.rmsnorm_residual_f16(xa, r, gamma, tmp, rows, dim)
    ops.window_gather(tmp, ya, B, Hh, W, dim, ws, shift)
    ops.rmsnorm_residual_f16_windows(xb, r, gamma, yb, B, Hh, W, dim, ws, shift, 1)
    torch.cuda.synchronize()
    assert torch.equal(xa, xb) and torch.equal(ya, yb)
    # (2) r in window order
    xa, xb = x0.clone(), x0.clone()
    ops.window_scatter(r, xa, B, Hh, W, dim, ws, shift, residual_into=True)
    ops.rmsnorm(xa, gamma, ya, rows, dim)
    ops.rmsnorm_residual_f16_windows(xb, r, gamma, yb, B, Hh, W, dim, ws, shift, 2)
    torch.cuda.synchronize()
    assert torch.equal(xa, xb) and torch.equal(ya, yb)


@pytest.mark.parametrize("dim", [520, 768, 1024])
@pytest.mark.parametrize("side", [36, 40, 48])
def test_rmsnorm_one_warp_per_row_has_the_bits_of_four(side, dim):
    """Many fp16 rows go to one warp each, few to four: the same rows in one call and a few at a time, plain, with a residual, to
    windows and from windows."""
    import torch
    import renderformer_cuda_b200 as pkg
    ops = pkg.ops
    g = torch.Generator(device="cuda").manual_seed(dim + side)
    copies = 2
    rows = copies * side * side
    gamma = 1 + 0.1 * torch.randn(dim, device="cuda", generator=g)
    x0 = torch.randn(rows, dim, device="cuda", generator=g).half()
    r0 = torch.randn(rows, dim, device="cuda", generator=g).half()
    for res in (None, r0):
        x, y, xs, ys = x0.clone(), torch.empty_like(x0), x0.clone(), torch.empty_like(x0)
        ops.rmsnorm_residual_f16(x, res, gamma, y, rows, dim)
        for i in range(0, rows, 300):
            n = min(300, rows - i)
            ops.rmsnorm_residual_f16(xs[i:i + n], None if res is None else res[i:i + n], gamma, ys[i:i + n], n, dim)
        assert torch.equal(x, xs) and torch.equal(y, ys)
        if side % 8:
            continue
        for operand in ([1] if res is None else [1, 2]):
            xw, yw = x0.clone(), torch.empty_like(x0)
            ops.rmsnorm_residual_f16_windows(xw, res, gamma, yw, copies, side, side, dim, 8, 4, operand)
            def to_win(t):
                t = torch.roll(t.view(copies, side, side, dim), (4, 4), (1, 2)).view(copies, side // 8, 8, side // 8, 8, dim)
                return t.permute(0, 1, 3, 2, 4, 5).reshape(rows, dim).contiguous()
            def from_win(t):
                t = t.view(copies, side // 8, side // 8, 8, 8, dim).permute(0, 1, 3, 2, 4, 5).reshape(copies, side, side, dim)
                return torch.roll(t, (-4, -4), (1, 2)).reshape(rows, dim).contiguous()
            xs, ys = x0.clone(), torch.empty_like(x0)
            rs = None if res is None else (from_win(res) if operand == 2 else res)
            for i in range(0, rows, 300):
                n = min(300, rows - i)
                ops.rmsnorm_residual_f16(xs[i:i + n], None if rs is None else rs[i:i + n], gamma, ys[i:i + n], n, dim)
            assert torch.equal(xw, xs) and torch.equal(yw, to_win(ys) if operand == 1 else ys)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n", [1, 61, 3000])
def test_rope_tables_and_view_geometry_have_the_same_bits_for_many_and_few_tokens(n, hd):
    """Few tokens take two angles a thread, many eight: the same tokens in a small call and repeated in a large one."""
    import math
    import torch
    import renderformer_cuda_b200 as pkg
    from renderformer_cuda_b200 import _abi
    import ctypes
    ops, L, VP = pkg.ops, _abi.load("rfk.h"), ctypes.c_void_p
    g = torch.Generator(device="cuda").manual_seed(n)
    nf = min(6, hd // 2 // 9)
    freqs = torch.tensor([math.pi * 10000.0 ** (-i / nf) for i in range(nf)], device="cuda")
    pos = (torch.rand(n, 9, device="cuda", generator=g) * 4 - 2).half()
    tables = lambda t, m: [torch.empty(m, hd, device="cuda", dtype=torch.float16) for _ in range(2)]
    few = tables(pos, n)
    ops.triangle_rope_freqs(pos, freqs, *few, 1, n, nf, hd)
    copies = (1 << 20) // (hd // 4) // n + 1
    many = tables(pos, copies * n)
    ops.triangle_rope_freqs(pos.repeat(copies, 1).contiguous(), freqs, *many, 1, copies * n, nf, hd)
    for a, b in zip(few, many):
        assert torch.equal(b.view(copies, n, hd), a.expand(copies, n, hd))
    vn = torch.randn(n, 9, device="cuda", generator=g).half()
    c2w = torch.eye(4, device="cuda")
    c2w[:3, :] = torch.randn(3, 4, device="cuda", generator=g)
    centre = torch.zeros(3, device="cuda")
    def geometry(tri, normals, m):
        out = [torch.empty_like(tri), torch.empty_like(tri), torch.empty(m, 9, device="cuda", dtype=torch.float16), *tables(tri, m)]
        rc = L.rfk_view_geometry(*(VP(t.data_ptr()) for t in (c2w, tri, normals, centre, freqs, *out)), m, 0, m, nf, hd,
                                 VP(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        return out
    copies = 100000 // (hd // 4) // n + 1
    for a, b in zip(geometry(pos, vn, n), geometry(pos.repeat(copies, 1).contiguous(), vn.repeat(copies, 1).contiguous(), copies * n)):
        assert torch.equal(b.view(copies, n, -1), a.expand(copies, n, -1))


@pytest.mark.parametrize("dtype", ["float16", "float32"])
@pytest.mark.parametrize("in_dim", [3, 9])
@pytest.mark.parametrize("rows,exps", [(1, (0.0, 5.0)), (31, (0.0, 5.0)), (33, (0.0, 4.0)), (1000, (0.0, 5.0))])
def test_nerf_pe_has_the_same_bits_for_many_and_few_rows(rows, exps, in_dim, dtype):
    """Few rows take a thread per coordinate, many a thread per row or two: octaves (doubling) and other bands, ragged tiles."""
    import torch
    import renderformer_cuda_b200 as pkg
    dt = getattr(torch, dtype)
    fn = pkg.ops.nerf_pe if dt == torch.float16 else pkg.ops.nerf_pe_f32
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, in_dim, device="cuda", generator=g).to(dt)
    few = torch.empty(rows, in_dim * 13, device="cuda", dtype=torch.float16)
    fn(x, few, 1, rows, in_dim, 6, *exps, True)
    copies = (1 << 16) // rows + 1
    many = torch.empty(copies * rows, in_dim * 13, device="cuda", dtype=torch.float16)
    fn(x.repeat(copies, 1).contiguous(), many, 1, copies * rows, in_dim, 6, *exps, True)
    assert torch.equal(many.view(copies, rows, -1), few.expand(copies, rows, -1))


@pytest.mark.parametrize("dim", [520, 1024])
@pytest.mark.parametrize("copies,side", [(1, 24), (1, 40), (2, 64), (3, 64)])
def test_window_norm_of_operands_in_l2_has_the_bits_of_the_other_split(copies, side, dim):
    """The layers' form of the norm to and from windows takes one warp a row from 1280 rows up, the operator four with a residual."""
    import ctypes
    import torch
    import renderformer_cuda_b200 as pkg
    from renderformer_cuda_b200 import _abi
    fn = _abi.load("rfk.h").rfk_rmsnorm_residual_f16_windows_in_l2
    fn.argtypes, fn.restype = [ctypes.c_void_p] * 4 + [ctypes.c_int] * 7 + [ctypes.c_float, ctypes.c_void_p], ctypes.c_int
    g = torch.Generator(device="cuda").manual_seed(dim + side)
    rows = copies * side * side
    gamma = 1 + 0.1 * torch.randn(dim, device="cuda", generator=g)
    x0, r = (torch.randn(rows, dim, device="cuda", generator=g).half() for _ in range(2))
    for operand in (1, 2):
        x, y, xw, yw = x0.clone(), torch.empty_like(x0), x0.clone(), torch.empty_like(x0)
        pkg.ops.rmsnorm_residual_f16_windows(x, r, gamma, y, copies, side, side, dim, 8, 4, operand)
        rc = fn(*(ctypes.c_void_p(t.data_ptr()) for t in (xw, r, gamma, yw)), copies, side, side, dim, 8, 4, operand, pkg.ops.K_EPS_FP16,
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert rc == 0 and torch.equal(x, xw) and torch.equal(y, yw)
