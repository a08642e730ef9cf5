"""Small output tiles of the projection kernel (64 x 32 to 128 x 128, one per CTA) at the edges of tiles, stages and of the
rule that chooses them. Oracle: the single-CTA kernel on the same operands, bit for bit - the K blocks are added in the
same order on every tile - and torch fp32 for the sizes themselves (fp16 operands, fp32 sums, one rounding: 2^-11 relative,
plus the fp32 sum of at most 4096 products of magnitude 1 / sqrt(K))."""
import pytest
import torch

import renderformer_cuda_b200 as pkg

pytestmark = pytest.mark.gpu
ops = pkg.ops


@pytest.fixture(autouse=True)
def _paths():
    ops.gemm_error(clear=True)
    yield
    ops.gemm_set_path(0)
    torch.cuda.synchronize()
    assert ops.gemm_error(clear=True) == 0


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 8), (63, 40, 64), (64, 32, 128), (65, 33 * 8, 136), (129, 1024, 200), (256, 1024, 1024), (256, 1024, 4096),
    (576, 1024, 1024), (577, 1000, 1096), (1024, 1024, 1024), (1025, 1032, 328), (1600, 1024, 1024), (2304, 1024, 264),
    (2368, 1024, 64), (2369, 1024, 64)])
@pytest.mark.parametrize("epilogue", ["none", "bias", "residual", "in_place", "swiglu"])
def test_same_bits_as_the_large_tiles(M, N, K, epilogue):
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, w = rnd(M, K).half(), (rnd(N, K) * K ** -0.5).half()
    kw = {}
    if epilogue == "bias":
        kw["bias"] = rnd(N).half()
    if epilogue == "swiglu":
        kw["w_up"] = (rnd(N, K) * K ** -0.5).half()
    r = rnd(M, N).half()
    got = []
    for path in (0, 3):
        ops.gemm_set_path(path)
        c = r.clone() if epilogue == "in_place" else torch.full((M, N), 7.0, device="cuda", dtype=torch.float16)
        if epilogue in ("residual", "in_place"):
            kw["residual"] = c if epilogue == "in_place" else r
        ops.gemm_f16(a, w, c, M, N, K, **kw)
        got.append(c)
    assert torch.equal(got[0], got[1])
    want = a.float() @ w.float().t()
    if epilogue == "bias":
        want = want.half().float() + kw["bias"].float()
    if epilogue in ("residual", "in_place"):
        want = want + r.float()
    if epilogue == "swiglu":
        want = torch.nn.functional.silu(want) * (a.float() @ kw["w_up"].float().t())
    assert ((got[0].float() - want).abs() <= 2e-3 + 2e-3 * want.abs()).all()


@pytest.mark.parametrize("M,N,K", [(70, 48, 72), (300, 96, 256)])
def test_pitches_larger_than_the_rows(M, N, K):
    """Only the output's own columns are written, operands of a wider matrix are read in place."""
    g = torch.Generator(device="cuda").manual_seed(1)
    big_a = torch.randn(M, K + 24, device="cuda", generator=g).half()
    big_w = torch.randn(N, K + 8, device="cuda", generator=g).half()
    out = torch.full((M, N + 16), 7.0, device="cuda", dtype=torch.float16)
    ops.gemm_f16(big_a, big_w, out, M, N, K, lda=K + 24, ldw=K + 8, ldc=N + 16)
    want = torch.empty(M, N, device="cuda", dtype=torch.float16)
    ops.gemm_f16(big_a[:, :K].contiguous(), big_w[:, :K].contiguous(), want, M, N, K)
    assert torch.equal(out[:, :N], want) and (out[:, N:] == 7.0).all()


@pytest.mark.parametrize("M,seq,heads,parts,K,mask", [
    (32, 32, 4, 1, 72, 1), (64, 64, 16, 3, 1024, 3), (96, 32, 8, 3, 200, 2), (256, 256, 16, 1, 1024, 1),
    (256, 64, 16, 3, 1024, 3), (576, 64, 16, 3, 1024, 3), (960, 320, 4, 1, 136, 1), (1600, 1600, 16, 1, 1024, 1)])
def test_head_split_form_has_the_bits_of_the_pair_kernel(M, seq, heads, parts, K, mask):
    """The same rows as the head of a call that is large enough for the pair kernel: values and row statistics."""
    dim = heads * 64
    N = parts * dim
    g = torch.Generator(device="cuda").manual_seed(M + K)
    groups = -(-9600 // seq)
    a = torch.randn(groups * seq, K, device="cuda", generator=g).half()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).half()
    got = []
    for rows in (M, groups * seq):
        out = torch.full((parts, rows * dim), 7.0, device="cuda", dtype=torch.float16)
        ss = torch.full((parts, rows, dim // 256), -1.0, device="cuda", dtype=torch.float32)
        ops.gemm_f16_heads(a[:rows].contiguous(), w, out, ss, mask, rows, N, K, seq, heads, part_stride=rows * dim)
        got.append((out[:, :M * dim], ss[:, :M]))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert all(bool((got[0][1][p] >= 0).all()) == bool(mask >> p & 1) for p in range(parts))


def test_pair_path_serves_small_calls_with_the_pair_kernel():
    """In a fresh process: the pair kernel's occupancy query has run after one small call on path 2, and not after the same
    call on path 0, which goes to the small tiles."""
    import subprocess
    import sys
    from pathlib import Path
    code = """
import sys, torch, renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi
o, lib = pkg.ops, _abi.load("rfk.h")
a = torch.randn(77, 136, device="cuda").half(); w = torch.randn(1000, 136, device="cuda").half()
h = torch.randn(64, 64, device="cuda").half(); wh = torch.randn(256, 64, device="cuda").half()
out = torch.empty(77, 1000, device="cuda", dtype=torch.float16); outh = torch.empty(4, 64, 64, device="cuda", dtype=torch.float16)
o.gemm_set_path(int(sys.argv[1]))
if sys.argv[2] == "plain": o.gemm_f16(a, w, out, 77, 1000, 136)
else: o.gemm_f16_heads(h, wh, outh, None, 0, 64, 256, 64, 64, 4)
torch.cuda.synchronize()
print(lib.rfk_gemm_pair_clusters())
"""
    root = Path(__file__).resolve().parent.parent
    for form in ("plain", "heads"):
        for path in ("0", "2"):
            r = subprocess.run([sys.executable, "-c", code, path, form], capture_output=True, text=True, cwd=root)
            assert r.returncode == 0, r.stderr
            assert (int(r.stdout.split()[-1]) > 0) == (path == "2"), (form, path, r.stdout)
