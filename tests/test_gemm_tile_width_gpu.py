"""The pair kernel's tiles of 192 and of 256 columns (narrow_tile): every output is one sum over K in the same order, so both have
the bits of the single-CTA kernel. Shapes on both sides of the rule on 148 SMs, with remainders of 192 columns, 256 rows and 64 of K."""
import pytest
import torch

import renderformer_cuda_b200 as pkg

pytestmark = pytest.mark.gpu
H16 = torch.float16
ops = pkg.ops


@pytest.fixture(autouse=True)
def _paths():
    ops.gemm_error(clear=True)
    yield
    ops.gemm_set_path(0)
    torch.cuda.synchronize()
    assert ops.gemm_error(clear=True) == 0


def _rand(g, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).half()


# 192 columns: the first six; 256: the others
@pytest.mark.parametrize("M,N,K", [(2500, 1024, 1024), (4864, 1000, 200), (5665, 1024, 4096), (1600, 3072, 1024), (257, 200, 72), (1, 8, 8),
                                   (3400, 1024, 328), (4096, 3072, 1024), (6400, 1024, 136)])
@pytest.mark.parametrize("epilogue", ["plain", "bias", "residual"])
def test_tile_widths_have_the_same_bits(M, N, K, epilogue):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = _rand(g, M, K), _rand(g, N, K, scale=K ** -0.5)
    extra = {"bias": {"bias": _rand(g, N)}, "residual": {"residual": _rand(g, M, N)}}.get(epilogue, {})
    outs = []
    for path in (2, 3):
        ops.gemm_set_path(path)
        outs.append(torch.full((M, N), 7.0, device="cuda", dtype=H16))
        ops.gemm_f16(a, w, outs[-1], M, N, K, **extra)
    assert torch.equal(outs[0], outs[1])
    want = a.float() @ w.float().t()
    if epilogue == "residual":
        want = want + extra["residual"].float()
    if epilogue != "bias":
        # one fp16 rounding of the result, and fp32 sums of K products of about unit variance in another order
        assert ((outs[0].float() - want).abs() <= 1e-3 + 2.0 ** -10 * want.abs()).all()


@pytest.mark.parametrize("M,seq,parts,heads", [(5632, 5632, 1, 16), (2560, 64, 1, 16), (1600, 1600, 3, 16), (2304, 64, 3, 4)])
def test_head_split_without_statistics(M, seq, parts, heads):
    """A unit of 64 columns is one head wherever a tile of 192 columns begins, a part's last tile among them."""
    dim, K = heads * 64, 256
    g = torch.Generator(device="cuda").manual_seed(M + parts)
    a, w = _rand(g, M, K), _rand(g, parts * dim, K, scale=K ** -0.5)
    want = torch.empty(M, parts * dim, device="cuda", dtype=H16)
    ops.gemm_set_path(3)
    ops.gemm_f16(a, w, want, M, parts * dim, K)
    ops.gemm_set_path(2)
    out = torch.full((parts, M // seq, heads, seq, 64), 7.0, device="cuda", dtype=H16)
    ops.gemm_f16_heads(a, w, out, None, 0, M, parts * dim, K, seq, heads, part_stride=M * dim if parts > 1 else 0)
    assert torch.equal(out, want.view(M // seq, seq, parts, heads, 64).permute(2, 0, 3, 1, 4))
