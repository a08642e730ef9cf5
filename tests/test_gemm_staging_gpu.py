"""The pair kernel's two staging buffers from tile to tile: many tiles a pair with so few K blocks that the next accumulator is complete
when an epilogue ends, and tiles of an odd number of 64-column units (192 columns, or a tail of N), so that a tile does not begin with
the buffer that the one before it began with. Launched again and again, bit for bit against the single-CTA kernel, which stages nothing."""
import pytest
import torch

import renderformer_cuda_b200 as pkg

pytestmark = pytest.mark.gpu
H16 = torch.float16
ops = pkg.ops
LAUNCHES = 200


@pytest.fixture(autouse=True)
def _paths():
    ops.gemm_error(clear=True)
    yield
    ops.gemm_set_path(0)
    torch.cuda.synchronize()
    assert ops.gemm_error(clear=True) == 0


def _rand(g, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).half()


def _same_every_time(call, out, want):
    ops.gemm_set_path(2)
    bad = torch.zeros((), device="cuda", dtype=torch.int64)
    for _ in range(LAUNCHES):
        out.fill_(7.0)
        call(out)
        bad += (out != want).sum()
    assert bad.item() == 0


# 192-column tiles of three units, with tails of one (1024) and three; 256-column tiles with a tail of three (19000 x 448); SwiGLU tiles
# of two units with a tail of one
@pytest.mark.parametrize("M,N,K", [(3136, 3072, 64), (4800, 1024, 192), (5665, 1024, 72), (60000, 192, 64), (30000, 320, 128), (19000, 448, 64)])
@pytest.mark.parametrize("epilogue", ["plain", "bias", "swiglu", "residual"])
def test_tiles_with_odd_numbers_of_units(M, N, K, epilogue):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = _rand(g, M, K), _rand(g, N, K, scale=K ** -0.5)
    extra = {"bias": {"bias": _rand(g, N)}, "swiglu": {"w_up": _rand(g, N, K, scale=K ** -0.5)},
             "residual": {"residual": _rand(g, M, N)}}.get(epilogue, {})
    want, out = (torch.empty(M, N, device="cuda", dtype=H16) for _ in "wo")
    ops.gemm_set_path(3)
    ops.gemm_f16(a, w, want, M, N, K, **extra)
    _same_every_time(lambda o: ops.gemm_f16(a, w, o, M, N, K, **extra), out, want)


@pytest.mark.parametrize("M,seq,parts,heads", [(5632, 5632, 1, 16), (7168, 64, 1, 16), (3136, 64, 3, 16), (9216, 64, 3, 4)])
def test_head_split_tiles(M, seq, parts, heads):
    dim, K = heads * 64, 64
    g = torch.Generator(device="cuda").manual_seed(M + parts)
    a, w = _rand(g, M, K), _rand(g, parts * dim, K, scale=K ** -0.5)
    want = torch.empty(M, parts * dim, device="cuda", dtype=H16)
    ops.gemm_set_path(3)
    ops.gemm_f16(a, w, want, M, parts * dim, K)
    out = torch.empty(parts, M // seq, heads, seq, 64, device="cuda", dtype=H16)
    _same_every_time(lambda o: ops.gemm_f16_heads(a, w, o, None, 0, M, parts * dim, K, seq, heads, part_stride=M * dim if parts > 1 else 0),
                     out, want.view(M // seq, seq, parts, heads, 64).permute(2, 0, 3, 1, 4).contiguous())
