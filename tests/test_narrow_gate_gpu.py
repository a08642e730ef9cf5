"""Gate products on pairs with 64 hidden units (129 to 256 rows of the models' FFN): the bits of the pair kernel's wide tiles, which sum K in the same
order, at ragged rows, a tail of the hidden units, few and odd numbers of K blocks, and against torch in fp64 (the fp32 sum and one rounding to fp16)."""
import pytest
import torch

import renderformer_cuda_b200 as pkg

pytestmark = pytest.mark.gpu
ops = pkg.ops


@pytest.mark.parametrize("M", [129, 200, 256])
@pytest.mark.parametrize("N,K", [(4096, 1024), (4096, 72), (2440, 200), (4600, 1600)])
def test_narrow_gate_has_the_bits_of_the_wide_tiles(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, w, u = rnd(M, K).half(), (rnd(N, K) / K ** 0.5).half(), (rnd(N, K) / K ** 0.5).half()
    got, want = (torch.full((M, N), 7.0, device="cuda", dtype=torch.half) for _ in range(2))
    ops.gemm_f16(a, w, got, M, N, K, w_up=u)
    ops.gemm_set_path(2)
    try:
        ops.gemm_f16(a, w, want, M, N, K, w_up=u)
    finally:
        ops.gemm_set_path(0)
    assert torch.equal(got, want)
    x = a.double()
    ref = torch.nn.functional.silu(x @ w.double().t()) * (x @ u.double().t())
    assert ((got.double() - ref).abs() <= 1e-4 + 2e-3 * ref.abs()).all()
