"""The compiled operator binding against the checked Python functions behind it: same results, same argument errors."""
import pytest
import torch

import renderformer_cuda_b200 as pkg

pytestmark = pytest.mark.gpu
ops = pkg.ops


def _norm_args(rows=3, dim=40):
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, dim, device="cuda", generator=g).half()
    return x, torch.ones(dim, device="cuda"), torch.empty_like(x), rows, dim


@pytest.mark.parametrize("call", ["positional", "default", "keyword", "int_for_float"])
def test_binding_matches_checked_function(call):
    x, gamma, y, rows, dim = _norm_args()
    want = torch.empty_like(y)
    eps = 1.0 if call == "int_for_float" else ops.K_EPS_FP16
    ops.rmsnorm.__wrapped__(x, gamma, want, rows, dim, eps)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        if call == "positional":
            ops.rmsnorm(x, gamma, y, rows, dim, eps)
        elif call == "default":
            ops.rmsnorm(x, gamma, y, rows, dim)
        elif call == "keyword":
            ops.rmsnorm(x, gamma, y, rows=rows, dim=dim)
        else:
            ops.rmsnorm(x, gamma, y, rows, dim, 1)
    stream.synchronize()
    assert torch.equal(y, want)


def test_binding_masks_and_status():
    s = torch.randn(4, 24, device="cuda")
    mask = torch.rand(4, 24, device="cuda") > 0.3
    a, b = s.clone(), s.clone()
    ops.masked_softmax_inplace(a, mask, 4, 24, 4)
    ops.masked_softmax_inplace(b, mask.to(torch.uint8), 4, 24, 4)
    assert torch.equal(a, b)
    x, gamma, y, rows, dim = _norm_args()
    with pytest.raises(ops.RfkError) as e:
        ops.rmsnorm(x, gamma, None, rows, dim)          # the C side's own check
    assert "rfk_rmsnorm failed" in str(e.value)
    for bad, text in ((x.float(), "x must be torch.float16"), (x.cpu(), "x must be a CUDA tensor"),
                      (torch.empty(dim, rows, device="cuda", dtype=torch.float16).t(), "x must be contiguous")):
        with pytest.raises(ValueError, match=text):
            ops.rmsnorm(bad, gamma, y, rows, dim)
