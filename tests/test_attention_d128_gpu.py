"""tcgen05 attention with 128-wide heads (two swizzle sub-tiles per operand row, two score buffers): tile edges, padded
keys, the key split and its merge, row statistics, and a running reference that turns out wrong. Oracle: torch fp32
attention on the same fp16 inputs. Tolerance: probabilities and outputs are rounded to fp16 (2^-11 each) and up to 2^8 of
reference slack does not change a relative rounding, so an output of magnitude up to 4 is within 4e-3 + 4e-3 |want|."""
import ctypes

import pytest
import torch

import renderformer_cuda_b200 as pkg
from renderformer_cuda_b200 import _abi

pytestmark = pytest.mark.gpu
D = 128


@pytest.fixture(autouse=True)
def tc_path():
    pkg.ops.flash_attention_error(clear=True)
    pkg.ops.flash_attention_set_path(2)      # the tcgen05 kernel or an error
    yield
    pkg.ops.flash_attention_set_path(0)
    torch.cuda.synchronize()
    assert pkg.ops.flash_attention_error(clear=True) == 0


def _qkv(B, Hh, Sq, Sk, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(Sq * 31 + Sk)
    return tuple((torch.randn(B, Hh, n, D, device="cuda", generator=g) * s).half() for n, s in ((Sq, scale), (Sk, scale), (Sk, 1.0)))


def _close(got, want, what):
    err = (got.float() - want.float()).abs()
    assert torch.isfinite(got.float()).all(), what
    assert (err <= 4e-3 + 4e-3 * want.float().abs()).all(), f"{what}: max error {err.max().item():.2e}"
    assert err.mean() < 5e-4, f"{what}: mean error {err.mean().item():.2e}"


def _ex(q, k, v, o, B, Hh, Sq, Sk, n_keys, D, q_row_ss=None, ss_tiles=0, norm_dim=0, workspace=None, v_shared=False):
    """What the layers call: flash_attention_ex for both head sizes (the public form takes 64-wide heads)."""
    lib = _abi.load("rfk.h")
    fn = lib.rfk_flash_attention_ex_wide
    fn.argtypes, fn.restype = lib.rfk_flash_attention_ex.argtypes, ctypes.c_int
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())
    rc = fn(p(q), p(k), p(v), p(o), p(q_row_ss), ss_tiles, norm_dim, pkg.ops.K_EPS_FP16, p(workspace),
            0 if workspace is None else workspace.numel(), int(v_shared), B, Hh, Sq, Sk, n_keys, D, 0, D ** -0.5,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, rc


def _want(Q, K, V, n_keys):
    return torch.nn.functional.scaled_dot_product_attention(Q.float(), K[:, :, :n_keys].float(), V[:, :, :n_keys].float())


@pytest.mark.parametrize("B,Hh,Sq,Sk,n_keys,scale", [
    (1, 1, 128, 64, 64, 1.0), (1, 2, 129, 128, 65, 1.0), (1, 1, 1, 5, 3, 1.0), (2, 3, 300, 1000, 993, 1.0),
    (1, 2, 256, 384, 384, 1.0), (1, 8, 512, 2048, 2041, 2.0)])
def test_matches_fp32_attention(B, Hh, Sq, Sk, n_keys, scale):
    Q, K, V = _qkv(B, Hh, Sq, Sk, scale)
    O = torch.full_like(Q, 7.0)
    pkg.ops.flash_attention(Q, K, V, O, B, Hh, Sq, Sk, n_keys, D)
    _close(O, _want(Q, K, V, n_keys), "whole units")
    O2 = torch.full((B, Sq, Hh * D), 7.0, device="cuda", dtype=torch.float16)
    pkg.ops.flash_attention(Q, K, V, O2, B, Hh, Sq, Sk, n_keys, D, o_bshd=True)
    assert torch.equal(O2.view(B, Sq, Hh, D).permute(0, 2, 1, 3), O)


@pytest.mark.parametrize("B,Hh,Sq,Sk,n_keys", [(1, 1, 256, 4096, 4096), (1, 8, 700, 3000, 2995), (3, 2, 256, 2600, 2593), (1, 8, 4672, 3000, 2995)])
def test_key_split_merges_and_repeats(B, Hh, Sq, Sk, n_keys):
    Q, K, V = _qkv(B, Hh, Sq, Sk)
    ws = pkg.ops.flash_attention_workspace()
    outs = []
    for _ in range(2):
        O = torch.full_like(Q, 7.0)
        _ex(Q, K, V, O, B, Hh, Sq, Sk, n_keys, D, workspace=ws)
        outs.append(O)
    _close(outs[0], _want(Q, K, V, n_keys), "split")
    assert torch.equal(outs[0], outs[1]) and not ws[:1024].any()


def test_row_statistics_and_shared_values():
    B, Hh, Sq, Sk, n_keys = 2, 2, 320, 500, 491
    Q, K, V = _qkv(B, Hh, Sq, Sk)
    Q = (Q.float() * 3).half()
    dim = Hh * D
    rows = Q.permute(0, 2, 1, 3).reshape(B * Sq, dim).float()
    ss = torch.stack([rows[:, :128].pow(2).sum(-1), rows[:, 128:].pow(2).sum(-1)], -1).contiguous()
    O = torch.empty_like(Q)
    _ex(Q, K, V[0].contiguous(), O, B, Hh, Sq, Sk, n_keys, D, q_row_ss=ss, ss_tiles=2, norm_dim=dim,
                               v_shared=True)
    rinv = torch.rsqrt(ss.sum(-1) / dim + pkg.ops.K_EPS_FP16).view(B, 1, Sq, 1)
    _close(O, _want(Q.float() * rinv, K, V[:1].expand(B, -1, -1, -1), n_keys), "row statistics")


@pytest.mark.parametrize("boost", [60.0, 250.0])
def test_running_reference_is_wrong(boost):
    """Keys that beat the running reference by far (2^65) and by more than fp32's range (2^128), in columns of both
    exponential paths, and scores that rise along all keys."""
    B, Hh, Sq, Sk = 1, 2, 256, 1024
    Q, K, V = _qkv(B, Hh, Sq, Sk)
    d = torch.nn.functional.normalize(Q.float().mean(2, keepdim=True), dim=-1)
    Q = (Q.float() + 6.0 * d).half()
    Kf = K.float() + 40.0 * torch.linspace(0.0, 1.0, Sk, device="cuda").view(1, 1, Sk, 1) * d
    Kf[:, :, 64 * 3 + 8, :] += boost * d[:, :, 0, :]
    Kf[:, :, 64 * 9 + 3, :] += 1.5 * boost * d[:, :, 0, :]
    K = Kf.half()
    O = torch.full_like(Q, 7.0)
    pkg.ops.flash_attention(Q, K, V, O, B, Hh, Sq, Sk, Sk, D)
    _close(O, _want(Q, K, V, Sk), "wrong reference")


def _distance(O, Q, K, V, n_keys):
    """Distance of O from the attention of the same fp16 inputs in 64 bits, relative (2-norm)."""
    err = ref = 0.0
    for b in range(Q.shape[0]):
        for h in range(Q.shape[1]):
            p = torch.softmax(Q[b, h].double() @ K[b, h, :n_keys].double().t() * D ** -0.5, -1)
            want = p @ V[b, h, :n_keys].double()
            err, ref = err + float((O[b, h].double() - want).pow(2).sum()), ref + float(want.pow(2).sum())
    return (err / ref) ** 0.5


@pytest.mark.parametrize("split", [False, True], ids=["whole", "split"])
@pytest.mark.parametrize("B,Hh,Sq,Sk,n_keys,scale", [
    (1, 8, 1600, 4608, 4607, 1.0), (2, 3, 300, 1000, 993, 1.0), (1, 8, 1024, 1536, 1532, 2.0), (1, 4, 700, 3000, 2995, 3.0)])
def test_no_further_from_64_bits_than_the_mma_kernel(B, Hh, Sq, Sk, n_keys, scale, split):
    """Both kernels round the same probabilities (relative to the row's running maximum, exponentials of the special-function
    unit) and the same outputs to fp16; what is left is the order of fp32 sums, 2^-24 against roundings of 2^-11. Measured
    on whole units: equal to 1e-4, and 1.03 to 1.21 with a reference that trails the maximum. A piece of a split unit has a
    maximum of its own."""
    Q, K, V = _qkv(B, Hh, Sq, Sk, scale)
    O, M = torch.empty_like(Q), torch.empty_like(Q)
    _ex(Q, K, V, O, B, Hh, Sq, Sk, n_keys, D, workspace=pkg.ops.flash_attention_workspace() if split else None)
    pkg.ops.flash_attention_set_path(1)
    pkg.ops.flash_attention(Q, K, V, M, B, Hh, Sq, Sk, n_keys, D)
    got, mma = _distance(O, Q, K, V, n_keys), _distance(M, Q, K, V, n_keys)
    print(f"distance from 64 bits: {got:.4e}, mma.sync kernel {mma:.4e}, ratio {got / mma:.4f}")
    assert got <= 1.002 * mma, (got, mma)


@pytest.mark.parametrize("split", [False, True], ids=["whole", "split"])
@pytest.mark.parametrize("n_out", [1, 64, 100, 640, 4096])
def test_keys_with_a_score_of_minus_infinity(n_out, split):
    """Keys switched off through an operand column (1 in every query, -inf in the key): none of a tile, whole tiles from the
    first on, every piece of a unit, every key of a head (output 0, as from the mma.sync kernel)."""
    B, Hh, Sq, Sk = 1, 2, 130, 4096
    Q, K, V = _qkv(B, Hh, Sq, Sk)
    Q[..., -1] = 1.0
    K[..., -1] = 0.0
    K[:, 0, :n_out, -1] = -float("inf")
    O, M = torch.full_like(Q, 7.0), torch.full_like(Q, 7.0)
    _ex(Q, K, V, O, B, Hh, Sq, Sk, Sk, D, workspace=pkg.ops.flash_attention_workspace() if split else None)
    pkg.ops.flash_attention_set_path(1)
    pkg.ops.flash_attention(Q, K, V, M, B, Hh, Sq, Sk, Sk, D)
    assert torch.isfinite(M.float()).all()
    _close(O, M, "keys at -inf")
    if n_out == Sk:
        assert not O[:, 0].any()


@pytest.mark.parametrize("n_out", [64, 640, 1024])
def test_keys_with_a_score_of_minus_infinity_on_64_wide_heads(n_out):
    """The same in the kernel's other form, whose common tile does not take the maximum first."""
    g = torch.Generator(device="cuda").manual_seed(n_out)
    Q, K, V = (torch.randn(1, 2, n, 64, device="cuda", generator=g).half() for n in (130, 1024, 1024))
    Q[..., -1] = 1.0
    K[..., -1] = 0.0
    K[:, 0, :n_out, -1] = -float("inf")
    outs = []
    for path in (2, 1):
        pkg.ops.flash_attention_set_path(path)
        outs.append(torch.full_like(Q, 7.0))
        pkg.ops.flash_attention(Q, K, V, outs[-1], 1, 2, 130, 1024, 1024, 64)
    assert torch.isfinite(outs[1].float()).all()
    _close(outs[0], outs[1], "keys at -inf")
    assert n_out < 1024 or not outs[0][:, 0].any()


def _ordered(q, k, v, o, B, Hh, Sq, Sk, n_keys):
    lib = _abi.load("rfk.h")
    fn = lib.rfk_flash_attention_ordered
    fn.argtypes, fn.restype = [ctypes.c_void_p] * 4 + [ctypes.c_int] * 7 + [ctypes.c_float, ctypes.c_void_p], ctypes.c_int
    rc = fn(*(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, o)), B, Hh, Sq, Sk, n_keys, D, 0, D ** -0.5,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, rc


@pytest.mark.parametrize("B,Hh,Sq,Sk,n_keys,scale", [
    (1, 1, 1, 5, 3, 1.0), (1, 2, 129, 128, 65, 1.0), (1, 2, 64, 64, 64, 1.0), (2, 3, 300, 1000, 993, 2.0), (1, 8, 1600, 1408, 1407, 1.0),
    (1, 8, 4096, 584, 581, 3.0), (3, 40, 257, 300, 290, 1.0)])
def test_ordered_form_has_the_bits_of_the_mma_sync_kernel(B, Hh, Sq, Sk, n_keys, scale):
    """Sessions with an image head keep the bits of the mma.sync kernel: grids of one and of two blocks per CTA, ragged
    queries and keys, references that move in every tile (scores rising along the keys), a row without a finite score."""
    Q, K, V = _qkv(B, Hh, Sq, Sk, scale)
    d = torch.nn.functional.normalize(Q.float().mean(2, keepdim=True), dim=-1)
    K = (K.float() + 4.0 * torch.linspace(0.0, 1.0, Sk, device="cuda").view(1, 1, Sk, 1) * d).half()
    Q[0, 0, Sq // 2] = -float("inf")
    K[0, 0] = K[0, 0].abs() + 0.01
    got, want = torch.full_like(Q, 7.0), torch.full_like(Q, 9.0)
    _ordered(Q, K, V, got, B, Hh, Sq, Sk, n_keys)
    pkg.ops.flash_attention_set_path(1)
    pkg.ops.flash_attention(Q, K, V, want, B, Hh, Sq, Sk, n_keys, D)
    assert torch.equal(got, want)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("Sq,Sk", [(1, 64), (128, 333), (300, 1000)])
def test_one_block_per_cta_has_the_bits_of_two(hd, Sq, Sk):
    """A call whose blocks of 128 queries all find an SM runs one per CTA; the same heads among copies of themselves share
    theirs."""
    g = torch.Generator(device="cuda").manual_seed(Sq)
    Q, K, V = (torch.randn(1, 2, n, hd, device="cuda", generator=g).half() * s for n, s in ((Sq, 4.0), (Sk, 1.0), (Sk, 1.0)))
    alone = torch.empty_like(Q)
    pkg.ops.flash_attention(Q, K, V, alone, 1, 2, Sq, Sk, Sk, hd)
    copies = 100
    Qm, Km, Vm = (t.expand(copies, -1, -1, -1).contiguous() for t in (Q, K, V))
    many = torch.empty_like(Qm)
    pkg.ops.flash_attention(Qm, Km, Vm, many, copies, 2, Sq, Sk, Sk, hd)
    assert torch.equal(many, alone.expand(copies, -1, -1, -1))


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("windows,heads", [(1, 1), (4, 8), (25, 3)])
def test_window_attention_of_128_wide_heads_has_the_bits_of_the_separate_steps(windows, heads, masked):
    """Sessions with an image head: library Q K^T with the scale as its alpha, swin softmax over the score matrix, library P V
    and a transpose, against the one kernel. Rows of large scores, a window whose mask leaves single keys, a row of nothing."""
    g = torch.Generator(device="cuda").manual_seed(windows * 10 + heads)
    BH, scale = windows * heads, D ** -0.5
    Q, K, V = (torch.randn(BH, 64, D, device="cuda", generator=g).half() for _ in range(3))
    Q[:, 10:20] *= 8
    mask = None
    if masked:
        mask = (torch.rand(windows, 64, 64, device="cuda", generator=g) < 0.5).to(torch.uint8)
        mask[0] = torch.eye(64, device="cuda", dtype=torch.uint8)
        mask[0, 5] = 0
    scores = (torch.bmm(Q, K.transpose(1, 2), out_dtype=torch.float32) * scale).contiguous()
    pkg.ops.swin_softmax_probs_inplace(scores, mask, windows, heads, 64, windows)
    P = scores.view(torch.float16).view(BH, 64, 128)[:, :, :64].contiguous()
    want = torch.bmm(P, V).view(windows, heads, 64, D).permute(0, 2, 1, 3).reshape(windows * 64, heads * D)
    got = torch.full_like(want, 7.0)
    fn = _abi.load("rfk.h").rfk_window_attention_steps
    fn.argtypes, fn.restype = [ctypes.c_void_p] * 5 + [ctypes.c_int] * 3 + [ctypes.c_float, ctypes.c_void_p], ctypes.c_int
    rc = fn(*(ctypes.c_void_p(0 if t is None else t.data_ptr()) for t in (Q, K, V, got, mask)), windows, heads, windows, scale,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0 and torch.equal(got, want)
