"""CPU tests of the rule that sends a head-split projection to small tiles or to CTA pairs (rfk_gemm_heads_tile, host only): the
smallest tile whose CTAs all run at once, and never one that the device cannot place."""
import ctypes

import pytest

import renderformer_cuda_b200 as pkg  # noqa: F401
from renderformer_cuda_b200 import _abi

TILES = ((64, 64), (128, 64), (128, 128))


def _tile(M, N, resident):
    return _abi.load("rfk.h").rfk_gemm_heads_tile(M, N, (ctypes.c_int * 3)(*resident))


@pytest.mark.parametrize("M", [1, 32, 64, 65, 256, 576, 577, 1024, 1600, 2304, 4096])
@pytest.mark.parametrize("N", [256, 1024, 3072])
@pytest.mark.parametrize("resident", [(132, 132, 140), (0, 132, 140), (132, 0, 0), (0, 0, 140), (0, 0, 0), (4, 4, 2)])
def test_smallest_tile_that_runs_at_once(M, N, resident):
    fits = [i + 1 for i, (bm, bn) in enumerate(TILES) if -(-M // bm) * -(-N // bn) <= resident[i]]
    got = _tile(M, N, resident)
    assert got == (fits[0] if fits else 0)
    assert got == 0 or resident[got - 1] > 0          # a cluster that cannot be placed: the pair kernel, not a failing launch


def test_bad_arguments():
    assert _tile(0, 256, (1, 1, 1)) == -1 and _tile(64, 0, (1, 1, 1)) == -1
    assert _abi.load("rfk.h").rfk_gemm_heads_tile(64, 256, None) == -1


@pytest.mark.parametrize("pairs", [1, 7, 60, 66, 74])
@pytest.mark.parametrize("M,N", [(1, 8), (257, 200), (2500, 1024), (4096, 1024), (4864, 1024), (5665, 1024), (5120, 768), (3136, 3072), (60000, 192)])
def test_pair_tiles_are_narrow_where_the_placed_pairs_need_no_more_rounds(M, N, pairs):
    """The rounds are those of the pairs that the device runs at once, which a launch is limited to, not of half its SMs."""
    rounds = lambda cols: -(-(-(-M // 256) * -(-N // cols)) // pairs)
    got = _abi.load("rfk.h").rfk_gemm_pair_tile(M, N, pairs)
    assert got == (192 if rounds(192) == rounds(256) else 256)


def test_pair_tile_without_a_pair_is_refused():
    tile = _abi.load("rfk.h").rfk_gemm_pair_tile
    assert tile(4096, 1024, 0) == tile(4096, 1024, -1) == tile(0, 8, 74) == tile(8, 0, 74) == -1
