"""CPU tests of the operators' compiled binding: where it is missing or was built for another torch, the checked function behind
an operator serves it (and its argument errors), and this is said once. A bound operator is copied and pickled like the function
it stands for."""
import copy
import pickle
import sys
import warnings

import pytest
import torch

import renderformer_cuda_b200 as pkg

ops = pkg.ops


@pytest.fixture
def unbound(monkeypatch):
    """ops as before its first call, with one operator to call."""
    ops._binding.cache_clear()
    monkeypatch.setattr(ops, "silu", ops.silu)
    yield ops._native(ops.silu.__wrapped__)
    ops._binding.cache_clear()


def _refused(op):
    x = torch.zeros(8, dtype=torch.float16)
    with pytest.raises(ValueError, match="CUDA tensor"):   # the checked function's own refusal
        op(x, x, 8)


def test_without_the_binding(unbound, monkeypatch):
    import renderformer_cuda_b200
    monkeypatch.setitem(sys.modules, "renderformer_cuda_b200._native", None)
    monkeypatch.delattr(renderformer_cuda_b200, "_native", raising=False)
    with pytest.warns(RuntimeWarning, match="not built"):
        _refused(unbound)
    assert ops.silu.__name__ == "silu" and not type(ops.silu).__name__ == "Op"
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        _refused(unbound)


def test_binding_of_another_torch(unbound, monkeypatch):
    monkeypatch.setattr(torch, "__version__", "0.1")
    with pytest.warns(RuntimeWarning, match="this is torch 0.1"):
        _refused(unbound)


def test_binding_of_this_torch_is_used(unbound):
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        _refused(unbound)
    assert type(ops.silu).__name__ == "Op"


@pytest.mark.parametrize("bound", [False, True])
def test_operators_are_copied_and_pickled_by_name(bound):
    """A program keeps an operator in an object that it copies, or hands it to another process."""
    if bound:
        _refused(ops.silu)
    assert (type(ops.silu).__name__ == "Op") >= bound
    assert pickle.loads(pickle.dumps(ops.silu)) is ops.silu
    assert copy.deepcopy({"act": ops.silu})["act"] is ops.silu and copy.copy(ops.silu) is ops.silu
