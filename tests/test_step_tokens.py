"""The tokens that a decode step of the hybrid decoder is given: which shapes it takes."""
import pytest
import torch

from deepseek_v4_2080ti_b200.models.qwen_hybrid import _step_ids


@pytest.mark.parametrize("shape", [(3,), (1,), ()])
def test_one_token_each_or_one_for_all(shape):
    ids = torch.arange(5, 5 + max(1, torch.Size(shape).numel()), dtype=torch.int64).reshape(shape)
    got = _step_ids(ids, 3, "cpu")
    assert got.dtype == torch.int32 and got.is_contiguous() and torch.equal(got, ids.expand(3).int())


# what a copy into a vector of three takes no other way: a matrix of three values is not three tokens
@pytest.mark.parametrize("shape", [(3, 1), (1, 3), (1, 1), (1, 1, 3), (6,), (2,), (0,)])
def test_other_shapes_are_refused(shape):
    ids = torch.zeros(shape, dtype=torch.int32)
    with pytest.raises(RuntimeError):
        torch.empty(3, dtype=torch.int32).copy_(ids)
    with pytest.raises(RuntimeError):
        _step_ids(ids, 3, "cpu")
