"""FP4 experts of one block have one shape."""
import pytest
import torch

from deepseek_v4_2080ti_b200.ops import moe


def _matrix(n, k):
    return torch.randint(0, 256, (n, k // 2), dtype=torch.uint8), torch.randint(0, 256, (n, k // 32), dtype=torch.uint8)


# one block of rows or of inputs beside several of them, in both layouts
@pytest.mark.parametrize("first,other", [((256, 384), (128, 384)), ((256, 384), (256, 128)), ((128, 384), (256, 384)), ((128, 128), (128, 384)),
                                         ((256, 192), (256, 64)), ((256, 192), (128, 192)), ((128, 384), (128, 192))])
def test_another_shape_beside_the_first_is_refused(first, other):
    with pytest.raises((RuntimeError, ValueError, AssertionError)):
        moe.ExpertWeights.from_fp4(*map(list, zip(_matrix(*first), _matrix(*other))))


def test_scales_of_another_matrix_are_refused():
    (q, s), (_, s2) = _matrix(128, 384), _matrix(128, 128)
    with pytest.raises((RuntimeError, ValueError, AssertionError)):
        moe.ExpertWeights.from_fp4([q, q], [s, s2])
