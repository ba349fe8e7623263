"""Which output heads are multiplied in splits of K (``gemm.pick_splits_f32``)."""
import pytest


@pytest.mark.parametrize("t", [1, 8, 32, 64])
def test_heads_are_split_where_a_wave_is_nearly_empty_only(t):
    """Partial sums of a head that fills its waves cost more than they save: a whole vocabulary is not split, a slice one tile past the
    SMs is, while its rows are few."""
    from deepseek_v4_2080ti_b200.ops import gemm
    for n in (25600, 37888, 38016, 50304, 75968, 129280, 151936, 248320):
        assert gemm.pick_splits_f32(t, n, 5120) == 1, n
    assert gemm.pick_splits_f32(t, 18944, 5120) == 1                    # 148 tiles
    assert tuple(gemm.pick_splits_f32(t, n, 5120) for n in (18992, 19456)) == {1: (3, 3), 8: (3, 3), 32: (3, 2), 64: (1, 1)}[t]
