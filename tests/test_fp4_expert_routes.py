"""Which route block-scaled FP4 experts take (``moe.fp4_terms_pay``)."""
import pytest

from deepseek_v4_2080ti_b200.ops import moe


def _pay(experts, h, inter, rows, total=None):
    w13, w2 = (moe.ExpertWeights(moe.WF_FP4, None, None, n, k, experts) for n, k in ((2 * inter, h), (h, inter)))
    assert w13.block_scaled and w2.block_scaled
    return moe.fp4_terms_pay(rows, total or experts, w13, w2)


@pytest.mark.parametrize("experts,h,inter", [(256, 4096, 2048), (32, 4096, 2048), (256, 7168, 2048), (128, 6144, 1024)])
def test_many_experts(experts, h, inter):
    assert all(_pay(experts, h, inter, r) for r in (6, 64, 1000, 64 * experts, 160 * experts))
    assert not any(_pay(experts, h, inter, r) for r in (161 * experts, 1000 * experts))


def test_few_experts_fill_the_tiles_of_unpacked_weights_sooner():
    assert _pay(8, 4096, 2048, 2) and _pay(8, 4096, 2048, 64 * 8)
    assert not _pay(8, 4096, 2048, 65 * 8)


def test_small_blocks_stay_unpacked():
    assert not any(_pay(8, 2048, 768, r) for r in (1, 8, 64, 1000))
    assert not _pay(64, 2048, 768, 8) and _pay(64, 2048, 768, 16)


def test_rows_of_experts_held_elsewhere_do_not_count():
    assert not _pay(32, 4096, 2048, 12000) and _pay(32, 4096, 2048, 12000, total=256)
