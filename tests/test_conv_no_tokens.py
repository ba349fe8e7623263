"""A causal convolution over no tokens: nothing to do, and no error."""
import pytest


@pytest.mark.parametrize("tokens,kw,channels,rc", [(0, 4, 264, 0), (0, 3, 264, -6), (0, 4, 260, -6)])
def test_no_tokens_leave_everything_as_it_is(tokens, kw, channels, rc):
    from deepseek_v4_2080ti_b200.ops import _lib
    assert _lib.lib().b200_conv_silu(None, channels, None, None, None, channels, tokens, channels, kw, 1, None) == rc
