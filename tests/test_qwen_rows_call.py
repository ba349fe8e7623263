"""The call that issues a prompt portion natively refuses tables of another layout than its own."""
import ctypes

import pytest


@pytest.mark.parametrize("layer_words,row_words,ok", [(25, 27, True), (24, 27, False), (25, 26, False), (26, 27, False), (25, 28, False)])
def test_tables_of_other_sizes_are_refused(layer_words, row_words, ok):
    from deepseek_v4_2080ti_b200.ops import _lib
    table, run = (ctypes.c_longlong * 50)(), (ctypes.c_longlong * 30)()
    run[:7] = 40, 256, 512, 2, 1, 1, 2                    # tokens, hidden, feed-forward, heads
    f = ctypes.c_float(1e-6)
    rc = _lib.lib().b200_qwen_rows(table, 2, layer_words, run, row_words, f, f, None)     # no scratch: plans only
    assert (rc == 0 and run[24] > 0) if ok else rc == -6
