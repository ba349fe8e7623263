"""Where FP4 codes and scales go in the two layouts of ``moe.prepack_fp4``."""
import pytest
import torch

from deepseek_v4_2080ti_b200.ops import moe


@pytest.mark.parametrize("n,k", [(128, 128), (200, 384), (384, 1024), (256, 192), (130, 64)])
def test_layout_byte_by_byte(n, k):
    torch.manual_seed(n + k)
    q, s = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8), torch.randint(0, 256, (n, k // 32), dtype=torch.uint8)
    out = moe.prepack_fp4(q, s)
    bk = 128 if k % 128 == 0 else 64
    assert out.shape == ((n + 127) // 128, k // bk, bk * 68) and out.is_contiguous()
    for r in range(0, n, 7):
        for j in range(0, k // 2, 5):                      # byte j: inputs 2 j and 2 j + 1
            b, i = divmod(2 * j, bk)
            at = (i // 32 * 128 + r % 128) * 16 + i % 32 // 2 if bk == 128 else r % 128 * 32 + i // 2
            assert out[r // 128, b, at] == q[r, j]
        for g in range(k // 32):
            b, i = divmod(32 * g, bk)
            at = bk * 64 + (16 * (r % 32) + 4 * (r % 128 // 32) + i // 32 if bk == 128 else r % 128 * 2 + i // 32)
            assert out[r // 128, b, at] == (min(int(s[r, g]), 254) if bk == 128 else s[r, g])
    pad = out[-1].view(k // bk, -1)[:, :bk * 64].view(k // bk, -1, 128, 16 if bk == 128 else 32)[:, :, (n - 1) % 128 + 1:]
    assert not pad.any()
    stacked = moe.ExpertWeights.from_fp4([q, q.flip(0), q], [s, s, s.flip(1)])
    assert all(torch.equal(stacked.weight[i], moe.prepack_fp4(a, b)) for i, (a, b) in enumerate([(q, s), (q.flip(0), s), (q, s.flip(1))]))
