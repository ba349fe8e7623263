"""GGUF weights decoded into tensor memory: the token tiles that take that path, up to the first that does not, for every format."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("tname", ["Q8_0", "Q4_K", "Q5_K", "Q6_K", "Q3_K", "Q2_K", "IQ1_M", "IQ2_XXS", "IQ2_XS", "IQ3_XXS", "IQ4_XS"])
@pytest.mark.parametrize("t", [16, 17, 64, 65, 128, 129])
def test_token_tiles(tname, t):
    from deepseek_v4_2080ti_b200.formats import gguf as G
    from deepseek_v4_2080ti_b200.ops import _lib, gguf_gemm
    ty, n, k = G.GGMLType[tname], 200, 1280                 # a ragged feature tile, 20 k-blocks: more than a ring holds
    torch.manual_seed(t)
    raw = G.quantize(torch.randn(n, k, device="cuda") * 0.05, ty)
    w = G.dequantize(raw, ty, k).bfloat16().double()
    x = torch.randn(t, k, device="cuda").bfloat16()
    y = gguf_gemm.linear(x, gguf_gemm.GGUFLinear.from_raw(raw, ty, n, k), out_f32=True)
    torch.cuda.synchronize()
    _lib.check_status()
    want = x.double() @ w.t()
    # Both sides round the decoded weights to bf16, and differ where their fp32 steps put a value on the other side of a tie: one
    # weight in 2^10 or so by 2^-8 of itself (2^-8 * 2^-5 = 2^-13 of a sum); fp32 sums of 1280 products stay below that too.
    assert ((y.double() - want).norm() / want.norm()).item() < 2.0 ** -12
