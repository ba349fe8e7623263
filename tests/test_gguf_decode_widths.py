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


@pytest.mark.gpu
@pytest.mark.parametrize("tname,d,dmin,scales,codes,ones,zero", [("Q4_K", 0, 2, 4, 16, 0x33, 0x30), ("Q2_K", 80, 82, 0, 16, 0xFF, 0xFC)])
@pytest.mark.parametrize("t", [3, 200])
def test_infinite_block_scale(tname, d, dmin, scales, codes, ones, zero, t):
    """A block scale of infinity: infinite where every code is above zero, not a number where one is zero, other rows as they were."""
    from deepseek_v4_2080ti_b200.formats import gguf as G
    from deepseek_v4_2080ti_b200.ops import _lib, gguf_gemm
    ty, n, k = G.GGMLType[tname], 128, 512
    torch.manual_seed(t)
    raw = G.quantize(torch.randn(n, k, device="cuda") * 0.05, ty)
    rows = raw.view(torch.uint8).view(n, -1)
    for row in (5, 6):
        rows[row, d:d + 2] = torch.tensor([0x00, 0x7C], dtype=torch.uint8, device="cuda")
        rows[row, dmin:dmin + 2] = 0
        rows[row, scales:scales + (12 if tname == "Q4_K" else 16)] = 1
        rows[row, codes:codes + (128 if tname == "Q4_K" else 64)] = ones
    rows[6, codes + 7] = zero
    x = torch.rand(t, k, device="cuda").add(0.5).bfloat16()
    y = gguf_gemm.linear(x, gguf_gemm.GGUFLinear.from_raw(raw, ty, n, k), out_f32=True)
    torch.cuda.synchronize()
    _lib.check_status()
    assert (y[:, 5] == float("inf")).all() and y[:, 6].isnan().all()
    assert y[:, :5].isfinite().all() and y[:, 7:].isfinite().all()
