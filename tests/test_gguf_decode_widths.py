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


@pytest.mark.gpu
@pytest.mark.parametrize("t", [256, 700])
@pytest.mark.parametrize("tname", ["Q4_K", "Q2_K"])
def test_weights_are_rounded_once_and_to_bf16(tname, t):
    """Identity rows give the weights themselves: scale x code - minimum in one fp32 step, then bf16, whatever the minimum is beside
    the scale.  (With an offset of the codes folded into the minimum, a minimum far below its scale loses bits.)  Tiles of up to 128 rows
    and of 256: the identity 32 rows at a time, and all of it."""
    from deepseek_v4_2080ti_b200.formats import gguf as G
    from deepseek_v4_2080ti_b200.ops import _lib, gguf_gemm
    ty, n, k = G.GGMLType[tname], 384, 256
    g = torch.Generator(device="cuda").manual_seed(t)
    bits = lambda *s: torch.randint(0, 256, s, generator=g, device="cuda", dtype=torch.uint8)
    d, dmin = (torch.exp2(torch.rand(n, generator=g, device="cuda") * 14 - lo).half() for lo in (8, 14))
    two = lambda v: v.view(torch.uint8).view(n, 2)
    if tname == "Q4_K":
        s, q = bits(n, 12), bits(n, 128)
        raw = torch.cat([two(d), two(dmin), s, q], 1)
        s = s.long()
        sc = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6) << 4], 1)
        mn = torch.cat([s[:, 4:8] & 63, s[:, 8:] >> 4 | (s[:, 4:8] >> 6) << 4], 1)
        code = torch.stack([q.view(n, 4, 32) & 15, q.view(n, 4, 32) >> 4], 2).view(n, 8, 32)
    else:
        s, q = bits(n, 16), bits(n, 64)
        raw = torch.cat([s, q, two(d), two(dmin)], 1)
        sc, mn = (s & 15).long(), (s >> 4).long()
        code = torch.stack([q.view(n, 2, 32) >> 2 * j & 3 for j in range(4)], 2).view(n, 16, 16)
    sc, mn = ((a.float()[:, None] * b.float()).double() for a, b in ((d, sc), (dmin, mn)))           # one fp32 rounding each
    want = (sc[..., None] * code.double() - mn[..., None]).float().bfloat16().float().view(n, k)
    w = gguf_gemm.GGUFLinear.from_raw(raw.contiguous(), ty, n, k)
    eye = torch.eye(k, device="cuda").bfloat16()
    assert torch.equal(gguf_gemm.linear(torch.cat([eye, eye.new_zeros(t - k, k)]), w, out_f32=True)[:k].t(), want)
    for i in range(0, k, 32):
        assert torch.equal(gguf_gemm.linear(eye[i:i + 32].contiguous(), w, out_f32=True).t(), want[:, i:i + 32])
    torch.cuda.synchronize()
    _lib.check_status()
