"""4-bit and GGUF expert matrices in the weight-decoding GEMM (csrc/kernels/gemm_wdec_kernel.cuh): every token-tile width has its
own number of decoded slots and raw stages, and a CTA carries their phases from one tile to the next."""
import pytest
import torch

from deepseek_v4_2080ti_b200.formats import fp4 as fp4fmt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,hidden,inter", [(1, 192, 64), (12, 320, 192), (40, 64, 320), (100, 448, 128), (300, 192, 192)])
def test_fp4_experts_with_odd_k_blocks(rows, hidden, inter):
    """``rows`` tokens, all of them through each of 5 experts: token tiles of 16 to 256."""
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    torch.manual_seed(rows + hidden)
    e = 5
    mats = lambda n, k: [fp4fmt.quantize(torch.randn(n, k, device="cuda") * 0.1 * 2.0 ** (3 * i - 6)) for i in range(e)]
    w13, w2 = mats(2 * inter, hidden), mats(hidden, inter)
    x = torch.randn(rows, hidden, device="cuda").bfloat16()
    idx = torch.arange(e, device="cuda", dtype=torch.int32).repeat(rows, 1)
    wts = torch.rand(rows, e, device="cuda")
    args = (x, idx, wts, moe.ExpertWeights.from_fp4(*map(list, zip(*w13))), moe.ExpertWeights.from_fp4(*map(list, zip(*w2))), 0)
    y, again = moe.experts_forward(*args), moe.experts_forward(*args)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = torch.zeros(rows, hidden, dtype=torch.float64, device="cuda")
    for i in range(e):
        a, b = (fp4fmt.dequantize(*m[i]).double() for m in (w13, w2))
        gu = (x.double() @ a.t()).bfloat16().double()
        act = (torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]).bfloat16().double()
        ref += wts[:, i, None].double() * (act @ b.t()).bfloat16().double()
    # three roundings to bf16 on the way (2^-9 each at most, here of equal size on both sides) and one at the end
    assert ((y.double() - ref).norm() / ref.norm()).item() < 4 * 2.0 ** -9
    assert torch.equal(y, again)


# (tokens, hidden, expert width): 24 experts, six for each token, so 2, 24, 50, 100 and 250 rows an expert - token tiles of 16, 32,
# 64, 128 and 256.  The long side of a product is three times as many k-blocks as the deepest ring has stages (16), and the other
# product more work items than there are SMs, so that CTAs go from tile to tile with every phase of both rings; odd counts of
# k-blocks where the format has them.
LONG = [(8, 3136, 448), (8, 448, 3136), (96, 3136, 448), (96, 448, 3136), (200, 3136, 448), (400, 3136, 320), (1000, 3136, 192)]


def _through_experts(t, hidden, inter, w13, w2, values13, values2):
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    e, k = w13.experts, 6
    torch.manual_seed(t)
    x = torch.randn(t, hidden, device="cuda").bfloat16()
    idx = torch.rand(t, e, device="cuda").topk(k).indices.int().contiguous()
    wts = torch.rand(t, k, device="cuda")
    ys = [moe.experts_forward(x, idx, wts, w13, w2, 0) for _ in range(4)]
    torch.cuda.synchronize()
    _lib.check_status()
    ref = torch.zeros(t, hidden, dtype=torch.float64, device="cuda")
    for i in range(e):
        at, slot = (idx == i).nonzero(as_tuple=True)
        if at.numel() == 0:
            continue
        gu = (x[at].double() @ values13(i).t()).bfloat16().double()
        act = (torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]).bfloat16().double()
        ref.index_add_(0, at, wts[at, slot, None].double() * (act @ values2(i).t()).bfloat16().double())
    # three roundings to bf16 on the way (2^-9 each at most, here of equal size on both sides) and one at the end
    assert ((ys[0].double() - ref).norm() / ref.norm()).item() < 4 * 2.0 ** -9
    assert all(torch.equal(y, ys[0]) for y in ys[1:])


@pytest.mark.parametrize("t,hidden,inter", LONG)
def test_fp4_experts_over_many_stages_and_tiles(t, hidden, inter):
    from deepseek_v4_2080ti_b200.ops import moe
    torch.manual_seed(hidden)
    mats = lambda n, k: [fp4fmt.quantize(torch.randn(n, k, device="cuda") * 0.1) for _ in range(24)]
    w13, w2 = mats(2 * inter, hidden), mats(hidden, inter)
    _through_experts(t, hidden, inter, moe.ExpertWeights.from_fp4(*map(list, zip(*w13))), moe.ExpertWeights.from_fp4(*map(list, zip(*w2))),
                     lambda i: fp4fmt.dequantize(*w13[i]).double(), lambda i: fp4fmt.dequantize(*w2[i]).double())


@pytest.mark.parametrize("types", [("Q4_K", "Q2_K"), ("Q2_K", "Q4_K"), ("Q5_K", "Q6_K"), ("Q8_0", "Q3_K")])
@pytest.mark.parametrize("t,hidden,inter", [(8, 3328, 512), (96, 512, 3328), (200, 3328, 512), (400, 3328, 256)])
def test_gguf_experts_over_many_stages_and_tiles(types, t, hidden, inter):
    from deepseek_v4_2080ti_b200.formats import gguf as G
    from deepseek_v4_2080ti_b200.ops import moe
    torch.manual_seed(hidden)
    ty = [G.GGMLType[n] for n in types]
    raw = [[G.quantize(torch.randn(n, k, device="cuda") * 0.1, q) for _ in range(4)] for q, n, k in ((ty[0], 2 * inter, hidden), (ty[1], hidden, inter))]
    w13, w2 = (moe.ExpertWeights.from_gguf(r * 6, q, n, k) for r, q, n, k in ((raw[0], ty[0], 2 * inter, hidden), (raw[1], ty[1], hidden, inter)))
    # the kernel rounds decoded weights to bf16
    value = lambda j, k: [G.dequantize(r, ty[j], k).bfloat16().double() for r in raw[j]]
    v13, v2 = value(0, hidden), value(1, inter)
    _through_experts(t, hidden, inter, w13, w2, lambda i: v13[i % 4], lambda i: v2[i % 4])


def test_fp4_codes_and_scales_over_their_range():
    """Every code under scales from 2^-127 up, through a one-hot input: the weight itself comes out, in bf16."""
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    n, k = 128, 64
    codes = torch.arange(n * k, device="cuda").view(n, k) % 16
    packed = (codes[:, 0::2] | codes[:, 1::2] << 4).to(torch.uint8)
    scale = (torch.arange(n * 2, device="cuda").view(n, 2) * 149 // 255).to(torch.uint8)           # exponents 0 .. 148
    w = fp4fmt.level_table("cuda")[codes].double() * torch.exp2(scale.double() - 127).repeat_interleave(32, 1)
    ew = moe.ExpertWeights.from_fp4([packed], [scale])
    x = torch.eye(k, device="cuda").bfloat16()
    idx = torch.zeros(k, 1, dtype=torch.int32, device="cuda")
    # the first product alone: the grouped GEMM over the plan of one expert
    i32 = lambda *s: torch.empty(*s, dtype=torch.int32, device="cuda")
    off, rr, rt, wk, nw, wk2, nw2 = i32(2), i32(k, 1), i32(k), i32(64, 4), i32(1), i32(64, 4), i32(1)
    L, p, s = _lib.lib(), _lib.ptr, _lib.stream()
    _lib.check(L.b200_moe_plan(p(idx), k, 1, 0, 1, p(off), p(rr), p(rt), p(wk), p(nw), 1, 64, p(wk2), p(nw2), 1, 64, 64, s), "plan")
    out = torch.empty(k, n, dtype=torch.bfloat16, device="cuda")
    _lib.check(L.b200_gemm_wdec_grouped(ew.wfmt, p(ew.weight), p(ew.scales), p(x), p(out), k, n, k, 1, p(wk), p(nw), 64,
                                        p(_lib.status_word(x.device)), s), "grouped")
    torch.cuda.synchronize()
    _lib.check_status()
    got, want = out.t().double(), w
    normal = want.abs() >= 2.0 ** -126
    assert torch.equal(got[normal], want[normal]) and (got[~normal].abs() <= 2.0 ** -125).all()
