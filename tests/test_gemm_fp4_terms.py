"""Grouped FP4 products on the block-scaled tensor pipe (csrc/kernels/gemm_fp4_terms.cu, mx_terms.cuh)."""
import pytest
import torch

from deepseek_v4_2080ti_b200.formats import fp4 as fp4fmt

pytestmark = pytest.mark.gpu


def _gather(x):
    """Terms of the rows of ``x`` as one expert's: (xq, sf, outside, rest, counters)."""
    from deepseek_v4_2080ti_b200.ops import _lib
    r, k = x.shape
    e = lambda *s, d=torch.int32: torch.empty(*s, dtype=d, device="cuda")
    token, off = torch.arange(r, device="cuda", dtype=torch.int32), torch.tensor([0, r], device="cuda", dtype=torch.int32)
    xq, sf, outside, rest, cnt = e(2, r, k, d=torch.uint8), e(k // 128, r, 4, d=torch.uint8), e(r), e(r, k, d=torch.bfloat16), e(296)
    L, p = _lib.lib(), _lib.ptr
    _lib.check(L.b200_moe_gather_terms(p(x), p(token), p(off), 1, p(xq), p(sf), p(outside), p(rest), r, k, p(cnt), cnt.numel(), _lib.stream()),
               "gather")
    return xq, sf, outside, rest, cnt


def _product(x, q, scale):
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    r, k = x.shape
    n = q.shape[0]
    ew = moe.ExpertWeights.from_fp4([q], [scale])
    xq, sf, outside, rest, cnt = _gather(x)
    (tok, floats, _), mg = moe._fp4_terms_plan(), (n + 255) // 256
    work = torch.tensor([[0, m, r0, min(tok, r - r0)] for m in range(mg) for r0 in range(0, r, tok)], device="cuda", dtype=torch.int32)
    num = torch.tensor([work.shape[0]], device="cuda", dtype=torch.int32)
    part = torch.empty(floats, device="cuda")
    out = torch.full((r, n), 7.0, dtype=torch.bfloat16, device="cuda")
    L, p = _lib.lib(), _lib.ptr
    _lib.check(L.b200_gemm_fp4_terms(p(ew.weight), p(xq), p(sf), p(outside), p(rest), p(out), r, n, k, 1, p(work), p(num), work.shape[0],
                                     p(part), p(cnt), p(_lib.status_word(x.device)), _lib.stream()), "fp4 product")
    torch.cuda.synchronize()
    _lib.check_status()
    assert not cnt.any()
    return out


def _weights(n, k, spread=3):
    q = torch.randint(0, 256, (n, k // 2), device="cuda", dtype=torch.uint8)
    s = torch.randint(127 - spread, 128 + spread, (n, k // 32), device="cuda", dtype=torch.uint8)
    return q, s, fp4fmt.dequantize(q, s).double()


@pytest.mark.parametrize("k", [128, 384])
def test_terms_are_exact_or_small_beside_the_block(k):
    """hi + 2^-5 mid under the block's scale is the value itself down to 2^-14 of the block's largest, and off by at most 2^-22 of it
    below; where that would be more than a quarter of a block, its large values are in ``rest`` instead."""
    torch.manual_seed(k)
    x = torch.randn(40, k, device="cuda") * torch.exp2(torch.randint(-40, 40, (40, k // 32), device="cuda").float()).repeat_interleave(32, 1)
    x[1] = 0
    x[2, ::7] *= 2.0 ** -12
    x[3, ::32] *= 2.0 ** 30                       # one value far above the others
    x[4, 5] = float("inf")
    x[5, 9] = float("nan")
    x[6] = torch.exp2(-(torch.arange(k, device="cuda").float() % 32))
    x = x.bfloat16()
    xq, sf, outside, rest, _ = _gather(x)
    torch.cuda.synchronize()
    order = torch.tensor([0, 4, 1, 5, 2, 6, 3, 7], device="cuda")            # of eight neighbours the even ones are stored first
    v = xq.view(2, 40, k // 8, 8)[..., order].reshape(2, 40, k).view(torch.float8_e4m3fn).double()
    scale = torch.exp2(sf.permute(1, 0, 2).reshape(40, k // 32).double() - 127).repeat_interleave(32, 1)
    got = (v[0] + v[1] / 32) * scale
    out = outside.bool()
    assert out.tolist() == [i in (3, 4, 5, 6) for i in range(40)]
    got = torch.where(out[:, None], got + torch.nan_to_num(rest.double(), posinf=0.0), got)
    want = x.double()
    fine = want.isfinite()
    top = want.where(fine, torch.zeros_like(want)).abs().view(40, -1, 32).amax(-1).repeat_interleave(32, 1)
    err = (got - want).abs()
    exact = fine & (want.abs() >= top * 2.0 ** -13)
    assert (err[exact] == 0).all() and (err[fine] <= top[fine] * 2.0 ** -22).all()
    assert torch.equal(rest[4, 5], x[4, 5]) and rest[5, 9].isnan()
    # small values beside large ones: the smallest quarter of a block by 2^-8 of the value at the quarter, the others not at all
    small = x[3].double().abs().view(-1, 32)
    assert (err[3].view(-1, 32).amax(-1) <= small.kthvalue(9, -1).values * 2.0 ** -8).all()


# rows around tiles of 64 and boxes of 16; features around pairs of 128; one to many blocks of inputs
@pytest.mark.parametrize("r,n,k", [(1, 8, 128), (1, 128, 256), (3, 136, 128), (15, 255, 640), (16, 264, 384), (17, 512, 128), (33, 384, 256),
                                   (63, 128, 4096), (64, 520, 512), (65, 256, 1152), (130, 1000, 384), (2, 8192, 2048), (200, 2560, 256)])
def test_product_against_64_bits(r, n, k):
    torch.manual_seed(r * 7 + n + k)
    x = torch.randn(r, k, device="cuda").bfloat16()
    q, s, w = _weights(n, k)
    got, ref = _product(x, q, s).double(), x.double() @ w.t()
    # the terms are exact, so what is left are fp32 sums (of K products) and one rounding to bf16, half a place of 2^-8
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ w.abs().t()) * k * 2.0 ** -24
    assert ((got - ref).abs() <= bound).all()


def test_values_outside_the_terms_reach_the_product():
    torch.manual_seed(1)
    r, n, k = 70, 384, 640
    x = torch.randn(r, k, device="cuda") * 1e-3
    x[3, 70], x[3, 500], x[65, 129] = 3e8, -1e9, 7e7
    x = x.bfloat16()
    q, s, w = _weights(n, k)
    codes = torch.stack([q & 15, q >> 4], -1).view(n, k)
    for i, j in ((3, 70), (3, 500), (65, 129)):            # their weights are zero in some features
        codes[::3, j] = 0
    q = (codes[:, 0::2] | codes[:, 1::2] << 4).contiguous()
    w = fp4fmt.dequantize(q, s).double()
    got, ref = _product(x, q, s).double(), x.double() @ w.t()
    bound = ref.abs() * 2.0 ** -8 + (x.double().abs() @ w.abs().t()) * k * 2.0 ** -24
    assert ((got - ref).abs() <= bound).all()
    x[7, 11] = float("inf")
    got, ref = _product(x, q, s).double(), x.double() @ w.t()
    assert torch.equal(got[7].isnan(), ref[7].isnan()) and torch.equal(got[7].isinf(), ref[7].isinf()) and got[8].isfinite().all()


# More tiles than SMs: whole waves of one tile a CTA, in which the rings wrap many times and phases pass from tile to tile, then a tail of
# many tiles, of few (which have a bounded number of contributors each), of none.
WAVES = [(300, 10240, 2048), (256, 9472, 640), (640, 9472, 1152), (64, 38400, 2304), (130, 25344, 384), (65, 18944, 4096)]


@pytest.mark.parametrize("outliers", [False, True])
@pytest.mark.parametrize("r,n,k", WAVES)
def test_whole_waves_and_their_tail(r, n, k, outliers):
    torch.manual_seed(r + n + k)
    x = torch.randn(r, k, device="cuda")
    if outliers:                                           # in rows of every token tile, whose feature tiles are in waves and in the tail
        x[::9, ::37] *= 1e-4
        x[::9, 5::64] = 3e8
    x = x.bfloat16()
    q, s, w = _weights(n, k)
    got, again = _product(x, q, s), _product(x, q, s)
    ref, size = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    assert torch.equal(got, again)
    assert ((got.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * k * 2.0 ** -24).all()


def test_every_code_and_scale_comes_out():
    """A one-hot input of 1: the weight itself, under scales over the range that bf16 holds; 255 is taken as 254."""
    n, k = 256, 128
    codes = torch.arange(n * k, device="cuda").view(n, k) % 16
    q = (codes[:, 0::2] | codes[:, 1::2] << 4).to(torch.uint8)
    s = (torch.arange(n * 4, device="cuda").view(n, 4) % 252 + 2).to(torch.uint8)
    w = fp4fmt.level_table("cuda")[codes].double() * torch.exp2(s.double() - 127).repeat_interleave(32, 1)
    got = _product(torch.eye(k, device="cuda").bfloat16(), q, s).double().t()
    fits = w.abs() < 2.0 ** 127
    assert torch.equal(got[fits], w[fits])
    s[0, 0] = 255
    codes[0, :32] = 2
    q = (codes[:, 0::2] | codes[:, 1::2] << 4).to(torch.uint8)
    assert _product(torch.eye(k, device="cuda").bfloat16() * 0.5, q, s)[0, 0].item() == 2.0 ** 126


@pytest.mark.parametrize("t,lo", [(1, 0), (9, 0), (40, 2), (300, 2), (1100, 0)])
def test_experts_match_the_general_path(t, lo, monkeypatch):
    """The same experts through the kernel that unpacks weights to bf16: both are exact but for fp32 sums and the same roundings."""
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    torch.manual_seed(t)
    e, el, k, h, inter = 12, 8, 3, 384, 256
    m13, m2 = ([fp4fmt.quantize(torch.randn(n, kk, device="cuda") * 0.1) for _ in range(el)] for n, kk in ((2 * inter, h), (h, inter)))
    w13, w2 = (moe.ExpertWeights.from_fp4(*map(list, zip(*m))) for m in (m13, m2))
    x = torch.randn(t, h, device="cuda").bfloat16()
    idx = torch.rand(t, e, device="cuda").topk(k).indices.int().contiguous()
    wts = torch.rand(t, k, device="cuda")
    call = lambda: moe.experts_forward(x, idx, wts, w13, w2, lo, swiglu_limit=2.0)
    a, again = call(), call()

    # the general path takes its own layout
    def unscaled(q):
        n, kk = q[0].shape[0], q[0].shape[1] * 2
        codes = q[0].view(n // 128, 128, kk // 64, 32).permute(0, 2, 1, 3).reshape(n // 128, kk // 64, -1)
        sc = q[1].view(n // 128, 128, kk // 64, 2).permute(0, 2, 1, 3).reshape(n // 128, kk // 64, -1)
        return torch.cat([codes, sc], -1)
    monkeypatch.setattr(moe.ExpertWeights, "block_scaled", False)
    w13.weight, w2.weight = (torch.stack([unscaled(q) for q in m]) for m in (m13, m2))
    b = call()
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(a, again)
    # sums in another order move a rounding to bf16 now and then, twice on the way and once at the end
    assert ((a.double() - b.double()).norm() / b.double().norm()).item() < 2.0 ** -8


def _decode_layout(q, scales):
    """One matrix of whole 128-blocks as the decode-warp kernel has matrices of other widths."""
    n, kk = q.shape[0], q.shape[1] * 2
    codes = q.view(n // 128, 128, kk // 64, 32).permute(0, 2, 1, 3).reshape(n // 128, kk // 64, -1)
    sc = scales.view(n // 128, 128, kk // 64, 2).permute(0, 2, 1, 3).reshape(n // 128, kk // 64, -1)
    return torch.cat([codes, sc], -1)


# rows per expert around the token tiles of the decode-warp kernel (16 to 256)
@pytest.mark.parametrize("t,h,inter", [(1, 128, 128), (20, 384, 256), (70, 640, 128), (150, 256, 384), (300, 384, 256), (900, 2048, 384)])
def test_both_layouts_through_the_decode_warps(t, h, inter, monkeypatch):
    """The same codes and scales, in the same order of sums: equal results."""
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    torch.manual_seed(t)
    el, k = 8, 3
    m13, m2 = ([_weights(n, kk)[:2] for _ in range(el)] for n, kk in ((2 * inter, h), (h, inter)))
    w13, w2 = (moe.ExpertWeights.from_fp4(*map(list, zip(*m))) for m in (m13, m2))
    x = torch.randn(t, h, device="cuda").bfloat16()
    idx = torch.rand(t, el, device="cuda").topk(k).indices.int().contiguous()
    wts = torch.rand(t, k, device="cuda")
    monkeypatch.setattr(moe, "fp4_terms_pay", lambda *a: False)
    a = moe.experts_forward(x, idx, wts, w13, w2, 0, swiglu_limit=2.0)
    monkeypatch.setattr(moe.ExpertWeights, "block_scaled", False)
    w13.weight, w2.weight = (torch.stack([_decode_layout(*q) for q in m]) for m in (m13, m2))
    b = moe.experts_forward(x, idx, wts, w13, w2, 0, swiglu_limit=2.0)
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(a, b)


@pytest.mark.parametrize("terms", [True, False])
@pytest.mark.parametrize("t", [1, 30, 400])
@pytest.mark.parametrize("h,inter", [(256, 192), (192, 256)])
def test_one_matrix_of_whole_blocks_beside_another(t, h, inter, terms, monkeypatch):
    """Hidden or expert width of 64-blocks only: one product may take terms, the other unpacks."""
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    monkeypatch.setattr(moe, "fp4_terms_pay", lambda *a: terms)
    torch.manual_seed(t + h)
    el, k = 4, 2
    m13, m2 = ([_weights(n, kk, 1) for _ in range(el)] for n, kk in ((2 * inter, h), (h, inter)))
    w13, w2 = (moe.ExpertWeights.from_fp4([q[0] for q in m], [q[1] for q in m]) for m in (m13, m2))
    assert w13.block_scaled != w2.block_scaled
    x = (torch.randn(t, h, device="cuda") * 0.02).bfloat16()
    idx = torch.rand(t, el, device="cuda").topk(k).indices.int().contiguous()
    wts = torch.rand(t, k, device="cuda")
    got = moe.experts_forward(x, idx, wts, w13, w2, 0).double()
    torch.cuda.synchronize()
    _lib.check_status()
    want = torch.zeros(t, h, dtype=torch.float64, device="cuda")
    for e in range(el):
        rows, col = (idx == e).nonzero(as_tuple=True)
        gu = x[rows].double() @ m13[e][2].t()
        act = torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]
        want.index_add_(0, rows, wts[rows, col].double()[:, None] * (act @ m2[e][2].t()))
    # four roundings to bf16 on the way (gate, up, unit, expert) and one at the end
    assert ((got - want).norm() / want.norm()).item() < 2.0 ** -7


# the same shapes and ranges of held experts as above, one with as many tiles as SMs and more, and one whose rows are few for many SMs
@pytest.mark.parametrize("t,lo,el,h,inter", [(1, 0, 8, 384, 256), (9, 0, 8, 384, 256), (40, 2, 8, 384, 256), (300, 2, 8, 384, 256),
                                             (1100, 0, 8, 384, 256), (700, 0, 48, 1024, 512), (6, 0, 8, 2048, 768)])
def test_experts_as_terms_match_the_unpacked(t, lo, el, h, inter, monkeypatch):
    """Both routes of block-scaled experts: exact but for fp32 sums and the same roundings."""
    from deepseek_v4_2080ti_b200.ops import _lib, moe
    torch.manual_seed(t)
    k = 3
    m13, m2 = ([fp4fmt.quantize(torch.randn(n, kk, device="cuda") * 0.1) for _ in range(el)] for n, kk in ((2 * inter, h), (h, inter)))
    w13, w2 = (moe.ExpertWeights.from_fp4(*map(list, zip(*m))) for m in (m13, m2))
    x = torch.randn(t, h, device="cuda").bfloat16()
    idx = torch.rand(t, el + 4, device="cuda").topk(k).indices.int().contiguous()
    wts = torch.rand(t, k, device="cuda")
    out = []
    for terms in (True, True, False):
        monkeypatch.setattr(moe, "fp4_terms_pay", lambda *a: terms)
        out.append(moe.experts_forward(x, idx, wts, w13, w2, lo, swiglu_limit=2.0))
    torch.cuda.synchronize()
    _lib.check_status()
    assert torch.equal(out[0], out[1])
    # sums in another order move a rounding to bf16 now and then, twice on the way and once at the end
    assert ((out[0].double() - out[2].double()).norm() / out[2].double().norm()).item() < 2.0 ** -8
