"""FP8 block-128 products from pairs of FP8 terms (csrc/kernels/gemm_fp8_terms.cu, gemm_fp8_pair.cu)."""
import pytest
import torch

from deepseek_v4_2080ti_b200.formats import fp8 as fp8fmt

# (tokens, features, inputs): both sides of every tile width (16, 32, 64 tokens; 256 on pairs), ragged feature counts, an odd
# number of weight tiles, one K block, runs that cut tiles several times, more runs than one per tile, narrow matrices whose tiles
# are shared by a few contributors each (one CTA and pairs, one and several token tiles), and ones with a CTA per tile
SHAPES = [(1, 128, 128), (1, 5120, 4096), (16, 384, 512), (17, 1000, 1280), (32, 1536, 4096), (33, 201, 640), (64, 12288, 512),
          (65, 128, 128), (100, 384, 1024), (128, 200, 384), (129, 640, 2560), (256, 1024, 4096), (257, 5120, 1024),
          (300, 33, 256), (700, 3072, 1152), (2, 576, 7168), (40, 576, 7168), (65, 576, 7168), (300, 576, 7168), (8, 2048, 5120),
          (129, 2048, 5120), (500, 2048, 5120), (64, 5120, 4096), (200, 5120, 4096), (1, 128, 6144), (10, 18944, 256), (70, 18944, 384)]


def _terms(xt, t, k):
    """What the stored layout says of every activation: (hi + mid) times its block's scale, plus what lies outside."""
    tok = xt.tok
    cap = tok // 2 if tok == 256 else tok
    n, kb = xt.sx.shape[:2]
    b = xt.xq.reshape(n, kb, tok // cap, 2, cap, 8, 16)
    rows = torch.arange(cap, device=b.device)[:, None]
    src = torch.arange(8, device=b.device)[None] ^ (rows & 7)
    b = torch.gather(b, 5, src[None, None, None, None, :, :, None].expand_as(b))
    b = b.reshape(n, kb, tok // cap, 2, cap, 32, 4)[..., [0, 2, 1, 3]]
    hi, mid = (b[:, :, :, i].contiguous().view(f).float() for i, f in ((0, torch.float8_e5m2), (1, torch.float8_e4m3fn)))
    v = (hi + mid).reshape(n, kb, tok, 128) * xt.sx.abs()[..., None]
    v = v.permute(0, 2, 1, 3).reshape(n * tok, k)[:t]
    outside = (xt.sx < 0).permute(0, 2, 1).reshape(n * tok, kb)[:t].repeat_interleave(128, 1)
    return torch.where(outside, v + xt.rest.float(), v)


def _bound(x):
    """How far a block's terms may be off: 2^-9 of a value in its smallest quarter (2^-10 of the units in which that value is at
    least 2^-2), and 2^-21 of its largest where that is less."""
    b = x.float().view(x.shape[0], -1, 128).abs()
    quarter = torch.where(b > 0, b, float("inf")).sort(-1).values
    at = ((b > 0).sum(-1, keepdim=True) // 4).clamp_max(127)
    q = torch.gather(quarter, -1, at) * 2.0 ** -8
    return torch.minimum(q, b.amax(-1, keepdim=True) * 2.0 ** -21).expand_as(b).reshape(x.shape)


def _outliers(t, k, exponent, device="cuda"):
    """Normal rows with two values of size 2^exponent in every block of 128."""
    x = torch.randn(t, k, device=device)
    x.view(t, -1, 128)[:, :, 5] = 2.0 ** exponent
    x.view(t, -1, 128)[:, :, 77] = -1.5 * 2.0 ** exponent
    return x.bfloat16()


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1, 20, 64, 65, 200, 300])
def test_terms_are_exact(t):
    from deepseek_v4_2080ti_b200.ops import gemm
    torch.manual_seed(t)
    x = (torch.randn(t, 384, device="cuda") * torch.exp(2 * torch.randn(t, 384, device="cuda"))).bfloat16()
    x[0, :128] = 0
    got, xf = _terms(gemm.split_terms(x), t, 384), x.float()
    top = xf.view(t, 3, 128).abs().amax(-1, keepdim=True).expand(t, 3, 128).reshape(t, 384)
    small = xf.abs() < top * 2.0 ** -13
    assert torch.equal(got[~small], xf[~small])
    assert ((got - xf).abs() <= _bound(x)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1, 40, 90])
@pytest.mark.parametrize("make", [
    lambda t: _outliers(t, 384, 11), lambda t: _outliers(t, 384, 14), lambda t: _outliers(t, 384, 40),
    lambda t: (torch.randn(t, 384, device="cuda") * torch.exp2(torch.randint(-120, 120, (t, 384), device="cuda").float())).bfloat16(),
    lambda t: torch.where(torch.rand(t, 384, device="cuda") < 0.95, torch.zeros((), device="cuda"),      # sparse rows
                          torch.exp2(torch.randint(-60, 60, (t, 384), device="cuda").float())).bfloat16()])
def test_wide_blocks_keep_their_small_values(t, make):
    from deepseek_v4_2080ti_b200.ops import gemm
    torch.manual_seed(t)
    x = make(t)
    assert ((_terms(gemm.split_terms(x), t, 384) - x.float()).abs() <= _bound(x)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1, 6, 32, 33, 64, 65, 100, 300])
@pytest.mark.parametrize("exponent", [8, 10, 11, 12, 14, 18, 30])
def test_large_values_whose_weights_are_zero_hide_nothing(t, exponent):
    """The large values of every block meet weights of zero: what is left is the product of the others."""
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    torch.manual_seed(t + exponent)
    n, k = 320, 640
    wf = torch.randn(n, k, device="cuda") * 0.05
    wf.view(n, -1, 128)[:, :, 5] = wf.view(n, -1, 128)[:, :, 77] = 0
    q, s = fp8fmt.quantize_block128(wf)
    x = _outliers(t, k, exponent)
    w = gemm.PackedLinear.from_fp8(q, s)
    y, z = gemm.linear_terms(gemm.split_terms(x), w), gemm.linear(x, w)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = x.double() @ fp8fmt.dequantize_block128(q, s).double().t()
    # 2^-9 of the result: its rounding to bf16 (2^-9 at most, 2^-9 / sqrt 3 in the mean) and the terms (a quarter of the values
    # off by up to 2^-8 of the value at the quarter, a third of the mean size); 2^-9 more where the decode warps round the weights
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -9
    assert ((z.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8


@pytest.mark.gpu
@pytest.mark.parametrize("t,n,k", [(3, 200, 256), (30, 1000, 1280), (64, 384, 2560), (70, 33, 384), (257, 640, 2560), (300, 5120, 1024)])
def test_values_outside_the_terms_are_multiplied(t, n, k):
    """Outliers with weights like any other, in some blocks of some rows, runs cut and whole, with a residual."""
    from deepseek_v4_2080ti_b200.ops import gemm
    torch.manual_seed(t + n + k)
    q, s = fp8fmt.quantize_block128(torch.randn(n, k, device="cuda") * 0.05)
    w, wd = gemm.PackedLinear.from_fp8(q, s), fp8fmt.dequantize_block128(q, s).double()
    x = torch.randn(t, k, device="cuda").bfloat16()
    blocks = torch.rand(t, k // 128, 1, device="cuda") < 0.2
    x = torch.where(blocks, _outliers(t, k, 16).view(t, -1, 128), x.view(t, -1, 128)).view(t, k)
    r = torch.randn(t, n, device="cuda").bfloat16()
    xt = gemm.split_terms(x)
    assert (xt.sx[..., :].lt(0).any())
    y, again, z = gemm.linear_terms(xt, w), gemm.linear_terms(xt, w), gemm.linear_terms(xt, w, residual=r)
    ref = x.double() @ wd.t()
    rel = lambda a, b: ((a.double() - b).norm(dim=1) / b.norm(dim=1)).max().item()
    assert rel(y, ref) < 2.0 ** -8 and rel(z, ref + r.double()) < 2.0 ** -8          # every row: at most the rounding to bf16
    assert torch.equal(y, again)


@pytest.mark.gpu
@pytest.mark.parametrize("t,n,k", SHAPES)
def test_product_matches_64_bit(t, n, k):
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    torch.manual_seed(t + n + k)
    q, s = fp8fmt.quantize_block128(torch.randn(n, k, device="cuda") * 0.05)
    w = gemm.PackedLinear.from_fp8(q, s)
    x = torch.randn(t, k, device="cuda").bfloat16()
    x[:, ::7] *= 8.0
    r = torch.randn(t, n, device="cuda").bfloat16()
    wide = torch.empty(t, n + 1, dtype=torch.bfloat16, device="cuda")
    out = wide.view(-1)[1:t * n + 1].view(t, n)                      # rows that no 16-byte access fits
    xt = gemm.split_terms(x)
    y, z, u = gemm.linear_terms(xt, w), gemm.linear_terms(xt, w, residual=r), gemm.linear_terms(xt, w, out=out)
    again = gemm.linear_terms(xt, w)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = x.double() @ fp8fmt.dequantize_block128(q, s).double().t()
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    # rounding the result to bf16 is at most 2^-9 of each value; fp32 sums and subnormal terms stay far below
    assert rel(y, ref) < 2.0 ** -9 and rel(z, ref + r.double()) < 2.0 ** -9
    assert torch.equal(y, again) and torch.equal(y, u)


# pairs with more tiles than there are pairs: whole waves of neighbouring tiles, then a tail of none (148 tiles), of one to two tiles a pair,
# an odd last weight tile
WAVES = [(257, 18944, 256), (513, 19072, 384), (300, 38144, 256), (129, 56832, 128), (700, 12800, 896)]


@pytest.mark.gpu
@pytest.mark.parametrize("outliers", [False, True])
@pytest.mark.parametrize("t,n,k", WAVES)
def test_whole_waves_of_pair_tiles(t, n, k, outliers):
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    torch.manual_seed(t + n + k)
    q, s = fp8fmt.quantize_block128(torch.randn(n, k, device="cuda") * 0.05)
    w, wd = gemm.PackedLinear.from_fp8(q, s), fp8fmt.dequantize_block128(q, s).double()
    x = torch.randn(t, k, device="cuda").bfloat16()
    if outliers:                                           # in rows of every token tile, so in tiles of the waves and of the tail
        blocks = torch.rand(t, k // 128, 1, device="cuda") < 0.05
        x = torch.where(blocks, _outliers(t, k, 16).view(t, -1, 128), x.view(t, -1, 128)).view(t, k)
    r = torch.randn(t, n, device="cuda").bfloat16()
    xt = gemm.split_terms(x)
    assert bool(xt.sx.permute(0, 2, 1).reshape(-1, k // 128)[:t].lt(0).any()) == outliers
    y, again, z = gemm.linear_terms(xt, w), gemm.linear_terms(xt, w), gemm.linear_terms(xt, w, residual=r)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = x.double() @ wd.t()
    rel = lambda a, b: ((a.double() - b).norm(dim=1) / b.norm(dim=1)).max().item()
    assert rel(y, ref) < 2.0 ** -8 and rel(z, ref + r.double()) < 2.0 ** -8          # every row: at most the rounding to bf16
    assert torch.equal(y, again)


@pytest.mark.gpu
@pytest.mark.parametrize("t", [7, 40, 300])
def test_products_on_two_streams_share_no_scratch(t):
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    torch.manual_seed(t)
    q, s = fp8fmt.quantize_block128(torch.randn(2560, 2560, device="cuda") * 0.05)
    w = gemm.PackedLinear.from_fp8(q, s)
    xs = [torch.randn(t, 2560, device="cuda").bfloat16() for _ in range(2)]
    before = dict(gemm._workspaces)
    want = [gemm.linear(x, w) for x in xs]
    assert gemm._workspaces == before              # nothing kept per device, which the streams would meet in
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for x, st, ys in zip(xs, streams, got):
            with torch.cuda.stream(st):
                ys.append(gemm.linear(x, w))
    torch.cuda.synchronize()
    _lib.check_status()
    assert all(torch.equal(y, z) for ys, z in zip(got, want) for y in ys)


@pytest.mark.gpu
@pytest.mark.parametrize("t,n,k", [(1, 5120, 1280), (20, 1000, 640), (64, 201, 384), (65, 640, 2560), (300, 5120, 1024), (300, 33, 256)])
def test_products_stay_inside_their_buffers(t, n, k):
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    from deepseek_v4_2080ti_b200.utils import canary
    torch.manual_seed(t + n)
    q, s = fp8fmt.quantize_block128(torch.randn(n, k, device="cuda") * 0.05)
    w = gemm.PackedLinear.from_fp8(q, s)
    x = _outliers(t, k, 16)
    plain = gemm.split_terms(x)
    want = gemm.linear_terms(plain, w)
    with canary.enabled():
        buf = lambda n, dtype, name: canary.empty(n, dtype=dtype, device="cuda", name=name)
        xq, sx, rest = (buf(v.numel(), v.dtype, n) for v, n in ((plain.xq, "terms"), (plain.sx, "scales"), (plain.rest, "rest")))
        partial, out = buf(plain.partial_floats, torch.float32, "partial sums"), buf(t * n, torch.bfloat16, "product")
        counters = buf(plain.buf.numel() - plain.xq.numel() - 4 * plain.sx.numel() - 2 * plain.rest.numel() >> 2, torch.int32, "counters")
        L, p, st = _lib.lib(), _lib.ptr, _lib.stream()
        _lib.check(L.b200_split_terms(p(x), t, k, plain.tok, p(xq), p(sx), p(rest), p(counters), st), "split")
        _lib.check(L.b200_gemm_fp8_terms(p(w.weight), p(w.scales), p(xq), p(sx), p(rest), p(out), None, t, n, k, p(partial), p(counters),
                                         p(_lib.status_word(x.device)), st), "product")
        torch.cuda.synchronize()
        _lib.check_status()
        assert not canary.verify_all() and not counters.any()
    assert torch.equal(out.view(t, n), want)


@pytest.mark.parametrize("off", [2, 4, 8])
def test_rows_that_no_load_fits_are_refused(off):
    """The pointers are looked at before anything is launched: these are addresses of nothing."""
    import ctypes
    from deepseek_v4_2080ti_b200.ops import _lib
    lib, v, f = _lib.lib(), ctypes.c_void_p, ctypes.c_float(1e-6)
    good, bad = v(1 << 20), v((1 << 20) + off)
    terms = (v(2 << 20), v(3 << 20), v(4 << 20), v(5 << 20), None)
    assert lib.b200_split_terms(bad, 33, 256, 64, *terms) == -6
    if off < 8:
        assert lib.b200_split_terms(bad, 32, 256, 32, *terms) == -6
    assert lib.b200_silu_mul_terms(bad, 4, 256, 16, *terms) == -6
    for x, delta, gamma, out in ((bad, None, good, good), (good, bad, good, good), (good, None, bad, good), (good, None, good, bad)):
        assert lib.b200_rmsnorm_terms(x, delta, gamma, out, 4, 256, f, 1, 16, *terms) == -6
    for at in (0, 2, 3, 4):                        # weights, terms, their scales, what lies outside
        args = [good, good, good, good, good]
        args[at] = bad
        assert lib.b200_gemm_fp8_terms(*args, good, None, 4, 256, 256, good, good, good, None) == -6


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1, 5, 32])
def test_rows_aligned_to_eight_bytes(t):
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    torch.manual_seed(t)
    q, s = fp8fmt.quantize_block128(torch.randn(384, 1280, device="cuda") * 0.05)
    w = gemm.PackedLinear.from_fp8(q, s)
    wide = torch.randn(40 * 1280 + 4, device="cuda").bfloat16()
    x = wide[4:4 + t * 1280].view(t, 1280)
    assert torch.equal(gemm.linear(x, w), gemm.linear(x.clone(), w))
    with pytest.raises(_lib.KernelError):
        gemm.linear(wide[4:].view(40, 1280), w)    # past 32 rows they are refused, as they were


@pytest.mark.gpu
@pytest.mark.parametrize("t", [5, 40, 80])
def test_infinities_and_nans_stay_in_their_row(t):
    from deepseek_v4_2080ti_b200.ops import gemm
    torch.manual_seed(t)
    q, s = fp8fmt.quantize_block128(torch.randn(256, 256, device="cuda"))
    w, wd = gemm.PackedLinear.from_fp8(q, s), fp8fmt.dequantize_block128(q, s)
    x = torch.randn(t, 256, device="cuda").bfloat16()
    clean = gemm.linear_terms(gemm.split_terms(x), w)
    inf = float("inf")
    x[0, 5], x[1, 200] = inf, float("nan")
    x[2, 5], x[2, 77] = inf, -inf                 # two of a block
    x[3, 5], x[3, 200] = inf, inf                 # two blocks
    x[4, 200], x[4, 201], x[4, 202] = -inf, -inf, 2.0 ** 100
    y = gemm.linear_terms(gemm.split_terms(x), w).double()
    ref = x.double() @ wd.double().t()
    assert torch.equal(y[5:], clean[5:].double())
    for kind in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(kind(y[:5]), kind(ref[:5]))
    assert ref[2].isnan().any() and ref[2].isinf().any() and not ref[:5].isfinite().any()


@pytest.mark.gpu
@pytest.mark.parametrize("t,cols", [(1, 128), (3, 5120), (16, 8192), (33, 8320), (65, 20480), (300, 384)])
def test_norm_leaves_its_result_as_terms(t, cols):
    from deepseek_v4_2080ti_b200.ops import basic
    torch.manual_seed(t + cols)
    h, d = (torch.randn(t, cols, device="cuda").bfloat16() for _ in range(2))
    g = (torch.randn(cols, device="cuda") * 0.1).bfloat16()
    stream = h.clone()
    out, xt = basic.rmsnorm_terms(stream, d, g, 1e-6, True)
    assert torch.equal(stream, (h.float() + d.float()).bfloat16())
    ref = basic.rmsnorm_ref(stream, g, 1e-6, True)
    assert ((out.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-6).all()        # bf16 rounding, fp32 sums in any order
    got = _terms(xt, t, cols)
    assert ((got - out.float()).abs() <= _bound(out)).all()
    none, alone = basic.rmsnorm_terms(stream, None, g, 1e-6, True, want_bf16=False)
    assert none is None and torch.equal(_terms(alone, t, cols), got)


@pytest.mark.gpu
@pytest.mark.parametrize("t,inter", [(1, 128), (7, 17408), (64, 2176), (70, 384)])
def test_activation_leaves_its_result_as_terms(t, inter):
    from deepseek_v4_2080ti_b200.ops import basic
    torch.manual_seed(t + inter)
    gu = (torch.randn(t, 2 * inter, device="cuda") * 2).bfloat16()
    ref, got = basic.silu_mul_ref(gu), _terms(basic.silu_mul_terms(gu), t, inter)
    assert ((got - ref).abs() <= ref.abs() * 2.0 ** -8 + _bound(ref)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("b,hv,hk", [(1, 4, 2), (20, 4, 4), (33, 8, 2)])
def test_decode_mixer_leaves_its_result_as_terms(b, hv, hk):
    from deepseek_v4_2080ti_b200.ops import gdn, gemm
    torch.manual_seed(b)
    kd, vd, hidden = hk * 128, hv * 128, 512
    bf = lambda *s, std=1.0: (torch.randn(*s, device="cuda") * std).bfloat16()
    proj, x, w_ab, conv, gamma = bf(b, 2 * kd + 2 * vd), bf(b, hidden), bf(2 * hv, hidden, std=0.03), bf(2 * kd + vd, 4, std=0.3), bf(128)
    a_log, dt = torch.rand(hv, device="cuda"), torch.rand(hv, device="cuda")
    tails, states = bf(b, 3, 2 * kd + vd), torch.randn(b, hv, 128, 128, device="cuda") * 0.1
    slots = torch.randperm(b, device="cuda").int()
    args = lambda: (proj, x, w_ab, a_log, dt, conv, tails.clone(), states.clone(), slots, gamma, hv, hk)
    y = gdn.decode_fused(*args()).float()
    got = _terms(gdn.decode_fused(*args(), terms=gemm.Terms(b, vd, torch.device("cuda"))), b, vd)
    assert ((got - y).abs() <= _bound(y)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("t,n,k", [(65, 64, 5120), (129, 200, 1024), (333, 64, 5120), (700, 256, 512)])
def test_narrow_bf16_matrices(t, n, k):
    """Few feature tiles: the tokens are tiled finer."""
    from deepseek_v4_2080ti_b200.ops import gemm
    torch.manual_seed(t + n)
    x, w = torch.randn(t, k, device="cuda").bfloat16(), (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    ref = x.double() @ w.double().t()
    y, f = gemm.linear(x, gemm.PackedLinear.from_bf16(w)), gemm.linear(x, gemm.PackedLinear.from_bf16(w), out_f32=True)
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -9
    assert ((f.double() - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("t,k,h", [(1, 6, 4096), (3, 1, 8), (5, 9, 1032), (2, 4, 100)])
def test_expert_rows_are_combined(t, k, h):
    """Eight columns per thread, and rows that do not divide into eights; routes held elsewhere are skipped."""
    from deepseek_v4_2080ti_b200.ops import _lib
    torch.manual_seed(h)
    y, base = torch.randn(t * k, h, device="cuda").bfloat16(), torch.randn(t, h, device="cuda").bfloat16()
    rows = torch.randperm(t * k, device="cuda").int().view(t, k)
    rows[0, 0] = -1
    w, out = torch.rand(t, k, device="cuda"), torch.empty(t, h, dtype=torch.bfloat16, device="cuda")
    _lib.check(_lib.lib().b200_moe_combine(_lib.ptr(y), _lib.ptr(rows), _lib.ptr(w), _lib.ptr(base), _lib.ptr(out), t, k, h, _lib.stream()), "moe_combine")
    ref = base.double() + torch.where(rows[..., None] >= 0, w.double()[..., None] * y.double()[rows.clamp_min(0).long()], 0.0).sum(1)
    assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all()


# (tokens, features, inputs, us with the split, us of the kernel that takes its place): the two sides of the rule
ROUTES = [(1, 576, 7168, 9.4, 11.7), (1, 5120, 4096, 9.7, 14.1), (32, 576, 7168, 11.1, 21.7), (64, 34816, 5120, 45, 179), (65, 34816, 5120, 62, 59),
          (100, 14336, 5120, 38, 34), (128, 34816, 5120, 73, 61), (128, 12288, 5120, 37.5, 56), (128, 5120, 17408, 50, 67), (65, 576, 7168, 20, 32),
          (128, 1536, 7168, 26, 47), (129, 5120, 17408, 58, 132), (257, 7168, 2048, 33, 27), (256, 5120, 4096, 31, 40),
          (700, 5120, 4096, 49, 41), (700, 12288, 5120, 95, 89), (333, 12288, 5120, 76, 87), (1500, 2048, 5120, 58, 46),
          (1901, 1536, 7168, 77, 58), (1901, 7168, 2048, 76, 70), (1000, 5120, 17408, 173, 301), (1901, 34816, 5120, 642, 770),
          (1901, 4096, 4096, 101, 76), (1000, 2048, 5120, 43, 47), (1500, 7168, 2048, 69, 57)]


@pytest.mark.parametrize("t,n,k,terms_us,other_us", ROUTES)
def test_terms_are_chosen_where_they_are_faster(t, n, k, terms_us, other_us):
    from deepseek_v4_2080ti_b200.ops import gemm
    assert gemm.terms_pay(t, n, k) == (terms_us <= other_us)
    assert gemm.terms_pay(t, n, 255 * 128)         # more inputs than the decode warps take


def test_prefill_sized_batches_are_expanded_ragged_or_not():
    from deepseek_v4_2080ti_b200.ops import gemm
    w = gemm.PackedLinear(gemm.WF_FP8_B128, torch.empty(0), None, 5120, 4096)
    assert [gemm.expands(t, w) for t in (64, 2047, 2048, 2049, 3001, 8191, 8192)] == [False] * 2 + [True] * 5


@pytest.mark.gpu
@pytest.mark.parametrize("t,n,k", [(1, 576, 7168), (2, 200, 256), (65, 14336, 256), (128, 19072, 384), (257, 7168, 2048), (513, 12288, 256),
                                   (701, 5120, 512), (1501, 2048, 512), (2047, 1536, 640), (2049, 640, 384), (3001, 200, 256), (2048, 300, 384),
                                   (128, 384, 32768), (700, 128, 32640), (2100, 72, 32640)])
def test_every_route_of_linear_gives_the_same_product(t, n, k):
    """Both sides of each line that ``linear`` draws, and the prefill-sized batches past the last, against 64 bits."""
    from deepseek_v4_2080ti_b200.ops import _lib, gemm
    torch.manual_seed(t + n)
    q, s = fp8fmt.quantize_block128(torch.randn(n, k, device="cuda") * 0.05)
    w = gemm.PackedLinear.from_fp8(q, s)
    x, r = torch.randn(t, k, device="cuda").bfloat16(), torch.randn(t, n, device="cuda").bfloat16()
    y, z, other = gemm.linear(x, w), gemm.linear(x, w, residual=r), gemm.linear_terms(gemm.split_terms(x), w)
    torch.cuda.synchronize()
    _lib.check_status()
    ref = x.double() @ fp8fmt.dequantize_block128(q, s).double().t()
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    # the result rounded to bf16, and where the decode warps or the expansion take it every scaled weight too: 2^-9 at most each
    assert rel(y, ref) < 2.0 ** -8 and rel(z, ref + r.double()) < 2.0 ** -8 and rel(other, ref) < 2.0 ** -9
