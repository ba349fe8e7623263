"""Decode attention where its unrolled walk over the keys begins, ends and has remainders."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("group", [1, 4, 5, 6, 8])
@pytest.mark.parametrize("window,sinks", [(0, 0), (21, 3)])
def test_key_counts_around_a_chunk(group, window, sinks):
    from deepseek_v4_2080ti_b200.ops import _lib, attention
    g = torch.Generator(device="cuda").manual_seed(group)
    hkv, bs = 2, 16
    lens = [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40, 63, 64, 65, 97, 130]
    mb = (max(lens) + bs - 1) // bs
    b = len(lens)
    shape = (b * mb, hkv, bs, 128)
    kc, vc = (torch.randn(shape, generator=g, device="cuda").bfloat16() for _ in range(2))
    bt = torch.randperm(b * mb, generator=g, device="cuda").to(torch.int32).view(b, mb).contiguous()
    q = torch.randn(b, hkv * group, 128, generator=g, device="cuda").bfloat16()
    refs = []
    for i, n in enumerate(lens):
        k, v = (c[bt[i].long()].permute(0, 2, 1, 3).reshape(-1, hkv, 128) for c in (kc, vc))
        seen = list(range(n)) if not window or n <= window + sinks else [*range(sinks), *range(n - window, n)]
        k, v = (x[seen].double().repeat_interleave(group, 1) for x in (k, v))
        w = torch.einsum("hd,nhd->hn", q[i].double(), k).mul(128 ** -0.5).softmax(-1)
        refs.append(torch.einsum("hn,nhd->hd", w, v))
        for c in (kc, vc):                                  # what lies past the last key must not be read into the sums
            page, row = bt[i, n // bs:], n % bs
            if n < mb * bs:
                c[page[0].long(), :, row:] = float("nan")
                c[page[1:].long()] = float("nan")
    want = torch.stack(refs)
    kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    for splits in (1, 2, 3):
        out = attention.decode(q, kc, vc, bt, kv_len, splits=splits, max_kv_len=max(lens), window=window, sinks=sinks)
        torch.cuda.synchronize()
        _lib.check_status()
        # half a unit of the result's bf16 is at most 2^-8 of it; fp32 scores of magnitude 40 are wrong by up to 2^-18 in the
        # exponent, and values of up to 5 weighted by their exponentials by 2^-15: 2^-12 leaves room for sums of 130 of them
        assert ((out.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -12).all()


# the 8-bit caches over the same key counts (1: E4M3, 2: INT8, 3: E4M3 keys and 4-bit values), and pages whose size is no power of two
@pytest.mark.gpu
@pytest.mark.parametrize("group", [1, 3, 5, 6])
@pytest.mark.parametrize("fmt,bs", [(0, 1), (0, 5), (0, 48), (1, 16), (2, 48), (3, 7), (3, 64)])
def test_every_cache_format_and_page_size(group, fmt, bs):
    from deepseek_v4_2080ti_b200.ops import _lib, attention
    g = torch.Generator(device="cuda").manual_seed(group * 8 + fmt)
    hkv = 2
    lens = [1, 2, 6, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 47, 48, 49, 63, 65, 97, 130]
    mb = (max(lens) + bs - 1) // bs + 1
    b = len(lens)
    bt = torch.randperm(b * mb, generator=g, device="cuda").to(torch.int32).view(b, mb).contiguous()
    q = torch.randn(b, hkv * group, 128, generator=g, device="cuda").bfloat16()
    kv_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    shape = (b * mb, hkv, bs, 128)
    byte = lambda *s: torch.randint(0, 256, s, generator=g, device="cuda", dtype=torch.uint8)
    scale = lambda: torch.rand(*shape[:3], generator=g, device="cuda") * 0.01 + 0.002
    if fmt == 0:
        kc, vc = (torch.randn(shape, generator=g, device="cuda").bfloat16() for _ in range(2))
        kd, vd = kc.double(), vc.double()
        call = lambda n: attention.decode(q, kc, vc, bt, kv_len, splits=n, max_kv_len=max(lens))
    else:
        fp8 = lambda: torch.randn(shape, generator=g, device="cuda").mul(60).clamp(-400, 400).to(torch.float8_e4m3fn).view(torch.uint8)
        ks, vs, vm = scale(), scale(), scale() - 0.007
        k8 = byte(*shape) if fmt == 2 else fp8()
        v8 = {1: fp8, 2: lambda: byte(*shape), 3: lambda: byte(*shape[:3], 64)}[fmt]()
        value = lambda x: x.view(torch.int8).double() if fmt == 2 else x.view(torch.float8_e4m3fn).double()
        kd = value(k8) * ks.double()[..., None]
        if fmt == 3:
            vd = torch.stack([v8 & 15, v8 >> 4], -1).flatten(-2).double() * vs.double()[..., None] + vm.double()[..., None]
        else:
            vd = value(v8) * vs.double()[..., None]
        call = lambda n: attention.decode_kv8(fmt, q, k8, v8, ks, vs, bt, kv_len, splits=n, max_kv_len=max(lens), v_min=vm if fmt == 3 else None)
    want = torch.empty(b, hkv * group, 128, dtype=torch.float64, device="cuda")
    for i, n in enumerate(lens):
        k, v = (c[bt[i].long()].permute(0, 2, 1, 3).reshape(-1, hkv, 128)[:n].repeat_interleave(group, 1) for c in (kd, vd))
        w = torch.einsum("hd,nhd->hn", q[i].double(), k).mul(128 ** -0.5).softmax(-1)
        want[i] = torch.einsum("hn,nhd->hd", w, v)
    for splits in (1, 3):
        out = call(splits)
        torch.cuda.synchronize()
        _lib.check_status()
        assert ((out.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -12).all()       # as above


@pytest.mark.gpu
@pytest.mark.parametrize("group", [1, 5])
def test_four_keys_of_a_half_warp_share_one_maximum(group):
    """Up to five heads a group, the first four keys of a half-warp are weighted by 2^(score - the largest of the four): one that lies 140
    below it has no weight at all (2^-140 is flushed), and none by way of a key between the two either."""
    import ctypes

    import numpy as np

    from deepseek_v4_2080ti_b200.ops import _lib
    log2e, near = np.float32(1.4426950408889634), np.float32(0.6931472)
    scale = next(x for x in (near, np.nextafter(near, np.float32(0)), np.nextafter(near, np.float32(1))) if x * log2e == np.float32(1))
    n, per, bs = 64, 32, 16
    k, v = torch.zeros(n // bs, 1, bs, 128), torch.zeros(n // bs, 1, bs, 128)
    k[..., 0] = -1000.0                                    # scores: nothing beside those of the first half-warp's keys
    for key, score in ((0, -140.0), (8, -120.0), (16, -1000.0), (24, 0.0)):
        k[key // bs, 0, key % bs, 0] = score
    for key in (0, 8):
        v[key // bs, 0, key % bs] = 1.0
    q = torch.zeros(1, group, 128)
    q[..., 0] = 1.0
    q, k, v = (x.to("cuda", torch.bfloat16) for x in (q, k, v))
    bt, kv_len = torch.arange(n // bs, dtype=torch.int32, device="cuda"), torch.tensor([n], dtype=torch.int32, device="cuda")
    out, part = torch.empty_like(q), torch.full((group, n // per, 130), 7.0, device="cuda")
    p = _lib.ptr
    _lib.check(_lib.lib().b200_gqa_decode(p(q), p(k), p(v), p(out), None, p(bt), p(kv_len), p(part), 1, n // bs, bs, group, 1, n // per,
                                          ctypes.c_float(float(scale)), _lib.stream()), "gqa_decode")
    torch.cuda.synchronize()
    assert (part[:, 0, :128] == 2.0 ** -120).all() and (part[:, 0, 128] == 0).all() and (part[:, 0, 129] == 1).all()
