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
