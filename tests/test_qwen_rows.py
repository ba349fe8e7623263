"""A prompt portion through all layers in one native call (csrc/kernels/qwen_rows.cu) against the same launches issued one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens around the tiles of the FP8 term products (16, 32, 64, 128, 256) and of the attention and delta-rule chunks; two portions, so that
# the second starts from states, tails and a context
@pytest.mark.parametrize("first,second", [(1, 1), (5, 16), (17, 64), (65, 40), (128, 257), (300, 129)])
@pytest.mark.parametrize("gate", [True, False])
def test_native_portions_equal_the_launches_one_by_one(first, second, gate, monkeypatch):
    from deepseek_v4_2080ti_b200.models import qwen_hybrid as qh
    from deepseek_v4_2080ti_b200.ops import _lib
    cfg = qh.QwenHybridConfig.tiny(layers=4)
    cfg.attn_output_gate = gate
    rt = qh.build_synthetic(cfg, max_slots=2, max_context=1024)
    ids = torch.randint(0, cfg.vocab_size, (first + second,), device="cuda", dtype=torch.int32)
    calls = []
    real = rt._layers_native
    monkeypatch.setattr(rt, "_layers_native", lambda *a: calls.append(1) or real(*a))
    out = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(rt, "_issues_natively", lambda *a: False)
        slot = rt.allocate()
        a = rt.prefill(slot, ids[:first]).clone(), rt.last_logits.clone(), rt.launches
        b = rt.prefill(slot, ids[first:]).clone(), rt.last_logits.clone(), rt.launches
        out.append((a, b, rt.states[slot].clone(), rt.tails[slot].clone()))
        rt.free(slot)
    torch.cuda.synchronize()
    _lib.check_status()
    assert len(calls) == 2
    (a, b, s, t), (a2, b2, s2, t2) = out
    assert torch.equal(s, s2) and torch.equal(t, t2)
    for x, y in ((a, a2), (b, b2)):
        assert torch.equal(x[0], y[0]) and torch.equal(x[1], y[1]) and x[2] == y[2]


# both sides of the widest tile of one CTA
@pytest.mark.parametrize("first,second", [(127, 128), (129, 66)])
def test_portions_around_the_widest_single_tile(first, second, monkeypatch):
    test_native_portions_equal_the_launches_one_by_one(first, second, True, monkeypatch)


def test_portions_do_not_wait_for_the_device():
    """Prompts queue behind a long kernel: none of them may need the device to finish before it returns."""
    from deepseek_v4_2080ti_b200.models import qwen_hybrid as qh
    cfg = qh.QwenHybridConfig.tiny(layers=2)
    rt = qh.build_synthetic(cfg, max_slots=2, max_context=256)
    ids = torch.randint(0, cfg.vocab_size, (40,), device="cuda", dtype=torch.int32)
    slot = rt.allocate()
    rt.prefill(slot, ids)
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)                     # some 0.2 s
    done = torch.cuda.Event()
    done.record()
    rt.prefill(slot, ids[:33])
    assert not done.query()
    torch.cuda.synchronize()


# rows around what one launch carries; slots in any order, contexts around page edges
@pytest.mark.parametrize("b", [1, 3, 127, 128, 129, 300])
def test_step_rows_reach_the_device(b):
    import ctypes
    from deepseek_v4_2080ti_b200.ops import _lib
    torch.manual_seed(b)
    rows = torch.randint(0, 5000, (b, 4), dtype=torch.int32)
    rows[:, 2] = torch.randperm(b).int()
    tables = torch.randint(0, 9000, (b, 37), device="cuda", dtype=torch.int32)
    ids = torch.randint(0, 9000, (b,), device="cuda", dtype=torch.int32)
    o = [torch.full((b,), -1, dtype=torch.int32, device="cuda") for _ in range(5)]
    bt = torch.full((b, 37), -1, dtype=torch.int32, device="cuda")
    host = (ctypes.c_int * (4 * b))(*rows.flatten().tolist())
    _lib.check(_lib.lib().b200_step_meta(host, b, _lib.ptr(ids), _lib.ptr(tables), 37, *map(_lib.ptr, o), _lib.ptr(bt), _lib.stream()), "meta")
    want = [ids.cpu(), rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3]]
    assert all(torch.equal(a.cpu(), w) for a, w in zip(o, want)) and torch.equal(bt.cpu(), tables.cpu()[rows[:, 2].long()])
