"""A prompt portion through all layers in one native call (csrc/kernels/qwen_rows.cu) against the same launches issued one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens around the tiles of the FP8 term products (16, 32, 64, 256) and of the attention and delta-rule chunks; two portions, so that
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
