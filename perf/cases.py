"""The work this framework is timed on: requests served by the hybrid decoder, and routed-expert blocks.

Two kinds of case.

``serve``: requests through ``QwenHybridRuntime`` - a slot per request, ``prefill`` of each prompt, ``decode`` steps of the
whole batch with the tokens given, slots freed.  The model is an eighth of the benchmark configuration in depth and
vocabulary (8 of 64 layers: 6 Gated DeltaNet + 2 gated GQA, hidden 5120, feed-forward 17408, 18992 of 151936 rows of the
head), so that a layer weighs against the head as in the whole model and every step streams 3 GB of FP8 weights.

``experts``: one routed-expert block, ``moe.route`` + ``moe.experts_forward``, of the MoE families with all 256 experts on
one GPU: FP4 experts of the DeepSeek-V4-Flash shape (hidden 4096, width 2048, top 6) and GGUF experts of the
MiniMax-M2.7 shape (hidden 3072, width 1536, top 8; Q4_K gate / up, Q2_K down).
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

DEV = "cuda"
# Weights: N(0, 0.02); the matrices that add to the residual stream scaled down by the depth of the whole model (64 layers,
# two additions each), over embeddings that outweigh one addition, as in trained models.  With all of them at 0.02 the
# stream is made of a few large additions and amplifies the rounding of bf16 activations to 3 % in eight layers.
STD, STD_ADD, STD_EMBED = 0.02, 0.02 / 128 ** 0.5, 0.5
LAYERS, VOCAB, HIDDEN, WIDE = 8, 18992, 5120, 17408
HQ, HKV, D = 40, 8, 128                 # attention heads, key/value heads, width of every head
HK, HV = 16, 32                         # Gated DeltaNet key and value heads
KD, VD = HK * D, HV * D
EPS, ROT, THETA = 1e-6, 32, 1e7
EXPERTS, POOL = 256, 8                  # experts of a block; distinct ones among them
SHAPES = {"fp4": (4096, 2048, 6), "gguf": (3072, 1536, 8)}      # hidden, expert width, experts per token


def _serve(name, batch, prompt, new, ragged=False, kv="bf16"):
    return {"name": name, "kind": "serve", "batch": batch, "prompt": prompt, "new": new, "ragged": ragged, "kv": kv}


def _experts(name, fmt, tokens):
    return {"name": name, "kind": "experts", "fmt": fmt, "tokens": tokens}


def listed():
    return [
        _serve("chat_16+16", 1, 16, 16),                          # the shortest exchange: one request, weights streamed per token
        _serve("chat_512+64", 1, 512, 64),                        # an ordinary single request
        _serve("serve8_100+32", 8, 100, 32, ragged=True),         # a small server: eight requests of unequal length
        _serve("serve32_64+64", 32, 64, 64),                      # the benchmark's decode batch
        _serve("serve64_40+40", 64, 40, 40, ragged=True),         # a busy server, past the fused decode step's 32 rows
        _serve("fp8kv4_1500+48", 4, 1500, 48, kv="fp8"),          # longer contexts in the 8-bit cache
        _serve("prompt_333", 1, 333, 0),                          # prompts alone (first token only): short and ragged,
        _serve("prompt_1901", 1, 1901, 0),                        # middling and ragged,
        _serve("long_8192+32", 1, 8192, 32),                      # and the benchmark's 8192 tokens, continued
        _experts("fp4_experts_1", "fp4", 1),                      # decoding one token
        _experts("gguf_experts_24", "gguf", 24),                  # decoding a batch
        _experts("fp4_experts_2000", "fp4", 2000),                # a prompt portion
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.3:
        fmt = rng.choice(("fp4", "gguf"))
        return {"kind": "experts", "fmt": fmt, "tokens": _log(rng, 1, 2000)}
    batch = rng.choice((1, 1, 1, 2, 3, 5, 8, 13, 20, 32, 45, 64))
    prompt = _log(rng, 8, max(16, 6000 // batch if batch < 32 else 2400 // batch))
    new = rng.choice((0, 16, 24, 33)) if batch == 1 else rng.randint(8, 32)
    return {"kind": "serve", "batch": batch, "prompt": prompt, "new": new, "ragged": batch > 1 and rng.random() < 0.6,
            "kv": rng.choice(("bf16", "bf16", "bf16", "fp8"))}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed, *more):
    g = torch.Generator(device=DEV)
    n = int(seed) * 1_000_003
    for m in more:
        n = n * 8191 + m
    g.manual_seed(n % (1 << 62))
    return g


def _fp8(g, n, k, std=STD):
    """FP8 E4M3 [n, k] with one bf16 scale per 128 x 128 block, of N(0, std) weights."""
    w = torch.randn(n, k, generator=g, device=DEV) * std
    b = w.view(n // 128, 128, k // 128, 128)
    s = (b.abs().amax((1, 3)) / 448.0).bfloat16()
    b.div_(s.float()[:, None, :, None]).clamp_(-448.0, 448.0)
    return w.to(torch.float8_e4m3fn), s


def _bf16(g, *shape, std=STD, mean=0.0):
    return (torch.randn(*shape, generator=g, device=DEV) * std + mean).bfloat16()


def _is_full(i):
    return i % 4 == 3


def _layer(seed, i):
    """Tensors of decoder layer ``i`` by their name in a checkpoint; matrices as (fp8, scale)."""
    g = _gen(seed, 1, i)
    t = {"input_layernorm.weight": _bf16(g, HIDDEN, std=0.05), "post_attention_layernorm.weight": _bf16(g, HIDDEN, std=0.05),
         "mlp.gate_proj": _fp8(g, WIDE, HIDDEN), "mlp.up_proj": _fp8(g, WIDE, HIDDEN), "mlp.down_proj": _fp8(g, HIDDEN, WIDE, STD_ADD)}
    if _is_full(i):
        a = "self_attn."
        t |= {a + "q_proj": _fp8(g, 2 * HQ * D, HIDDEN), a + "k_proj": _fp8(g, HKV * D, HIDDEN), a + "v_proj": _fp8(g, HKV * D, HIDDEN),
              a + "o_proj": _fp8(g, HIDDEN, HQ * D, STD_ADD), a + "q_norm.weight": _bf16(g, D, std=0.05), a + "k_norm.weight": _bf16(g, D, std=0.05)}
    else:
        a = "linear_attn."
        u = torch.rand(2, HV, generator=g, device=DEV)
        t |= {a + "in_proj_qkv": _fp8(g, 2 * KD + VD, HIDDEN), a + "in_proj_z": _fp8(g, VD, HIDDEN), a + "out_proj": _fp8(g, HIDDEN, VD, STD_ADD),
              a + "in_proj_a.weight": _bf16(g, HV, HIDDEN), a + "in_proj_b.weight": _bf16(g, HV, HIDDEN),
              a + "conv1d.weight": _bf16(g, 2 * KD + VD, 1, 4, std=0.3), a + "A_log": torch.log(u[0] * 3.0 + 0.5).bfloat16(),
              a + "dt_bias": (u[1] * 2.0 - 1.0).bfloat16(), a + "norm.weight": _bf16(g, D, std=0.05, mean=1.0)}
    return t


def _ends(seed):
    g = _gen(seed, 2)
    return _bf16(g, VOCAB, HIDDEN, std=STD_EMBED), _bf16(g, VOCAB, HIDDEN), _bf16(g, HIDDEN, std=0.05)


def _checkpoint(seed):
    """(name, tensor) pairs as a reader of the checkpoint gives them."""
    embed, head, norm = _ends(seed)
    yield "model.language_model.embed_tokens.weight", embed
    yield "lm_head.weight", head
    yield "model.language_model.norm.weight", norm
    for i in range(LAYERS):
        for name, t in _layer(seed, i).items():
            name = f"model.language_model.layers.{i}.{name}"
            if isinstance(t, tuple):
                yield name + ".weight", t[0]
                yield name + ".weight_scale_inv", t[1]
            else:
                yield name, t


def _lengths(case):
    p = case["prompt"]
    return [max(1, p * (60 + (i * 37) % 81) // 100) if case["ragged"] else p for i in range(case["batch"])]


def _tokens(case, seed):
    """Prompts, and the tokens that every decode step is given [new, batch]."""
    g = _gen(seed, 3)
    ids = lambda *s: torch.randint(0, VOCAB, s, generator=g, device=DEV, dtype=torch.int32)
    return [ids(n) for n in _lengths(case)], ids(case["new"], case["batch"])


def _pool(fmt, seed):
    """POOL distinct experts, [(gate_up, down)], each matrix as (parts of the stored format, its values in 64 bits)."""
    h, inter, _ = SHAPES[fmt]
    g = _gen(seed, 4)
    make = {"fp4": (_fp4, _fp4), "gguf": (_q4_k, _q2_k)}[fmt]
    return [(make[0](g, 2 * inter, h), make[1](g, h, inter)) for _ in range(POOL)]


def _fp4(g, n, k):
    levels = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device=DEV)
    w = torch.randn(n, k, generator=g, device=DEV) * 2.2
    code = torch.bucketize(w.abs(), (levels[1:] + levels[:-1]) / 2).to(torch.uint8) | (w < 0).to(torch.uint8) << 3
    e = torch.randint(119, 122, (n, k // 32), generator=g, device=DEV, dtype=torch.uint8)

    def values():
        v = torch.where(code > 7, -levels[(code & 7).long()], levels[code.long() & 7]).double()
        return (v.view(n, k // 32, 32) * torch.exp2(e.double() - 127.0)[..., None]).view(n, k)
    return ((code[:, 0::2] | code[:, 1::2] << 4).contiguous(), e), values


def _halves(x):
    return x.contiguous().view(torch.uint8).view(*x.shape, 2)


def _q4_k(g, n, k):
    """Q4_K: blocks of 256 in 8 groups, value d sc q - dmin mn, 6-bit sc and mn packed in 12 bytes."""
    b = n * k // 256
    d = (torch.rand(b, generator=g, device=DEV) * 4e-5 + 9e-5).half()
    dmin = (d.float() * 7.5).half()
    sc = torch.randint(20, 64, (b, 8), generator=g, device=DEV, dtype=torch.uint8)
    q = torch.randint(0, 16, (b, 4, 2, 32), generator=g, device=DEV, dtype=torch.uint8)
    packed = torch.cat([sc[:, :4] | (sc[:, 4:] >> 4) << 6, sc[:, :4] | (sc[:, 4:] >> 4) << 6, (sc[:, 4:] & 15) | (sc[:, 4:] & 15) << 4], 1)
    raw = torch.cat([_halves(d), _halves(dmin), packed, (q[:, :, 0] | q[:, :, 1] << 4).view(b, 128)], 1).view(n, -1)

    def values():
        s = sc.double()[..., None]
        return (d.double()[:, None, None] * s * q.view(b, 8, 32).double() - dmin.double()[:, None, None] * s).view(n, k)
    return raw, values


def _q2_k(g, n, k):
    """Q2_K: blocks of 256 in 16 groups, value d sc q - dmin mn, sc and mn in the nibbles of a byte."""
    b = n * k // 256
    d = (torch.rand(b, generator=g, device=DEV) * 6e-4 + 1.5e-3).half()
    dmin = (d.float() * 1.5).half()
    sc = torch.randint(6, 16, (b, 16), generator=g, device=DEV, dtype=torch.uint8)
    q = torch.randint(0, 4, (b, 2, 4, 32), generator=g, device=DEV, dtype=torch.uint8)      # two halves of four 2-bit planes
    qs = (q[:, :, 0] | q[:, :, 1] << 2 | q[:, :, 2] << 4 | q[:, :, 3] << 6).view(b, 64)
    raw = torch.cat([sc | sc << 4, qs, _halves(d), _halves(dmin)], 1).view(n, -1)

    def values():
        s = sc.double()[..., None]
        return (d.double()[:, None, None] * s * q.view(b, 16, 16).double() - dmin.double()[:, None, None] * s).view(n, k)
    return raw, values


def _routing_inputs(case, seed):
    """Rows, router logits (some experts are liked more than others), selection bias, the shared expert's result."""
    h, _, _ = SHAPES[case["fmt"]]
    t, g = case["tokens"], _gen(seed, 5)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    return r(t, h).bfloat16(), r(t, EXPERTS) * 1.5 + r(EXPERTS) * 0.5, r(EXPERTS) * 0.02, r(t, h).bfloat16()


def _score(fmt):
    return ("sqrtsoftplus", 1.5) if fmt == "fp4" else ("sigmoid", 1.0)


def prepare(case, seed):
    if case["kind"] == "serve":
        from deepseek_v4_2080ti_b200.models import qwen_hybrid as qh
        cfg = qh.QwenHybridConfig(num_hidden_layers=LAYERS, vocab_size=VOCAB)
        weights = qh.QwenHybridWeights(cfg, _checkpoint(seed), DEV)
        prompts, given = _tokens(case, seed)
        longest = max(p.numel() for p in prompts) + case["new"]
        rt = qh.QwenHybridRuntime(cfg, weights, max_slots=case["batch"], max_context=(longest + 127) // 64 * 64, kv_cache_dtype=case["kv"])
        return {"case": case, "rt": rt, "prompts": prompts, "given": given}
    from deepseek_v4_2080ti_b200.ops import moe
    fmt = case["fmt"]
    h, inter, _ = SHAPES[fmt]
    parts = [(a[0], b[0]) for a, b in _pool(fmt, seed)] * (EXPERTS // POOL)
    if fmt == "fp4":
        w13, w2 = (moe.ExpertWeights.from_fp4([p[j][0] for p in parts], [p[j][1] for p in parts]) for j in (0, 1))
    else:
        from deepseek_v4_2080ti_b200.formats.gguf import GGMLType
        w13 = moe.ExpertWeights.from_gguf([p[0] for p in parts], GGMLType.Q4_K, 2 * inter, h)
        w2 = moe.ExpertWeights.from_gguf([p[1] for p in parts], GGMLType.Q2_K, h, inter)
    return {"case": case, "w13": w13, "w2": w2, "in": _routing_inputs(case, seed)}


def run(state):
    case = state["case"]
    if case["kind"] == "experts":
        from deepseek_v4_2080ti_b200.ops import moe
        x, logits, bias, shared = state["in"]
        score, scale = _score(case["fmt"])
        idx, wts = moe.route(logits, bias, SHAPES[case["fmt"]][2], score, True, scale)
        y = moe.experts_forward(x, idx, wts, state["w13"], state["w2"], 0, base=shared)
        return {"experts": idx, "weights": wts, "out": y}
    rt = state["rt"]
    slots = [rt.allocate() for _ in state["prompts"]]
    first = []
    for slot, prompt in zip(slots, state["prompts"]):
        rt.prefill(slot, prompt)
        first.append(rt.last_logits)
    steps = []
    for ids in state["given"]:
        rt.decode(slots, ids)
        steps.append(rt.last_logits.clone())          # the step's buffer is written again by the next one
    for slot in reversed(slots):                      # the next requests get the same slots
        rt.free(slot)
    return {"first": torch.cat(first), "steps": torch.stack(steps) if steps else None, "states": rt.states, "tails": rt.tails}


# ------------------------------------------------------------------------------------------------ what a pass needs
MATRIX = {False: (2 * KD + 2 * VD) * HIDDEN + VD * HIDDEN, True: (2 * HQ + 2 * HKV) * D * HIDDEN + HQ * D * HIDDEN}


def _layer_params():
    """FP8 and bf16 weights of all layers."""
    n = sum(MATRIX[_is_full(i)] + 3 * WIDE * HIDDEN for i in range(LAYERS))
    return n, sum(2 * HV * HIDDEN for i in range(LAYERS) if not _is_full(i))


def _distinct(case):
    """Expected number of experts that get a token."""
    k = SHAPES[case["fmt"]][2]
    return EXPERTS * (1.0 - (1.0 - k / EXPERTS) ** case["tokens"])


def work(case):
    if case["kind"] == "experts":
        h, inter, k = SHAPES[case["fmt"]]
        t = case["tokens"]
        bits = (4.25, 4.25) if case["fmt"] == "fp4" else (4.5, 2.625)
        expert = (2 * h * inter * bits[0] + h * inter * bits[1]) / 8
        return {"bytes": _distinct(case) * expert + 6 * t * h + 4 * t * EXPERTS + 8 * t * k, "flops": 6.0 * t * k * h * inter}
    fp8, bf16 = _layer_params()
    lens, new = _lengths(case), case["new"]
    full = sum(_is_full(i) for i in range(LAYERS))
    lin = LAYERS - full
    kv_row = 2 * full * HKV * (2 * D if case["kv"] == "bf16" else D + 4)
    head = 2 * VOCAB * HIDDEN
    weights = fp8 + 4 * fp8 / (128 * 128) + 2 * bf16 + head
    state = lin * HV * D * D * 4
    b = flops = 0.0
    for n in lens:                                      # a prompt: the weights once, its rows, its state and cache rows written
        b += weights + n * (2 * HIDDEN + 4) + state + n * kv_row + 4 * VOCAB
        flops += 2.0 * n * (fp8 + bf16) + 2.0 * VOCAB * HIDDEN + full * 2.0 * n * n * HQ * D + lin * n * HV * 6.0 * D * D
    for j in range(new):                                # a step: the weights once, states read and written, contexts read
        ctx = sum(n + j + 1 for n in lens)
        b += weights + len(lens) * (2 * state + 4 * VOCAB) + ctx * kv_row
        flops += len(lens) * (2.0 * (fp8 + bf16 + VOCAB * HIDDEN) + lin * HV * 6.0 * D * D) + full * 4.0 * ctx * HQ * D
    return {"bytes": b, "flops": flops}


def tolerance(case):
    """bf16 activations between the kernels.  Served requests are 0.007 to 0.013 off the 64-bit values (2-norm, each output) at
    every size, rounding of stored activations through 8 layers, so two correct evaluations with unrelated roundings
    differ by up to 0.018, and their largest single difference, over the millions of values of an output, was 0.24 to 0.38 of
    its root mean square; one expert block is 0.003 off."""
    return {"rel": 0.03, "max": 0.8} if case["kind"] == "serve" else {"rel": 0.01, "max": 0.1, "differ": 0.001}


# ------------------------------------------------------------------------------------------------ 64-bit statement
def _mat(t):
    w, s = t
    n, k = w.shape
    return (w.double().view(n // 128, 128, k // 128, 128) * s.double()[:, None, :, None]).view(n, k)


def _norm(x, gamma, add=1.0):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * (add + gamma.double())


def _rope(x, pos):
    half = ROT // 2
    inv = THETA ** (-torch.arange(0, ROT, 2, device=DEV, dtype=torch.float64) / ROT)
    ang = pos.double()[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:ROT]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., ROT:]], -1)


def _attention(x, t, pre):
    """x [B, L, hidden], all rows causal from position 0."""
    b, n, _ = x.shape
    pos = torch.arange(n, device=DEV)
    qg = (x @ _mat(t[pre + "q_proj"]).t()).view(b, n, HQ, 2 * D)
    k = _rope(_norm((x @ _mat(t[pre + "k_proj"]).t()).view(b, n, HKV, D), t[pre + "k_norm.weight"]), pos)
    v = (x @ _mat(t[pre + "v_proj"]).t()).view(b, n, HKV, D)
    q = _rope(_norm(qg[..., :D], t[pre + "q_norm.weight"]), pos)
    out = torch.empty(b, n, HQ, D, dtype=torch.float64, device=DEV)
    rep = HQ // HKV
    for i in range(b):
        for h in range(HQ):
            for lo in range(0, n, 2048):
                hi = min(n, lo + 2048)
                s = q[i, lo:hi, h] @ k[i, :hi, h // rep].t() / math.sqrt(D)
                s.masked_fill_(pos[None, :hi] > pos[lo:hi, None], float("-inf"))
                out[i, lo:hi, h] = s.softmax(-1) @ v[i, :hi, h // rep]
    out *= torch.sigmoid(qg[..., D:])
    return out.view(b, n, HQ * D) @ _mat(t[pre + "o_proj"]).t()


def _delta_rule(x, t, pre, live):
    """x [B, L, hidden]; ``live`` [B, L]: rows that are there.  Returns (result, state [B, HV, D, D], qkv rows)."""
    b, n, _ = x.shape
    qkv = x @ _mat(t[pre + "in_proj_qkv"]).t()
    z = (x @ _mat(t[pre + "in_proj_z"]).t()).view(b, n, HV, D)
    beta = torch.sigmoid(x @ t[pre + "in_proj_b.weight"].double().t()) * live[..., None]
    g = -t[pre + "A_log"].double().exp() * F.softplus(x @ t[pre + "in_proj_a.weight"].double().t() + t[pre + "dt_bias"].double())
    decay = (g * live[..., None]).exp()
    w = t[pre + "conv1d.weight"].double().view(-1, 4)
    past = torch.cat([qkv.new_zeros(b, 3, qkv.shape[-1]), qkv], 1)
    mixed = F.silu(sum(past[:, j:j + n] * w[:, j] for j in range(4)))
    unit = lambda y: y * torch.rsqrt(y.square().sum(-1, keepdim=True) + 1e-6)
    q = unit(mixed[..., :KD].view(b, n, HK, D)).repeat_interleave(HV // HK, 2) * D ** -0.5
    k = unit(mixed[..., KD:2 * KD].view(b, n, HK, D)).repeat_interleave(HV // HK, 2)
    v = mixed[..., 2 * KD:].view(b, n, HV, D)
    s = x.new_zeros(b, HV, D, D)
    core = torch.empty_like(v)
    for i in range(n):
        s *= decay[:, i, :, None, None]
        d = (v[:, i] - (k[:, i, :, None] @ s)[:, :, 0]) * beta[:, i, :, None]
        s += k[:, i, :, :, None] * d[:, :, None]
        core[:, i] = (q[:, i, :, None] @ s)[:, :, 0]
    y = _norm(core, t[pre + "norm.weight"], 0.0) * F.silu(z)
    return y.reshape(b, n, VD) @ _mat(t[pre + "out_proj"]).t(), s, qkv


def _exact_serve(case, seed):
    prompts, given = _tokens(case, seed)
    lens, new = [p.numel() for p in prompts], case["new"]
    batch, total = len(lens), max(lens) + new
    ids = torch.zeros(batch, total, dtype=torch.long, device=DEV)
    for i, p in enumerate(prompts):
        ids[i, :lens[i] + new] = torch.cat([p, given[:, i]]).long()
    end = torch.tensor(lens, device=DEV) + new
    live = (torch.arange(total, device=DEV)[None] < end[:, None]).double()
    embed, head, norm = _ends(seed)
    h = embed[ids].double()
    states, tails = [], []
    for l in range(LAYERS):
        t = _layer(seed, l)
        x = _norm(h, t["input_layernorm.weight"])
        if _is_full(l):
            h = h + _attention(x, t, "self_attn.")
        else:
            y, s, qkv = _delta_rule(x, t, "linear_attn.", live)
            h = h + y
            states.append(s)
            past = torch.cat([qkv.new_zeros(batch, 3, qkv.shape[-1]), qkv], 1)
            tails.append(torch.stack([past[i, int(e):int(e) + 3] for i, e in enumerate(end)]))
        x = _norm(h, t["post_attention_layernorm.weight"])
        gate, up, down = (_mat(t["mlp." + m + "_proj"]) for m in ("gate", "up", "down"))
        for i in range(batch):
            h[i] += (F.silu(x[i] @ gate.t()) * (x[i] @ up.t())) @ down.t()
        del gate, up, down
    rows = torch.stack([h[i, n - 1:n + new] for i, n in enumerate(lens)])               # [batch, 1 + new, hidden]
    logits = _norm(rows, norm) @ head.double().t()
    return {"first": logits[:, 0], "steps": logits[:, 1:].transpose(0, 1) if new else None, "states": torch.stack(states, 1), "tails": torch.stack(tails, 1)}


def _exact_experts(case, seed):
    x, logits, bias, shared = (v.double() for v in _routing_inputs(case, seed))
    fmt = case["fmt"]
    _, inter, k = SHAPES[fmt]
    name, scale = _score(fmt)
    score = F.softplus(logits).sqrt() if name == "sqrtsoftplus" else torch.sigmoid(logits)
    idx = (score + bias).topk(k, -1).indices
    wts = score.gather(-1, idx)
    wts = wts / wts.sum(-1, keepdim=True) * scale
    out = shared.clone()
    for j, ((_, w13), (_, w2)) in enumerate(_pool(fmt, seed)):
        here = idx % POOL == j                                                # experts j, j + POOL, ... have the same weights
        for c in range(k):
            rows = here[:, c].nonzero()[:, 0]
            if rows.numel():
                gu = x[rows] @ w13().t()
                out[rows] += wts[rows, c, None] * ((F.silu(gu[:, :inter]) * gu[:, inter:]) @ w2().t())
    return {"experts": None, "weights": wts, "out": out}


@torch.no_grad()
def exact(case, seed):
    return _exact_serve(case, seed) if case["kind"] == "serve" else _exact_experts(case, seed)
