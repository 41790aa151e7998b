"""The calls whose speed is watched, with their inputs, their exact results and how far a correct result may be from them.

A case is a call that a program built on the library makes: whole steps of a model through `Engine`, and single layers, mixers
and feed-forwards through their parts' `forward`, which is how another arrangement is put together.  Sizes are those of
`bench.py` (GPT-J-6B) and of the design benchmarks (width 2,048 or 4,096, heads of 128, 16 experts).

    listed()          the cases that stand for the library's use
    draw(rng)         one more of the same ranges
    prepare(c, seed)  weights, cache and inputs on the device, from the seed alone
    run(state)        one pass
    exact(c, seed)    its results in 64 bits, from torch alone
    work(c)           bytes and operations that no implementation can do without
    tolerance(c)      what another correct implementation at the same precision may differ by
"""
from __future__ import annotations

import math
import zlib

import torch
import torch.nn.functional as F

import qstream_b200 as qs
from qstream_b200.cache import SequenceCache
from qstream_b200.config import AttentionSpec, BlockSpec, MlpSpec, NormSpec, PositionHalfSpec, PositionSpec
from qstream_b200.config.specs import DecayAttentionSpec, GatedDeltaSpec, GlaSpec, Mamba2Spec, RoutedExpertsSpec
from qstream_b200.engine.step import StepBatch, StepContext
from qstream_b200.parts import Runtime, build_block, part_class

DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
BYTES = {"bfloat16": 2, "float32": 4}
DEVICE = "cuda"


def listed():
    return [
        # a short request on a small model, from its prompt to its last token: launches and latency are all there is to it
        {"name": "request 1x24+8", "kind": "request", "seqs": 1, "tokens": 24, "new": 8},
        # the headline workload: one decode step of GPT-J-6B for eight users in mid-conversation
        {"name": "decode 8x1024", "kind": "decode", "seqs": 8, "tokens": 1024},
        # a layer of the same model over a whole prompt: the long-prompt half of serving it
        {"name": "layer bf16 2048", "kind": "layer", "dtype": "bfloat16", "width": 4096, "seqs": 1, "tokens": 2048},
        # the 32-bit engine, which users run to check a model and the tests run throughout: a ragged pair of prompts
        {"name": "layer fp32 2x350", "kind": "layer", "dtype": "float32", "width": 2048, "seqs": 2, "tokens": 700},
        # grouped-key attention with a cap and a gate: prompts of three users arriving together
        {"name": "attention prompt 3", "kind": "attention", "step": "prompt", "seqs": 3, "tokens": 2047},
        # the same mixer while 32 users decode
        {"name": "attention decode 32", "kind": "attention", "step": "decode", "seqs": 32, "tokens": 2048},
        # routed experts in a decode step of eight users, at the larger width
        {"name": "experts 8", "kind": "experts", "width": 4096, "tokens": 8},
        # routed experts over a batch of prompts
        {"name": "experts 3000", "kind": "experts", "width": 2048, "tokens": 3000},
        # linear attention with a decay per head over one long prompt
        {"name": "lightning 4096", "kind": "lightning", "seqs": 1, "tokens": 4096},
        # gated linear attention (a decay per key channel) over two unequal prompts
        {"name": "gla 2x1700", "kind": "gla", "seqs": 2, "tokens": 3401},
        # Mamba-2 over one prompt
        {"name": "mamba2 2048", "kind": "mamba2", "seqs": 1, "tokens": 2048},
        # the gated delta rule over one prompt of an odd length
        {"name": "delta 1999", "kind": "delta", "seqs": 1, "tokens": 1999},
    ]


def draw(rng):
    def log(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))

    kind = rng.choice(("request", "decode", "layer", "layer", "attention", "attention", "experts", "experts", "lightning", "gla", "mamba2", "delta"))
    if kind == "request":
        return {"kind": kind, "seqs": log(1, 4), "tokens": log(4, 120), "new": rng.randint(3, 8)}
    if kind == "decode":
        return {"kind": kind, "seqs": log(1, 8), "tokens": log(32, 1024)}
    if kind == "layer":
        if rng.random() < 0.5:
            return {"kind": kind, "dtype": "float32", "width": 2048, "seqs": rng.randint(1, 3), "tokens": log(4, 700)}
        return {"kind": kind, "dtype": "bfloat16", "width": rng.choice((2048, 4096)), "seqs": rng.randint(1, 4), "tokens": log(8, 2048)}
    if kind == "attention":
        if rng.random() < 0.5:
            return {"kind": kind, "step": "decode", "seqs": log(1, 32), "tokens": log(16, 2048)}
        return {"kind": kind, "step": "prompt", "seqs": rng.randint(1, 4), "tokens": log(8, 2047)}
    if kind == "experts":
        if rng.random() < 0.5:
            return {"kind": kind, "width": rng.choice((2048, 4096)), "tokens": log(1, 32)}
        return {"kind": kind, "width": 2048, "tokens": log(33, 3000)}
    if rng.random() < 0.3:                              # a decode step: one token per sequence
        n = log(1, 32)
        return {"kind": kind, "seqs": n, "tokens": n}
    most = {"lightning": 4096, "gla": 3401, "mamba2": 2048, "delta": 1999}[kind]
    return {"kind": kind, "seqs": rng.randint(1, 4), "tokens": log(32, most)}


# ---------------------------------------------------------------------------------------------------- inputs from a seed

def _random(seed, name, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    """Normal numbers that depend on the seed and the name alone."""
    g = torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
    t = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32 if dtype == torch.float32 else torch.bfloat16)
    return t.mul_(std).add_(mean).to(dtype)


def _uniform(seed, name, shape, lo, hi):
    g = torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
    return torch.rand(shape, generator=g, device=DEVICE, dtype=torch.float32) * (hi - lo) + lo


def _tokens(seed, name, n, vocab):
    g = torch.Generator().manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))
    return torch.randint(0, vocab, (n,), generator=g).tolist()


def _lengths(total, seqs):
    """`total` tokens over `seqs` sequences, unequally where there are several: 4 : 3 : 2 : 2 ..., at least one each."""
    shares = [max(2, 4 - i) for i in range(seqs)]
    total = max(total, seqs)
    out = [max(1, total * s // sum(shares)) for s in shares]
    out[0] += total - sum(out)
    return out


def _step(cache, slots, new_tokens):
    """A step in which `slots[i]` brings `new_tokens[i]` tokens."""
    cache.prepare(slots, new_tokens)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32).to(DEVICE)      # noqa: E731
    p0 = [cache.length(s) for s in slots]
    slot_of = [s for s, n in zip(slots, new_tokens) for _ in range(n)]
    pos_of = [p + i for p, n in zip(p0, new_tokens) for i in range(n)]
    start = [0]
    for n in new_tokens:
        start.append(start[-1] + n)
    batch = StepBatch(n_seq=len(slots), n_tokens=len(slot_of), n_want=0, tokens=i32([0] * len(slot_of)), tok_slot=i32(slot_of),
                      tok_pos=i32(pos_of), want_rows=i32([]), seq_slot=i32(slots), seq_start=i32(start), seq_p0=i32(p0),
                      slots=list(slots), new_tokens=list(new_tokens), p0=p0, decode=all(n == 1 for n in new_tokens),
                      max_new=max(new_tokens), max_total=max(p + n for p, n in zip(p0, new_tokens)))
    return StepContext(batch, cache, torch.zeros(1, dtype=torch.int32, device=DEVICE))


def _cache(part, seqs, tokens, dtype):
    kv, state = part.kv_need(), part.state_need()
    pages = sum(-(-n // 64) for n in tokens)
    return SequenceCache({0: kv} if kv else {}, {0: state} if state else {}, 64 * pages, seqs, max(tokens), DTYPES[dtype], DEVICE)


# ---------------------------------------------------------------------------------------------------- GPT-J, whole and by layer

def _gptj(case):
    """(width, layers, heads, head size, inner, vocabulary)."""
    if case["kind"] == "decode":
        return 4096, 28, 16, 256, 16384, 50400
    if case["kind"] == "request":
        return 2048, 8, 16, 128, 8192, 32000
    width = case["width"]
    return width, 1, 16, width // 16, 4 * width, 0


ROT = 64


def _layer_shapes(D, inner):
    """Own names of a GPT-J layer's tensors: (shape, standard deviation, mean)."""
    return {"ln.weight": ((D,), 0.1, 1.0), "ln.bias": ((D,), 0.02, 0.0), "q": ((D, D), 0.02, 0.0), "k": ((D, D), 0.02, 0.0),
            "v": ((D, D), 0.02, 0.0), "out": ((D, D), 0.02, 0.0), "up": ((inner, D), 0.02, 0.0), "up_bias": ((inner,), 0.02, 0.0),
            "down": ((D, inner), 0.02, 0.0), "down_bias": ((D,), 0.02, 0.0)}


CHECKPOINT = {"ln.weight": "ln_1.weight", "ln.bias": "ln_1.bias", "q": "attn.q_proj.weight", "k": "attn.k_proj.weight",
              "v": "attn.v_proj.weight", "out": "attn.out_proj.weight", "up": "mlp.fc_in.weight", "up_bias": "mlp.fc_in.bias",
              "down": "mlp.fc_out.weight", "down_bias": "mlp.fc_out.bias"}


def _layer_tensors(seed, i, D, inner, dtype):
    return {n: _random(seed, f"{i}.{n}", shape, std, mean, dtype) for n, (shape, std, mean) in _layer_shapes(D, inner).items()}


def _ends(seed, D, vocab, dtype):
    """The model's tensors outside its layers, by checkpoint name."""
    made = {"transformer.wte.weight": ((vocab, D), 1.0, 0.0), "transformer.ln_f.weight": ((D,), 0.1, 1.0),
            "transformer.ln_f.bias": ((D,), 0.02, 0.0), "lm_head.weight": ((vocab, D), 0.02, 0.0), "lm_head.bias": ((vocab,), 0.02, 0.0)}
    return {n: _random(seed, n, shape, std, mean, dtype) for n, (shape, std, mean) in made.items()}


def _model(case, seed):
    D, L, H, _, inner, vocab = _gptj(case)
    config = qs.GptjConfig.from_dict(dict(n_layer=L, n_embd=D, n_head=H, n_positions=8192, vocab_size=vocab, rotary_dim=ROT, n_inner=inner,
                                          activation_function="gelu_new", layer_norm_epsilon=1e-5, architectures=["GPTJForCausalLM"]))
    tensors = _ends(seed, D, vocab, torch.bfloat16)
    for i in range(L):
        tensors.update({f"transformer.h.{i}.{CHECKPOINT[n]}": t for n, t in _layer_tensors(seed, i, D, inner, torch.bfloat16).items()})
    return qs.CausalLM(config.model_spec(), tensors, "bfloat16", DEVICE, config)


def _decode_lengths(case):
    """The users' contexts before the step: all of one length for a full batch, unequal for others."""
    n, most = case["seqs"], case["tokens"]
    return [most] * n if n == 8 else [max(1, most - (most * i) // (2 * n)) for i in range(n)]


def _prepare_model(case, seed):
    model = _model(case, seed)
    vocab = model.vocab_size
    n = case["seqs"]
    if case["kind"] == "request":
        engine = qs.Engine(model, max_batch=n, max_context=256, max_tokens=256 * n)
        lengths = _lengths(case["tokens"], n)
        prompts = [_tokens(seed, f"prompt{i}", m, vocab) for i, m in enumerate(lengths)]
        more = [[[t] for t in _tokens(seed, f"more{j}", n, vocab)] for j in range(case["new"])]
        return {"kind": "request", "engine": engine, "prompts": prompts, "more": more}
    engine = qs.Engine(model, max_batch=n, max_context=4096, max_tokens=4096 * n)
    slots = [engine.acquire() for _ in range(n)]
    for i, m in enumerate(_decode_lengths(case)):
        engine.step([slots[i]], [_tokens(seed, f"context{i}", m, vocab)])
    feed = [[[t] for t in _tokens(seed, f"feed{j}", n, vocab)] for j in range(64)]
    return {"kind": "decode", "engine": engine, "slots": slots, "feed": feed, "at": 0}


def _run_request(s):
    """A request served from beginning to end; its tokens are given, so that one pass is like another."""
    engine = s["engine"]
    slots = [engine.acquire() for _ in s["prompts"]]
    logits = [engine.step(slots, s["prompts"]).clone()]
    for tokens in s["more"]:
        logits.append(engine.step(slots, tokens).clone())
    for slot in slots:
        engine.release(slot)
    return logits


def _run_decode(s):
    """One step further in each user's sequence."""
    tokens = s["feed"][s["at"] % len(s["feed"])]
    s["at"] += 1
    return s["engine"].step(s["slots"], tokens)


def _norm64(x, w, b):
    m = x.mean(-1, keepdim=True)
    v = (x - m).square().mean(-1, keepdim=True)
    return (x - m) / torch.sqrt(v + 1e-5) * w.double() + b.double()


def _rotate64(x, interleaved):
    """x [n, heads, dh] of one sequence from its first token on."""
    i = torch.arange(0, ROT, 2, dtype=torch.float64, device=x.device)
    ang = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * torch.pow(10000.0, -i / ROT)
    c, s = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
    y = x.clone()
    first, second = (slice(0, ROT, 2), slice(1, ROT, 2)) if interleaved else (slice(0, ROT // 2), slice(ROT // 2, ROT))
    a, b = x[..., first], x[..., second]
    y[..., first], y[..., second] = a * c - b * s, a * s + b * c
    return y


def _attend64(q, k, v, scale, cap=0.0, last_only=False):
    """q [n, H, dh], k [n, G, dh], v [n, G, dv] of one sequence -> [n, H, dv] ([1, H, dv] for the last query alone)."""
    n, H, G = k.shape[0], q.shape[1], k.shape[1]
    out = []
    rows = torch.arange(n, device=q.device)
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if not last_only:
            s = s.masked_fill(rows[None, :] > rows[:, None], -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, h * G // H])
    return torch.stack(out, 1)


def _gptj_layer64(x, lengths, w, H):
    D = x.shape[1]
    w = {n: t.double() for n, t in w.items()}
    h = _norm64(x, w["ln.weight"], w["ln.bias"])
    q, k, v = ((h @ w[n].T).view(-1, H, D // H) for n in ("q", "k", "v"))
    o, at = [], 0
    for n in lengths:
        r = slice(at, at + n)
        o.append(_attend64(_rotate64(q[r], True), _rotate64(k[r], True), v[r], (D // H) ** -0.5))
        at += n
    o = torch.cat(o).reshape(-1, D)
    g = F.gelu(h @ w["up"].T + w["up_bias"], approximate="tanh")
    return x + o @ w["out"].T + g @ w["down"].T + w["down_bias"]


def _exact_model(case, seed):
    D, L, H, _, inner, vocab = _gptj(case)
    n = case["seqs"]
    if case["kind"] == "request":
        lengths = _lengths(case["tokens"], n)
        texts = [_tokens(seed, f"prompt{i}", m, vocab) for i, m in enumerate(lengths)]
        more = [_tokens(seed, f"more{j}", n, vocab) for j in range(case["new"])]
    else:
        lengths = _decode_lengths(case)
        texts = [_tokens(seed, f"context{i}", m, vocab) for i, m in enumerate(lengths)]
        more = [_tokens(seed, "feed0", n, vocab)]
    texts = [t + [m[i] for m in more] for i, t in enumerate(texts)]
    ends = _ends(seed, D, vocab, torch.bfloat16)
    x = ends["transformer.wte.weight"][torch.tensor([t for text in texts for t in text], device=DEVICE)].double()
    whole = [len(t) for t in texts]
    for i in range(L):
        x = _gptj_layer64(x, whole, _layer_tensors(seed, i, D, inner, torch.bfloat16), H)
    first = [sum(whole[:i]) for i in range(n)]
    head, bias = ends["lm_head.weight"].double(), ends["lm_head.bias"].double()

    def logits(steps_in):
        rows = torch.tensor([first[i] + lengths[i] - 1 + steps_in for i in range(n)], device=DEVICE)
        return _norm64(x[rows], ends["transformer.ln_f.weight"], ends["transformer.ln_f.bias"]) @ head.T + bias

    return [logits(j) for j in range(len(more) + 1)] if case["kind"] == "request" else logits(1)


def _prepare_layer(case, seed):
    D, _, H, dh, inner, _ = _gptj(case)
    dtype = DTYPES[case["dtype"]]
    w = _layer_tensors(seed, 0, D, inner, dtype)
    norm = NormSpec(size=D, eps=1e-5, bias=True)
    spec = BlockSpec(arrangement="parallel", norms={"input": norm},
                     mixer=AttentionSpec(width=D, n_heads=H, n_kv_heads=H, head_dim=dh, position=PositionSpec(rotary_dim=ROT, base=10000.0, max_positions=8192)),
                     ffn=MlpSpec(width=D, inner=inner, activation="gelu_new"))
    block = build_block(spec, lambda part, decls: {n: w["ln." + n if part is norm else n] for n in decls}, Runtime(dtype, torch.device(DEVICE)))
    lengths = _lengths(case["tokens"], case["seqs"])
    cache = _cache(block.mixer, len(lengths), lengths, case["dtype"])
    slots = [cache.acquire() for _ in lengths]
    return {"kind": "layer", "block": block, "x": _random(seed, "x", (sum(lengths), D), 1.0, 0.0, dtype), "step": _step(cache, slots, lengths)}


def _run_layer(s):
    view = s["step"].kv(0)
    return [s["block"].forward(s["x"], s["step"], 0), view.k[:-1], view.v[:-1]]


def _exact_layer(case, seed):
    D, _, H, _, inner, _ = _gptj(case)
    dtype = DTYPES[case["dtype"]]
    lengths = _lengths(case["tokens"], case["seqs"])
    x = _random(seed, "x", (sum(lengths), D), 1.0, 0.0, dtype).double()
    return [_gptj_layer64(x, lengths, _layer_tensors(seed, 0, D, inner, dtype), H), None, None]


# ---------------------------------------------------------------------------------------------------- attention by itself

ATT_D, ATT_H, ATT_G, ATT_DH, ATT_CAP = 2048, 16, 4, 128, 50.0


def _part(role, spec, seed, shapes, dtype="bfloat16"):
    """A part with the tensors that `shapes` (own name -> (shape, standard deviation, mean) or a tensor) describes."""
    tensors = {n: t if isinstance(t, torch.Tensor) else _random(seed, n, t[0], t[1], t[2], DTYPES[dtype]) for n, t in shapes.items()}
    return part_class(role, spec.kind)(spec, tensors, Runtime(DTYPES[dtype], torch.device(DEVICE))), tensors


def _attention_shapes():
    hq, hkv = ATT_H * ATT_DH, ATT_G * ATT_DH
    return {"q": ((hq, ATT_D), 0.02, 0.0), "k": ((hkv, ATT_D), 0.02, 0.0), "v": ((hkv, ATT_D), 0.02, 0.0), "gate": ((hq, ATT_D), 0.02, 0.0),
            "out": ((ATT_D, hq), 0.02, 0.0)}


def _attention_lengths(case):
    if case["step"] == "prompt":
        return _lengths(case["tokens"], case["seqs"])
    most, n = case["tokens"], case["seqs"]
    return [max(1, most - (i * most) // (4 * n)) for i in range(n)]


def _prepare_attention(case, seed):
    spec = AttentionSpec(width=ATT_D, n_heads=ATT_H, n_kv_heads=ATT_G, head_dim=ATT_DH, softcap=ATT_CAP, gate=True,
                         position=PositionHalfSpec(rotary_dim=ROT, base=10000.0, max_positions=8192))
    part, _ = _part("mixer", spec, seed, _attention_shapes())
    lengths = _attention_lengths(case)
    decode = case["step"] == "decode"
    total = [n + 1 for n in lengths] if decode else lengths
    cache = _cache(part, len(lengths), total, "bfloat16")
    slots = [cache.acquire() for _ in lengths]
    if decode:                                          # the users' contexts, a few sequences at a time
        for i, n in enumerate(lengths):
            part.forward(_random(seed, f"context{i}", (n, ATT_D)), _step(cache, [slots[i]], [n]), 0)
            cache.commit([slots[i]], [n])
        lengths = [1] * len(slots)
    return {"kind": "mixer", "part": part, "h": _random(seed, "h", (sum(lengths), ATT_D)), "step": _step(cache, slots, lengths)}


def _exact_attention(case, seed):
    w = {n: _random(seed, n, *t).double() for n, t in _attention_shapes().items()}
    lengths = _attention_lengths(case)
    decode = case["step"] == "decode"
    h = _random(seed, "h", (len(lengths) if decode else sum(lengths), ATT_D)).double()
    out, at = [], 0
    for i, n in enumerate(lengths):
        mine = torch.cat([_random(seed, f"context{i}", (n, ATT_D)).double(), h[i:i + 1]]) if decode else h[at:at + n]
        at += n
        k = _rotate64((mine @ w["k"].T).view(-1, ATT_G, ATT_DH), False)
        v = (mine @ w["v"].T).view(-1, ATT_G, ATT_DH)
        if decode:
            q = torch.zeros(n + 1, ATT_H, ATT_DH, dtype=torch.float64, device=DEVICE)
            q[-1] = (mine[-1:] @ w["q"].T).view(ATT_H, ATT_DH)
            q = _rotate64(q, False)[-1:]
        else:
            q = _rotate64((mine @ w["q"].T).view(-1, ATT_H, ATT_DH), False)
        out.append(_attend64(q, k, v, ATT_DH ** -0.5, ATT_CAP, last_only=decode).reshape(-1, ATT_H * ATT_DH))
    return [torch.cat(out) * torch.sigmoid(h @ w["gate"].T) @ w["out"].T, None, None]


def _run_mixer(s):
    """The mixer's result and what it leaves for the next step: keys and values, or its states."""
    step = s["step"]
    out = s["part"].forward(s["h"], step, 0)
    if step.cache.has_entry(0):
        view = step.kv(0)
        return [out, view.k[:-1], view.v[:-1]]
    state = step.state(0)
    return [out, *(state[n] for n in sorted(state))] if isinstance(state, dict) else [out, state]


# ---------------------------------------------------------------------------------------------------- routed experts

EXPERTS, TOP = 16, 4


def _experts_shapes(case):
    D, inner = case["width"], case["width"] // 4
    shapes = {"router": ((EXPERTS, D), 0.02, 0.0)}
    for e in range(EXPERTS):
        shapes.update({f"up{e}": ((inner, D), 0.02, 0.0), f"gate{e}": ((inner, D), 0.02, 0.0), f"down{e}": ((D, inner), 0.02, 0.0)})
    return shapes


class _Rows:
    """What a feed-forward needs to know of its step: which rows are tokens, and whether each is a sequence's only one."""

    def __init__(self, n, decode):
        self.batch = StepBatch(n_seq=n if decode else 1, n_tokens=n, n_want=0, tokens=None, tok_slot=torch.zeros(n, dtype=torch.int32, device=DEVICE),
                               tok_pos=None, want_rows=None, seq_slot=None, seq_start=None, seq_p0=None, new_tokens=[1] * n if decode else [n],
                               decode=decode)


def _prepare_experts(case, seed):
    D = case["width"]
    spec = RoutedExpertsSpec(width=D, n_experts=EXPERTS, inner=D // 4, top=TOP, scores="softmax", correction=False, gated="act", activation="silu",
                             normalize=True)
    part, _ = _part("feed_forward", spec, seed, _experts_shapes(case))
    n = case["tokens"]
    return {"kind": "experts", "part": part, "h": _random(seed, "h", (n, D)), "step": _Rows(n, n <= 32)}


def _exact_experts(case, seed):
    w = {n: _random(seed, n, *t) for n, t in _experts_shapes(case).items()}
    h = _random(seed, "h", (case["tokens"], case["width"])).double()
    s, idx = torch.softmax(h @ w["router"].double().T, -1).topk(TOP, -1)
    s = s / s.sum(-1, keepdim=True)
    out = torch.zeros_like(h)
    for e in range(EXPERTS):
        t, j = (idx == e).nonzero(as_tuple=True)
        y = F.silu(h[t] @ w[f"gate{e}"].double().T) * (h[t] @ w[f"up{e}"].double().T)
        out.index_add_(0, t, y @ w[f"down{e}"].double().T * s[t, j][:, None])
    return out


# ---------------------------------------------------------------------------------------------------- mixers with a matrix of state per head

REC_D, LIGHT_H = 2048, 16
LIGHT_DECAY = tuple(1.0 - 2.0 ** (-5.0 - 5.0 * i / (LIGHT_H - 1)) for i in range(LIGHT_H))
GLA_DK, GLA_DV, GLA_RANK, GLA_TAU = 64, 128, 64, 16.0
SSD_H, SSD_DV, SSD_N, TAPS = 64, 64, 128, 4
DELTA_H, DELTA_G, DELTA_D, DELTA_RANK = 16, 8, 128, 64
EPS = 1e-5


def _step_biases(seed, n):
    """Biases behind which softplus gives step sizes between 0.001 and 0.1, as these mixers are initialised."""
    dt = torch.exp(_uniform(seed, "dt_bias", (n,), math.log(0.001), math.log(0.1)))
    return dt + torch.log(-torch.expm1(-dt))


def _rates(seed, n):
    return torch.log(_uniform(seed, "A_log", (n,), 1.0, 16.0))


def _recurrent(case, seed):
    """(spec, tensors) of the case's mixer."""
    D, kind = REC_D, case["kind"]
    if kind == "lightning":
        n = LIGHT_H * 128
        spec = DecayAttentionSpec(width=D, n_heads=LIGHT_H, key_dim=128, value_dim=128, decay=LIGHT_DECAY, eps=EPS)
        shapes = {**{m: ((n, D), 0.02, 0.0) for m in "qkvg"}, "o": ((D, n), 0.02, 0.0), "norm": ((n,), 0.1, 1.0)}
    elif kind == "gla":
        hk, hv = LIGHT_H * GLA_DK, LIGHT_H * GLA_DV
        spec = GlaSpec(width=D, n_heads=LIGHT_H, key_dim=GLA_DK, value_dim=GLA_DV, tau=GLA_TAU, eps=EPS, decay_rank=GLA_RANK)
        shapes = {"q": ((hk, D), 0.02, 0.0), "k": ((hk, D), 0.02, 0.0), "v": ((hv, D), 0.02, 0.0), "g": ((hv, D), 0.02, 0.0), "o": ((D, hv), 0.02, 0.0),
                  "norm": ((GLA_DV,), 0.1, 1.0), "a1": ((GLA_RANK, D), 0.02, 0.0), "a2": ((hk, GLA_RANK), 0.1, 0.0), "a2_bias": ((hk,), 0.5, 0.0)}
    elif kind == "mamba2":
        n = SSD_H * SSD_DV
        spec = Mamba2Spec(width=D, n_heads=SSD_H, value_dim=SSD_DV, state=SSD_N, groups=1, conv_taps=TAPS, norm_parts=1, eps=EPS)
        shapes = {"in": ((2 * n + 2 * SSD_N + SSD_H, D), 0.02, 0.0), "conv": ((n + 2 * SSD_N, TAPS), 0.3, 0.0), "conv_bias": ((n + 2 * SSD_N,), 0.02, 0.0),
                  "dt_bias": _step_biases(seed, SSD_H), "A_log": _rates(seed, SSD_H), "D": ((SSD_H,), 0.1, 1.0), "norm": ((n,), 0.1, 1.0),
                  "o": ((D, n), 0.02, 0.0)}
    else:
        hk, hv, R = DELTA_G * DELTA_D, DELTA_H * DELTA_D, DELTA_RANK
        spec = GatedDeltaSpec(width=D, n_heads=DELTA_H, n_qk_heads=DELTA_G, key_dim=DELTA_D, value_dim=DELTA_D, conv_taps=TAPS, eps=EPS, decay_rank=R,
                              gate_rank=R)
        shapes = {"q": ((hk, D), 0.02, 0.0), "k": ((hk, D), 0.02, 0.0), "v": ((hv, D), 0.02, 0.0), "conv_q": ((hk, TAPS), 0.3, 0.0),
                  "conv_k": ((hk, TAPS), 0.3, 0.0), "conv_v": ((hv, TAPS), 0.3, 0.0), "b": ((DELTA_H, D), 0.02, 0.0), "A_log": _rates(seed, DELTA_H),
                  "norm": ((DELTA_D,), 0.1, 1.0), "a1": ((R, D), 0.02, 0.0), "a2": ((DELTA_H * DELTA_D, R), 0.1, 0.0),
                  "dt_bias": _step_biases(seed, DELTA_H * DELTA_D), "g1": ((R, D), 0.02, 0.0), "g2": ((hv, R), 0.1, 0.0), "o": ((D, hv), 0.02, 0.0)}
    return spec, {n: t if isinstance(t, torch.Tensor) else _random(seed, n, *t) for n, t in shapes.items()}


def _prepare_recurrent(case, seed):
    spec, tensors = _recurrent(case, seed)
    part, _ = _part("mixer", spec, seed, tensors)
    lengths = _lengths(case["tokens"], case["seqs"])
    cache = _cache(part, len(lengths), lengths, "bfloat16")
    slots = [cache.acquire() for _ in lengths]
    return {"kind": "mixer", "part": part, "h": _random(seed, "h", (sum(lengths), REC_D)), "step": _step(cache, slots, lengths)}


def _scan64(q, k, v, decay, step=None, beta=None):
    """One sequence from an empty state: S <- diag(decay) S; S <- S + step k v^T, or with `beta` S <- S + beta k (v - S^T k)^T;
    o = S^T q.  q, k [n, H, dk], v [n, H, dv], decay [n, H, dk or 1] -> o [n, H, dv], S [H, dv, dk]."""
    S = torch.zeros(q.shape[1], v.shape[2], q.shape[2], dtype=torch.float64, device=q.device)
    o = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t][:, None, :]
        u = v[t] if beta is None else (v[t] - (S @ k[t][:, :, None])[..., 0]) * beta[t][:, None]
        kk = k[t] if step is None else k[t] * step[t][:, None]
        S = torch.baddbmm(S, u[:, :, None], kk[:, None, :])
        o[t] = (S @ q[t][:, :, None])[..., 0]
    return o, S


def _conv64(x, taps, bias=None):
    """A causal convolution per channel from the sequence's first token on, then silu; and the last inputs."""
    n = taps.shape[1]
    padded = F.pad(x, (0, 0, n - 1, 0))
    y = sum(padded[j:j + x.shape[0]] * taps.double()[:, j] for j in range(n))
    return F.silu(y if bias is None else y + bias.double()), padded[x.shape[0]:]


def _rms64(o, weight):
    """o [n, H, dv]: each head's RMS norm."""
    return o / torch.sqrt(o.square().mean(-1, keepdim=True) + EPS) * weight.double()


def _exact_recurrent(case, seed):
    _, w = _recurrent(case, seed)
    w = {n: t.double() for n, t in w.items()}
    lengths = _lengths(case["tokens"], case["seqs"])
    h_all = _random(seed, "h", (sum(lengths), REC_D)).double()
    outs, states, convs, at = [], [], [], 0
    for n in lengths:
        h = h_all[at:at + n]
        at += n
        if case["kind"] == "lightning":
            q, k, v = (F.silu(h @ w[m].T).view(n, LIGHT_H, 128) for m in "qkv")
            o, S = _scan64(q, k, v, torch.tensor(LIGHT_DECAY, dtype=torch.float32, device=DEVICE).double()[None, :, None].expand(n, -1, -1))
            y = _rms64(o.reshape(n, -1), w["norm"]) * torch.sigmoid(h @ w["g"].T)
        elif case["kind"] == "gla":
            q, k = ((h @ w[m].T).view(n, LIGHT_H, GLA_DK) for m in "qk")
            v = (h @ w["v"].T).view(n, LIGHT_H, GLA_DV)
            z = h @ w["a1"].T @ w["a2"].T + w["a2_bias"]
            o, S = _scan64(q * GLA_DK ** -0.5, k, v, torch.exp(F.logsigmoid(z) / GLA_TAU).view(n, LIGHT_H, GLA_DK))
            y = _rms64(o, w["norm"]).reshape(n, -1) * F.silu(h @ w["g"].T)
        elif case["kind"] == "mamba2":
            m = SSD_H * SSD_DV
            z, xbc, dt = torch.split(h @ w["in"].T, [m, m + 2 * SSD_N, SSD_H], -1)
            xbc, last = _conv64(xbc, w["conv"], w["conv_bias"])
            convs.append(last)
            x, B, C = torch.split(xbc, [m, SSD_N, SSD_N], -1)
            x, dt = x.reshape(n, SSD_H, SSD_DV), F.softplus(dt + w["dt_bias"])
            shared = lambda t: t[:, None, :].expand(n, SSD_H, SSD_N)      # noqa: E731
            o, S = _scan64(shared(C), shared(B), x, torch.exp(-torch.exp(w["A_log"]) * dt)[:, :, None], step=dt)
            y = (o + w["D"][:, None] * x).reshape(n, -1) * F.silu(z)
            y = _rms64(y, w["norm"])
        else:
            pre = [h @ w[m].T for m in "qkv"]
            post = [_conv64(x, w["conv_" + m]) for x, m in zip(pre, "qkv")]
            convs.append(torch.cat([last for _, last in post], -1))
            q, k = (y.view(n, DELTA_G, DELTA_D) for y, _ in post[:2])
            q, k = (x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6) for x in (q, k))
            q, k = (x.repeat_interleave(DELTA_H // DELTA_G, 1) for x in (q * DELTA_D ** -0.5, k))
            a = F.softplus(h @ w["a1"].T @ w["a2"].T + w["dt_bias"]).view(n, DELTA_H, DELTA_D)
            o, S = _scan64(q, k, post[2][0].view(n, DELTA_H, DELTA_D), torch.exp(-torch.exp(w["A_log"])[:, None] * a), beta=torch.sigmoid(h @ w["b"].T))
            y = _rms64(o, w["norm"]).reshape(n, -1) * torch.sigmoid(h @ w["g1"].T @ w["g2"].T)
        outs.append(y @ w["o"].T)
        states.append(S)
    more = [torch.stack(convs)] if convs else []
    return [torch.cat(outs), *more, torch.stack(states)]


# ---------------------------------------------------------------------------------------------------- the contract

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("request", "decode"):
        return _prepare_model(case, seed)
    if kind == "layer":
        return _prepare_layer(case, seed)
    if kind == "attention":
        return _prepare_attention(case, seed)
    if kind == "experts":
        return _prepare_experts(case, seed)
    return _prepare_recurrent(case, seed)


def run(state):
    kind = state["kind"]
    if kind == "request":
        return _run_request(state)
    if kind == "decode":
        return _run_decode(state)
    if kind == "layer":
        return _run_layer(state)
    if kind == "experts":
        return state["part"].forward(state["h"], state["step"])
    return _run_mixer(state)


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind in ("request", "decode"):
        return _exact_model(case, seed)
    if kind == "layer":
        return _exact_layer(case, seed)
    if kind == "attention":
        return _exact_attention(case, seed)
    if kind == "experts":
        return _exact_experts(case, seed)
    return _exact_recurrent(case, seed)


def _attention_work(queries, keys, pairs, H, G, dh, size):
    """Softmax attention: keys and values of `keys` tokens read once, `pairs` (query, key) pairs."""
    return 2 * keys * G * dh * size + 2 * queries * H * dh * size, 4.0 * pairs * H * dh


def work(case):
    kind = case["kind"]
    if kind in ("request", "decode", "layer"):
        D, L, H, dh, inner, vocab = _gptj(case)
        size = BYTES[case.get("dtype", "bfloat16")]
        weights = 4 * D * D + 2 * D * inner
        steps = []                                      # (new tokens, keys read, pairs, rows of logits)
        if kind == "layer":
            lengths = _lengths(case["tokens"], case["seqs"])
            steps.append((sum(lengths), sum(lengths), sum(n * (n + 1) / 2 for n in lengths), 0))
        elif kind == "decode":
            lengths = _decode_lengths(case)
            held = sum(lengths) + len(lengths)
            steps.append((len(lengths), held, held, len(lengths)))
        else:
            lengths = _lengths(case["tokens"], case["seqs"])
            steps.append((sum(lengths), sum(lengths), sum(n * (n + 1) / 2 for n in lengths), len(lengths)))
            for j in range(case["new"]):
                held = sum(lengths) + (j + 1) * len(lengths)
                steps.append((len(lengths), held, held, len(lengths)))
        total = flops = 0.0
        for new, keys, pairs, rows in steps:
            b, f = _attention_work(0, keys, pairs, H, H, dh, size)
            total += L * (weights * size + b) + 2 * new * D * size + (vocab * D * size if rows else 0) + rows * vocab * 4
            flops += L * (2.0 * new * weights + f) + 2.0 * rows * vocab * D
        return {"bytes": total, "flops": flops}
    if kind == "attention":
        lengths = _attention_lengths(case)
        hq, hkv = ATT_H * ATT_DH, ATT_G * ATT_DH
        weights = ATT_D * (3 * hq + 2 * hkv)
        if case["step"] == "decode":
            new, keys, pairs = len(lengths), sum(lengths) + len(lengths), sum(lengths) + len(lengths)
        else:
            new, keys, pairs = sum(lengths), sum(lengths), sum(n * (n + 1) / 2 for n in lengths)
        b, f = _attention_work(0, keys, pairs, ATT_H, ATT_G, ATT_DH, 2)
        return {"bytes": weights * 2 + b + 2 * new * ATT_D * 2, "flops": 2.0 * new * weights + f}
    if kind == "experts":
        D, n = case["width"], case["tokens"]
        inner = D // 4
        read = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** n)             # experts that some token chose
        return {"bytes": read * 3 * D * inner * 2 + EXPERTS * D * 2 + n * D * (2 + 4), "flops": 2.0 * n * D * EXPERTS + 6.0 * n * TOP * D * inner}
    n, seqs = max(case["tokens"], case["seqs"]), case["seqs"]
    D = REC_D
    if kind == "lightning":
        H, dk, dv, weights = LIGHT_H, 128, 128, 5 * D * LIGHT_H * 128
    elif kind == "gla":
        H, dk, dv = LIGHT_H, GLA_DK, GLA_DV
        weights = D * H * (2 * dk + 3 * dv) + GLA_RANK * (D + H * dk)
    elif kind == "mamba2":
        H, dk, dv = SSD_H, SSD_N, SSD_DV
        weights = D * (3 * H * dv + 2 * dk + H)
    else:
        H, dk, dv = DELTA_H, DELTA_D, DELTA_D
        weights = D * (2 * DELTA_G * dk + 2 * H * dv + H) + DELTA_RANK * (2 * D + H * dk + H * dv)
    per_element = 6.0 if kind == "delta" else 4.0       # the update and the reading of the state (the delta rule reads it twice)
    return {"bytes": weights * 2 + 2 * seqs * H * dk * dv * 4 + 2 * n * D * 2, "flops": 2.0 * n * weights + per_element * n * H * dk * dv}


# Four times the distance from `exact` that was measured on a B200 (2-norm): whole models 0.0066 (eight layers) and 0.0092 (28), a
# bfloat16 layer 0.0028, bfloat16 attention 0.0038, experts 0.0031, mixers with a state 0.0042, a float32 layer 3.3e-7.
TOLERANCE = {"request": 0.026, "decode": 0.037, "layer": 0.012, "attention": 0.015, "experts": 0.0125}


def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 1.5e-6}
    return {"rel": TOLERANCE.get(case["kind"], 0.017)}
