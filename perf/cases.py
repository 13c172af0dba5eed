"""The work this framework is used for, as cases that can be timed and compared with a plain computation in 64 bits.

Two kinds of calls: whole steps of an engine (``ModelRunner.step``, as the Python entry point and the benchmark call it:
token ids in, logits out) and single layers (an attention layer over its pages, a feed-forward, the output head with the
choice of the tokens, a routed feed-forward, a layer with a recurrent memory), each through the part's own ``forward``.
Sizes are those of the benchmark: the Qwen2.5 1.5B, 3B and 7B shapes and the sizes its other designs are measured at.  Weights
are random, N(0, 0.02), keys and values of earlier tokens random of the size that the projections give.  A whole step is that
of a model cut to a few layers of full size (as the benchmark's ``--layers`` does): with random weights every layer adds to
what a rounding in 16 bits does to the logits, and after all 28 they are 2 to 6 % off the 64-bit ones, too far to tell a right
answer from a wrong one.

Every input comes from the functions named ``_..._inputs`` (seed in, plain tensors out); ``prepare`` hands them to the
framework, ``exact`` computes with them in float64 and uses none of the framework's code.
"""
import math

import torch

DEV = "cuda:0"
PAGE = 16
EPS = 1e-6
THETA = 1000000.0
GENERATE = 128          # tokens a decoding request grows by before the batch is started over
SHAPES = {
    "1.5b": dict(width=1536, heads=12, kv_heads=2, head=128, inner=8960, vocab=151936, layers=28, tied=True),
    "3b": dict(width=2048, heads=16, kv_heads=2, head=128, inner=11008, vocab=151936, layers=36, tied=True),
    "7b": dict(width=3584, heads=28, kv_heads=4, head=128, inner=18944, vocab=152064, layers=28, tied=False),
}
# the sizes of the other designs: routed experts (``top`` of them as wide as a dense feed-forward), a gated delta rule
DESIGNS = {
    "1536": dict(width=1536, heads=12, kv_heads=6, head=128, inner=2240, experts=16, top=4, taps=4),
    "2048": dict(width=2048, heads=16, kv_heads=8, head=128, inner=2752, experts=32, top=4, taps=4),
}


# ---------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one user, one token at a time: the smallest call, where launches and latency count
        dict(name="decode_b1", kind="decode", shape="1.5b", layers=12, batch=1, context=512, ragged=False),
        # the benchmark's default: eight users with long contexts
        dict(name="decode_b8", kind="decode", shape="1.5b", layers=12, batch=8, context=4096, ragged=False),
        # a full server: 64 requests of all ages
        dict(name="decode_b64", kind="decode", shape="1.5b", layers=8, batch=64, context=1536, ragged=True),
        # one 2,048-token prompt (or one full portion of a longer one)
        dict(name="prompt_2048", kind="prompt", shape="1.5b", layers=2, tokens=2048),
        # a layer of the large shape at the longest contexts the benchmark serves: all decode
        dict(name="attention_7b_b64", kind="attention", shape="7b", dtype="bfloat16", portions=0, portion=0, singles=64, context=8192),
        # the same layer in a mixed step: portions of two prompts of odd sizes, one in the middle of its prompt, beside
        # requests that decode
        dict(name="attention_7b_mixed", kind="attention", shape="7b", dtype="bfloat16", portions=2, portion=1013, singles=37, context=3001),
        # the true 32-bit path, with which results are checked: a short prompt beside decoding requests
        dict(name="attention_fp32", kind="attention", shape="1.5b", dtype="float32", portions=1, portion=333, singles=7, context=777),
        # feed-forward of the large shape in a mixed step
        dict(name="mlp_7b_2111", kind="mlp", shape="7b", tokens=2111),
        # feed-forward of the middle shape at a medium batch
        dict(name="mlp_3b_48", kind="mlp", shape="3b", tokens=48),
        # the head for a full batch and the choice of tokens: greedy rows beside rows with a temperature and top-p
        dict(name="head_sample_64", kind="head", shape="7b", rows=64),
        # routed experts over a portion of a prompt
        dict(name="experts_2048", kind="experts", design="1536", tokens=2048),
        # the layer with a matrix memory per request: portions of three prompts of different lengths
        dict(name="delta_2048", kind="delta", design="1536", tokens=2048, portions=3),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "attention", "attention", "mlp", "mlp", "head", "experts", "delta"])
    if kind == "decode":
        batch = _log_int(rng, 1, 64)
        return dict(kind=kind, shape="1.5b", layers=rng.choice([4, 8, 12] if batch <= 16 else [4, 6, 8]), batch=batch,
                    context=_log_int(rng, 32, min(4096, 98304 // batch)), ragged=rng.random() < 0.7)
    if kind == "prompt":
        return dict(kind=kind, shape="1.5b", layers=rng.randint(1, 2), tokens=_log_int(rng, 17, 2048))
    if kind == "attention":
        if rng.random() < 0.2:
            return dict(kind=kind, shape="1.5b", dtype="float32", portions=rng.randint(0, 2), portion=_log_int(rng, 2, 150),
                        singles=rng.randint(1, 8), context=_log_int(rng, 16, 777))
        portions = rng.randint(0, 3)
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), dtype="bfloat16", portions=portions,
                    portion=_log_int(rng, 2, 2048 // max(1, portions)) if portions else 0, singles=_log_int(rng, 1, 64),
                    context=_log_int(rng, 16, 4096 if portions else 8192))
    if kind == "mlp":
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), tokens=_log_int(rng, 1, 2111))
    if kind == "head":
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), rows=_log_int(rng, 1, 64))
    if kind == "experts":
        return dict(kind=kind, design=rng.choice(sorted(DESIGNS)), tokens=_log_int(rng, 1, 2048))
    tokens = _log_int(rng, 4, 2048)
    return dict(kind=kind, design=rng.choice(sorted(DESIGNS)), tokens=tokens, portions=rng.randint(1, 4))


# ------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed((seed * 1000003 + salt * 7919 + 17) % (1 << 62))


def _randn(g, *shape, scale=1.0, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).mul_(scale).to(dtype)


def _contexts(case, n):
    """Tokens that each of n requests already holds: all the same, or of all ages up to ``context``; the same for every
    seed, as are all sizes."""
    c = case["context"]
    if not case.get("ragged", True):
        return [c] * n
    g = torch.Generator().manual_seed(c + n)
    return [max(1, c - int(x * c * 0.875)) for x in torch.rand(n, generator=g).tolist()]


def _ids(n, vocab, seed):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed + 9)).tolist()


def _attention_weights(s, g, dtype=torch.bfloat16):
    qkv = (s["heads"] + 2 * s["kv_heads"]) * s["head"]
    return dict(qkv_weight=_randn(g, qkv, s["width"], scale=0.02, dtype=dtype), qkv_bias=_randn(g, qkv, scale=0.02, dtype=torch.float32),
                o_weight=_randn(g, s["width"], s["heads"] * s["head"], scale=0.02, dtype=dtype))


def _mlp_weights(s, g):
    return dict(gate_up_weight=_randn(g, 2 * s["inner"], s["width"], scale=0.02), down_weight=_randn(g, s["width"], s["inner"], scale=0.02))


def _norm_weight(s, g):
    return _randn(g, s["width"], scale=0.02, dtype=torch.float32) + 1.0


def _layer_weights(s, seed, layer):
    g = _gen(seed, 100 + layer)
    return dict(mixer=_attention_weights(s, g), feed_forward=_mlp_weights(s, g), norm1=dict(weight=_norm_weight(s, g)),
                norm2=dict(weight=_norm_weight(s, g)))


def _end_weights(s, seed):
    g = _gen(seed, 1)
    return _randn(g, s["vocab"], s["width"], scale=0.02), _norm_weight(s, g)


def _kv(s, seed, layer, rows, dtype=torch.bfloat16):
    """Keys and values of ``rows`` earlier tokens of a layer, request after request: [2, rows, kv heads, head]."""
    return _randn(_gen(seed, 10000 + layer), 2, rows, s["kv_heads"], s["head"], scale=0.8, dtype=dtype)


def _places(starts, lens):
    """Page and offset of the first ``starts[i]`` tokens of each request when request i has ceil(lens[i] / PAGE) pages
    in a row, one request's after the other's."""
    page, off, base = [], [], 0
    for st, n in zip(starts, lens):
        pos = torch.arange(st)
        page.append(base + pos // PAGE)
        off.append(pos % PAGE)
        base += -(-n // PAGE)
    return torch.cat(page).to(DEV), torch.cat(off).to(DEV), base


def _attention_inputs(case, seed):
    """(weights, hidden rows, tokens per segment, starts, keys and values of the starts)"""
    s = SHAPES[case["shape"]]
    dtype = getattr(torch, case["dtype"])
    g = _gen(seed, 2)
    w = _attention_weights(s, g, dtype)
    lens = [max(2, case["portion"] - 13 * i) for i in range(case["portions"])] + [1] * case["singles"]
    starts = _contexts(case, len(lens))
    if case["portions"]:
        starts[0] = 0               # the first portion starts its prompt
    h = _randn(g, sum(lens), s["width"], dtype=dtype)
    return s, w, h, lens, starts, _kv(s, seed, 0, sum(starts), dtype)


def _head_inputs(case, seed):
    s, R = SHAPES[case["shape"]], case["rows"]
    g = _gen(seed, 3)
    w = _randn(g, s["vocab"], s["width"], scale=0.02)
    y = _randn(g, R, s["width"], scale=2.5)
    cpu = torch.Generator().manual_seed(seed + 3)
    temperature = [(0.0, 0.7, 1.0, 0.8)[i % 4] for i in range(R)]
    top_p = [(1.0, 0.9, 1.0, 0.95)[i % 4] for i in range(R)]
    return s, w, y, temperature, top_p, torch.rand(R, generator=cpu).tolist()


def _experts_inputs(case, seed):
    s, T = DESIGNS[case["design"]], case["tokens"]
    g = _gen(seed, 4)
    E, I, D = s["experts"], s["inner"], s["width"]
    w = dict(router_weight=_randn(g, E, D, scale=0.02, dtype=torch.float32), router_bias=_randn(g, E, scale=0.02, dtype=torch.float32),
             gate_up_weight=_randn(g, E * 2 * I, D, scale=0.02), down_weight=_randn(g, E * D, I, scale=0.02))
    return s, w, _randn(g, T, D)


def _delta_inputs(case, seed):
    s, T = DESIGNS[case["design"]], case["tokens"]
    g = _gen(seed, 5)
    H, G, d, D = s["heads"], s["kv_heads"], s["head"], s["width"]
    C = 2 * G * d + H * d
    w = dict(proj_weight=_randn(g, C + H * d + 2 * H, D, scale=0.02),
             conv_weight=_randn(g, C, s["taps"], scale=0.02, dtype=torch.float32) + 0.3, dt_bias=_randn(g, H, scale=0.02, dtype=torch.float32),
             a_log=torch.log(torch.rand(H, generator=g, device=DEV) * 0.98 + 0.02), out_norm=_randn(g, d, scale=0.02, dtype=torch.float32) + 1.0,
             o_weight=_randn(g, D, H * d, scale=0.02))
    n = min(case["portions"], T)
    lens = [T * (i + 1) // (n * (n + 1) // 2) or 1 for i in range(n - 1)]       # a short one, a longer one, ...
    lens.append(T - sum(lens))
    memory = _randn(g, n, H, d, d, scale=0.05, dtype=torch.float32)
    taps = _randn(g, n, s["taps"] - 1, C, scale=0.8, dtype=torch.float32)
    return s, w, _randn(g, T, D), lens, memory, taps


# ------------------------------------------------------------------------------------------------------------ prepare
def _assign(part, tensors):
    for attr, t in tensors.items():
        part.assign(attr, t)


def _engine(case, seed, max_seqs, max_len, pages):
    """A Qwen2 decoder of the case's size with its cache and step function."""
    import pico_vllm_b200  # noqa: F401
    from pico_vllm_b200.config import EngineConfig
    from pico_vllm_b200.engine import ModelRunner, make_cache
    from pico_vllm_b200.registry import build_model, config_from_dict
    s = SHAPES[case["shape"]]
    model = build_model(config_from_dict(dict(
        architectures=["Qwen2ForCausalLM"], vocab_size=s["vocab"], hidden_size=s["width"], num_hidden_layers=case["layers"],
        num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"], intermediate_size=s["inner"], rope_theta=THETA,
        rms_norm_eps=EPS, tie_word_embeddings=s["tied"], use_sliding_window=False, max_position_embeddings=32768, hidden_act="silu")))
    for i, block in enumerate(model.blocks):
        w = _layer_weights(s, seed, i)
        for name, part in block.parts().items():
            _assign(part, w[name])
    table, norm = _end_weights(s, seed)
    model.embed.assign("weight", table)
    model.final_norm.assign("weight", norm)
    model.materialize(DEV, torch.bfloat16)
    cfg = EngineConfig(dtype="bfloat16", page_size=PAGE, num_pages=pages, max_num_seqs=max_seqs, max_num_batched_tokens=2048,
                       max_model_len=max_len, device=DEV)
    cache = make_cache(model, cfg)
    return s, cache, ModelRunner(model, cache, cfg)


def _start_over(state):
    """The batch's requests end and others with as long contexts take their places (their keys and values lie in the
    same pages)."""
    cache = state["cache"]
    for slot in reversed(state["slots"]):
        cache.release(slot)
    state["slots"] = []
    for n in state["starts"]:
        slot = cache.acquire("request")
        cache.append(slot, n)
        cache.commit(slot)
        state["slots"].append(slot)
    state["at"] = 0


def _fill_pages(k, v, kv, starts, lens):
    page, off, n = _places(starts, lens)
    k[page, :, off] = kv[0]
    v[page, :, off] = kv[1]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "decode":
        B = case["batch"]
        starts = _contexts(case, B)
        pages = sum(-(-n // PAGE) for n in starts) + B * (GENERATE // PAGE + 1)
        s, cache, runner = _engine(case, seed, B, case["context"] + GENERATE + PAGE, pages)
        state = dict(kind=kind, cache=cache, runner=runner, slots=[], starts=starts)
        _start_over(state)
        for i in range(case["layers"]):
            g, at = cache.entry_group[i]
            t = cache.groups[g].tensors
            _fill_pages(t["k"][at], t["v"][at], _kv(s, seed, i, sum(starts)), starts, starts)
        ids = _ids(GENERATE * B, s["vocab"], seed)
        state["ids"] = [ids[i * B:(i + 1) * B] for i in range(GENERATE)]
        return state
    if kind == "prompt":
        T = case["tokens"]
        s, cache, runner = _engine(case, seed, 1, 2048 + PAGE, 2048 // PAGE + 1)
        return dict(kind=kind, cache=cache, runner=runner, ids=_ids(T, s["vocab"], seed), last=T - 1)
    if kind == "attention":
        return _prepare_attention(case, seed)
    if kind == "mlp":
        from pico_vllm_b200.parts import GatedMLP
        s = SHAPES[case["shape"]]
        g = _gen(seed, 6)
        part = GatedMLP(s["width"], s["inner"])
        _assign(part, _mlp_weights(s, g))
        part.materialize(DEV, torch.bfloat16)
        return dict(kind=kind, part=part, h=_randn(g, case["tokens"], s["width"]))
    if kind == "head":
        from pico_vllm_b200.parts import OutputHead
        from pico_vllm_b200.sampling import Sampler
        s, w, y, temperature, top_p, uniform = _head_inputs(case, seed)
        part = OutputHead(s["vocab"], s["width"])
        _assign(part, dict(weight=w))
        return dict(kind=kind, part=part, y=y, sampler=Sampler(DEV), args=(temperature, top_p, uniform),
                    tokens=torch.zeros(case["rows"], dtype=torch.int32, device=DEV))
    if kind == "experts":
        from pico_vllm_b200.parts import RoutedExperts
        s, w, h = _experts_inputs(case, seed)
        part = RoutedExperts(s["width"], s["inner"], s["experts"], s["top"])
        _assign(part, w)
        part.materialize(DEV, torch.bfloat16)
        return dict(kind=kind, part=part, h=h)
    return _prepare_delta(case, seed)


def _int32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _segments(lens, starts):
    """positions, segment of each token and first token of each segment"""
    pos = torch.cat([torch.arange(st, st + n) for n, st in zip(lens, starts)]).to(torch.int32).to(DEV)
    seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32).to(DEV)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return pos, seg, cu


def _prepare_attention(case, seed):
    from pico_vllm_b200.cache import CacheManager
    from pico_vllm_b200.config import EngineConfig
    from pico_vllm_b200.engine import Batch, GroupBatch
    from pico_vllm_b200.parts import GQAAttention, Rotary
    from pico_vllm_b200.parts.base import StepShape
    s, w, h, lens, starts, kv = _attention_inputs(case, seed)
    dtype = getattr(torch, case["dtype"])
    part = GQAAttention(s["width"], s["heads"], s["kv_heads"], s["head"], position=Rotary(s["head"], THETA))
    _assign(part, w)
    part.materialize(DEV, dtype)
    total = [n + st for n, st in zip(lens, starts)]
    pages = sum(-(-n // PAGE) for n in total)
    S, T = len(lens), sum(lens)
    cache = CacheManager([part.cache_spec()], PAGE, pages, S, max(total), dtype, DEV)
    slots = [cache.acquire("request") for _ in lens]
    for slot, n in zip(slots, total):
        cache.append(slot, n)
        cache.commit(slot)
    t = cache.groups[0].tensors
    _fill_pages(t["k"][0], t["v"][0], kv, starts, total)
    pos, seg, cu = _segments(lens, starts)
    rows = torch.from_numpy(cache.groups[0].tables[slots].copy()).clamp_(min=0).to(torch.int32).to(DEV)
    at = torch.cat([torch.from_numpy(cache.slot_mapping(0, slot, st, n)) for slot, st, n in zip(slots, starts, lens)]).to(DEV)
    shape = StepShape(num_tokens=T, num_segments=S, q_lens=lens, starts=starts, max_kv=max(total), decode_only=max(lens) == 1,
                      num_sms=torch.cuda.get_device_properties(DEV).multi_processor_count, engine=EngineConfig(dtype=case["dtype"]))
    plan = part.plan(shape)
    portions = [i for i, n in enumerate(lens) if n > 1]
    singles = [cu[i] for i, n in enumerate(lens) if n == 1]
    batch = Batch(num_tokens=T, num_segments=S, token_ids=_int32([0] * T), positions=pos, tok_seg=seg, seg_slots=_int32(slots),
                  cu_q=_int32(cu), logit_rows=_int32([]), num_logit_rows=0, groups={0: GroupBatch(at, rows)}, q_lens=lens,
                  kv_lens=total, plans={part.plan_key(): plan},
                  scratch=torch.empty(plan.scratch_floats, dtype=torch.float32, device=DEV) if plan.scratch_floats else None,
                  decode_only=max(lens) == 1, prefill_segs=_int32(portions) if len(portions) < S else None,
                  num_prefill_segs=len(portions), max_prefill_q=max([lens[i] for i in portions], default=0),
                  decode_tokens=_int32(singles) if len(singles) < T else None, num_decode_tokens=len(singles))
    view = cache.views()[0]
    return dict(kind="attention", part=part, h=h, batch=batch, view=view, cache=cache)


def _prepare_delta(case, seed):
    from pico_vllm_b200.engine import Batch
    from pico_vllm_b200.parts import GatedDeltaRule
    from pico_vllm_b200.parts.base import CacheView
    s, w, h, lens, memory, taps = _delta_inputs(case, seed)
    part = GatedDeltaRule(s["width"], s["heads"], s["kv_heads"], s["head"], s["head"], s["taps"], 1e-5, head_decay=True,
                          full_gate=True, gate_act="silu")
    _assign(part, w)
    part.materialize(DEV, torch.bfloat16)
    pos, seg, cu = _segments(lens, [0] * len(lens))
    T, S = sum(lens), len(lens)
    batch = Batch(num_tokens=T, num_segments=S, token_ids=_int32([0] * T), positions=pos, tok_seg=seg, seg_slots=_int32(list(range(S))),
                  cu_q=_int32(cu), logit_rows=_int32([]), num_logit_rows=0, groups={}, q_lens=lens, kv_lens=lens,
                  num_prefill_segs=S, max_prefill_q=max(lens))
    return dict(kind="delta", part=part, h=h, batch=batch, views=(CacheView(state=memory), CacheView(state=taps)))


# ---------------------------------------------------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "decode":
        from pico_vllm_b200.engine import StepItem
        if state["at"] == GENERATE:
            _start_over(state)
        ids = state["ids"][state["at"]]
        state["at"] += 1
        return state["runner"].step([StepItem(slot, [t], (0,)) for slot, t in zip(state["slots"], ids)])
    if kind == "prompt":
        from pico_vllm_b200.engine import StepItem
        slot = state["cache"].acquire("prompt")
        logits = state["runner"].step([StepItem(slot, state["ids"], (state["last"],))])
        state["cache"].release(slot)
        return logits
    if kind == "attention":
        out = state["part"].forward(state["h"], state["batch"], state["view"])
        return dict(out=out, k=state["view"].k, v=state["view"].v)
    if kind == "mlp":
        return state["part"].forward(state["h"], None)
    if kind == "head":
        logits = state["part"].forward(state["y"])
        state["sampler"].sample_async(logits, *state["args"], out=state["tokens"])
        return dict(logits=logits, tokens=state["tokens"])
    if kind == "experts":
        return state["part"].forward(state["h"], None)
    out = state["part"].forward(state["h"], state["batch"], state["views"])
    return dict(out=out, memory=state["views"][0].state, taps=state["views"][1].state)


# --------------------------------------------------------------------------------------------------------------- work
def _attention_work(s, lens, starts, item=2):
    T = sum(lens)
    qkv, q = (s["heads"] + 2 * s["kv_heads"]) * s["head"], s["heads"] * s["head"]
    weights = (qkv + q) * s["width"]
    seen = sum(n * st + n * (n + 1) / 2 for n, st in zip(lens, starts))
    kv = 2 * s["kv_heads"] * s["head"] * (sum(starts) + T)        # earlier rows read, new rows written
    return item * (weights + kv + 2 * T * s["width"]), 2 * T * weights + 4 * q * seen


def _mlp_work(s, T):
    n = 3 * s["width"] * s["inner"]
    return 2 * (n + 2 * T * s["width"]), 2 * T * n


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        s = SHAPES[case["shape"]]
        if kind == "decode":
            # (contexts of all ages: between an eighth of the longest and the longest; the middle of it)
            lens, starts = [1] * case["batch"], [int(case["context"] * (0.5625 if case["ragged"] else 1))] * case["batch"]
            rows = case["batch"]
        else:
            lens, starts, rows = [case["tokens"]], [0], 1
        T = sum(lens)
        ab, af = _attention_work(s, lens, starts)
        mb, mf = _mlp_work(s, T)
        act = 4 * T * s["width"] * 2            # rows between the layers of a step need not leave the chip
        head = s["vocab"] * s["width"]
        return dict(bytes=case["layers"] * (ab + mb - act) + 2 * head + 4 * rows * s["vocab"], flops=case["layers"] * (af + mf) + 2 * rows * head)
    if kind == "attention":
        s = SHAPES[case["shape"]]
        lens = [max(2, case["portion"] - 13 * i) for i in range(case["portions"])] + [1] * case["singles"]
        starts = [int(case["context"] * 0.5625)] * len(lens)
        if case["portions"]:
            starts[0] = 0
        b, f = _attention_work(s, lens, starts, 4 if case["dtype"] == "float32" else 2)
        return dict(bytes=b, flops=f)
    if kind == "mlp":
        b, f = _mlp_work(SHAPES[case["shape"]], case["tokens"])
        return dict(bytes=b, flops=f)
    if kind == "head":
        s, R = SHAPES[case["shape"]], case["rows"]
        n = s["vocab"] * s["width"]
        return dict(bytes=2 * n + 2 * R * s["width"] + 4 * R * s["vocab"], flops=2 * R * n)
    s, T = DESIGNS[case["design"]], case["tokens"]
    if kind == "experts":
        one = 3 * s["width"] * s["inner"]
        touched = s["experts"] * (1 - (1 - s["top"] / s["experts"]) ** T)
        return dict(bytes=2 * one * touched + 4 * s["experts"] * s["width"] + 4 * T * s["width"],
                    flops=2 * T * (s["top"] * one + s["experts"] * s["width"]))
    H, d, D = s["heads"], s["head"], s["width"]
    C = 2 * s["kv_heads"] * d + H * d
    weights = (C + H * d + 2 * H) * D + H * d * D
    n = min(case["portions"], T)
    state = n * (H * d * d + (s["taps"] - 1) * C) * 4
    return dict(bytes=2 * weights + 4 * T * D + 2 * state, flops=2 * T * weights + T * (2 * C * s["taps"] + H * 8 * d * d))


def tolerance(case):
    """Measured: the present kernels are 0.011 to 0.015 off the 64-bit logits in the decode steps and about 0.02 in the prompt
    steps (another correct implementation rounds elsewhere, and the two are as far from each other), 0.004 to 0.0063 in
    the layers in 16 bits, 1.2e-6 in 32 bits, 3.8e-6 in the logits of the head alone (the library's product)."""
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        return {"rel": 0.03}
    if kind == "attention":
        return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 0.02}
    if kind == "head":
        return {"rel": 2e-5, "differ": 0.0}
    return {"rel": 0.015}


# -------------------------------------------------------------------------------------------------------------- exact
F64 = torch.float64


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w.to(F64)


def _turn(x, pos):
    """x [T, heads, head] rotated by its positions: dimension i with i + head / 2."""
    half = x.shape[-1] // 2
    f = THETA ** (-torch.arange(half, dtype=F64, device=x.device) / half)
    a = (pos.to(F64)[:, None] * f)[:, None, :]
    c, s = torch.cos(a), torch.sin(a)
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(s, q, k, v, start):
    """Causal attention of the last len(q) of len(k) tokens."""
    n, H, G = q.shape[0], s["heads"], s["kv_heads"]
    out = torch.empty_like(q)
    mask = torch.arange(k.shape[0], device=q.device)[None, :] > (start + torch.arange(n, device=q.device))[:, None]
    for g in range(G):
        r = H // G
        p = torch.einsum("nhd,kd->hnk", q[:, g * r:(g + 1) * r], k[:, g]) * s["head"] ** -0.5
        p = torch.softmax(p.masked_fill_(mask, float("-inf")), -1)
        out[:, g * r:(g + 1) * r] = torch.einsum("hnk,kd->nhd", p, v[:, g])
    return out


def _exact_attention(s, w, h, lens, starts, kv, pos):
    """(output rows, new keys, new values); ``kv``: keys and values of the starts."""
    H, G, d = s["heads"], s["kv_heads"], s["head"]
    y = h @ w["qkv_weight"].to(F64).t() + w["qkv_bias"].to(F64)
    q = _turn(y[:, :H * d].view(-1, H, d), pos)
    k = _turn(y[:, H * d:(H + G) * d].view(-1, G, d), pos)
    v = y[:, (H + G) * d:].reshape(-1, G, d)
    out, at, past = torch.empty_like(q), 0, 0
    for n, st in zip(lens, starts):
        ks = torch.cat([kv[0, past:past + st].to(F64), k[at:at + n]])
        vs = torch.cat([kv[1, past:past + st].to(F64), v[at:at + n]])
        out[at:at + n] = _attend(s, q[at:at + n], ks, vs, st)
        at, past = at + n, past + st
    return out.reshape(-1, H * d) @ w["o_weight"].to(F64).t(), k, v


def _exact_mlp(w, h):
    g, u = (h @ w["gate_up_weight"].to(F64).t()).chunk(2, -1)
    return (g * torch.sigmoid(g) * u) @ w["down_weight"].to(F64).t()


def _exact_step(case, seed, ids, lens, starts, rows):
    s = SHAPES[case["shape"]]
    table, norm = _end_weights(s, seed)
    x = table[torch.tensor(ids, device=DEV)].to(F64)
    pos = torch.cat([torch.arange(st, st + n) for n, st in zip(lens, starts)]).to(DEV)
    for i in range(case["layers"]):
        w = _layer_weights(s, seed, i)
        kv = _kv(s, seed, i, sum(starts)) if sum(starts) else torch.empty(2, 0, s["kv_heads"], s["head"], device=DEV)
        x = x + _exact_attention(s, w["mixer"], _rms(x, w["norm1"]["weight"]), lens, starts, kv, pos)[0]
        x = x + _exact_mlp(w["feed_forward"], _rms(x, w["norm2"]["weight"]))
    return _rms(x[rows], norm) @ table.to(F64).t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        B = case["batch"]
        ids = _ids(GENERATE * B, SHAPES[case["shape"]]["vocab"], seed)[:B]
        return _exact_step(case, seed, ids, [1] * B, _contexts(case, B), list(range(B)))
    if kind == "prompt":
        T = case["tokens"]
        return _exact_step(case, seed, _ids(T, SHAPES[case["shape"]]["vocab"], seed), [T], [0], [T - 1])
    if kind == "attention":
        s, w, h, lens, starts, kv = _attention_inputs(case, seed)
        pos = torch.cat([torch.arange(st, st + n) for n, st in zip(lens, starts)]).to(DEV)
        out, k, v = _exact_attention(s, w, h.to(F64), lens, starts, kv, pos)
        total = [n + st for n, st in zip(lens, starts)]
        page, off, n_pages = _places(total, total)
        pages = []
        for new, old in ((k, kv[0]), (v, kv[1])):
            rows, at, past = [], 0, 0
            for n, st in zip(lens, starts):
                rows += [old[past:past + st].to(F64), new[at:at + n]]
                at, past = at + n, past + st
            t = torch.zeros(n_pages, s["kv_heads"], PAGE, s["head"], dtype=F64, device=DEV)
            t[page, :, off] = torch.cat(rows)
            pages.append(t)
        return dict(out=out, k=pages[0], v=pages[1])
    if kind == "mlp":
        s = SHAPES[case["shape"]]
        g = _gen(seed, 6)
        w = _mlp_weights(s, g)
        return _exact_mlp(w, _randn(g, case["tokens"], s["width"]).to(F64))
    if kind == "head":
        s, w, y, _, _, _ = _head_inputs(case, seed)
        return dict(logits=y.to(F64) @ w.to(F64).t(), tokens=None)
    if kind == "experts":
        s, w, h = _experts_inputs(case, seed)
        h, E, I, D = h.to(F64), s["experts"], s["inner"], s["width"]
        z = h @ w["router_weight"].to(F64).t() + w["router_bias"].to(F64)
        top, chosen = torch.topk(z, s["top"], -1)
        share = torch.softmax(top, -1)
        up, down = w["gate_up_weight"].view(E, 2 * I, D), w["down_weight"].view(E, D, I)
        out = torch.zeros_like(h)
        for e in range(E):
            t, j = torch.nonzero(chosen == e, as_tuple=True)
            out[t] += share[t, j][:, None] * _exact_mlp(dict(gate_up_weight=up[e], down_weight=down[e]), h[t])
        return out
    return _exact_delta(case, seed)


def _exact_delta(case, seed):
    s, w, h, lens, memory, taps = _delta_inputs(case, seed)
    H, G, d, h = s["heads"], s["kv_heads"], s["head"], h.to(F64)
    C, n_taps = 2 * G * d + H * d, s["taps"]
    z = h @ w["proj_weight"].to(F64).t()
    gate, beta = z[:, C:C + H * d], torch.sigmoid(z[:, C + H * d:C + H * d + H])
    dt = torch.nn.functional.softplus(z[:, C + H * d + H:] + w["dt_bias"].to(F64))
    keep = torch.exp(-torch.exp(w["a_log"].to(F64)) * dt)
    memory, outs, new_taps, at = memory.to(F64), [], [], 0
    for i, n in enumerate(lens):
        rows = torch.cat([taps[i].to(F64), z[at:at + n, :C]])
        new_taps.append(rows[-(n_taps - 1):])
        c = sum(rows[j:j + n] * w["conv_weight"].to(F64)[:, j] for j in range(n_taps))
        c = c * torch.sigmoid(c)
        q, k, v = c[:, :G * d].view(n, G, d), c[:, G * d:2 * G * d].view(n, G, d), c[:, 2 * G * d:].view(n, H, d)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
        S, o = memory[i], torch.empty(n, H, d, dtype=F64, device=h.device)        # S [H, value, key]
        for t in range(n):
            S = S * keep[at + t][:, None, None]
            u = beta[at + t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None, :]
            o[t] = torch.einsum("hvk,hk->hv", S, q[t])
        memory[i] = S
        outs.append(o)
        at += n
    o = torch.cat(outs)
    y = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * w["out_norm"].to(F64)
    y = y.reshape(-1, H * d) * (gate * torch.sigmoid(gate))
    return dict(out=y @ w["o_weight"].to(F64).t(), memory=memory, taps=torch.stack(new_taps))
