"""Workloads of this framework over which its speed is measured, with their inputs and their exact results.

A case is a plain dict; ``kind`` says which public entry points it goes through:

  step        ``ModelRunner.step`` of an OPT model (``LLMEngine``'s runner): token ids in, float32 logits out.  A prompt
              step brings whole prompts or portions, a decode step one token per request over a filled cache.
  linear      ``ops.linear``: one product with bias and activation, both storage types, decode and prompt row counts.
  attention   ``ops.attention_plain``: the 32-bit path's paged attention, prompts and single tokens.
  experts     ``RoutedExperts.forward``: router, grouping, the experts' two products, weighted sum.
  delta       ``ops.delta_rule``: the gated delta rule over the requests' tokens, state read and moved on.
  hgrn2       ``ops.hgrn2_scan``: the gated linear recurrence, likewise.
  grouped     ``ops.gqa_attention_tiles`` / ``ops.gqa_attention_single``: windowed attention with shared key heads.
  latent      ``ops.latent_attention``: attention over a paged cache of latent rows.

Sizes are those of OPT-125M to OPT-6.7B and of the ``w2048`` / ``w4096`` designs that ``bench.py`` measures.
"""
from __future__ import annotations

import math
import random

import torch

from swifttransformer_b200 import ops
from swifttransformer_b200.config import OptConfig
from swifttransformer_b200.engine.engine import LLMEngine
from swifttransformer_b200.engine.step import StepContext, StepEntry
from swifttransformer_b200.models.base import CausalLM
from swifttransformer_b200.models.registry import build_model_def
from swifttransformer_b200.parts.moe import RoutedExperts

DEV = "cuda"
TYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
PAGE = 16
EPS = 1e-5


# ------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one request's token through the smallest product of a layer (OPT-1.3B's output projection)
        dict(name="linear_bf16_one_row", kind="linear", dtype="bf16", rows=1, k=2048, out=2048, act="none"),
        # a batch of eight decoding in the 32-bit path (OPT-6.7B's output projection)
        dict(name="linear_f32_decode", kind="linear", dtype="f32", rows=8, k=4096, out=4096, act="none"),
        # a prompt of a thousand tokens in the 32-bit path (OPT-1.3B's first feed-forward product)
        dict(name="linear_f32_prompt", kind="linear", dtype="f32", rows=1000, k=2048, out=8192, act="relu"),
        # three prompts of unequal length in the 32-bit path (OPT-1.3B's heads)
        dict(name="attention_f32_prompt", kind="attention", dtype="f32", requests=3, tokens=700, context=0, heads=32, dim=64),
        # eight requests of about 512 tokens decoding together: the benchmark's step, on four of OPT-1.3B's layers
        dict(name="step_decode_8", kind="step", dtype="bf16", requests=8, tokens=8, context=4096, width=2048, heads=32,
             ffn=8192, layers=4, vocab=50272),
        # prompts of 2000 tokens in all in one step: the benchmark's prefill, ragged
        dict(name="step_prompt_2000", kind="step", dtype="bf16", requests=3, tokens=2000, context=0, width=2048, heads=32,
             ffn=8192, layers=4, vocab=50272),
        # a batch of eight decoding through a mixture of gated experts (the w2048 Pikadra mixture)
        dict(name="experts_decode_8", kind="experts", dtype="bf16", tokens=8, width=2048, experts=8, top=2, inner=512,
             limit=0.0),
        # a prompt of 2000 tokens through a mixture of clamped experts (the w2048 Nafelix mixture)
        dict(name="experts_prompt_2000", kind="experts", dtype="bf16", tokens=2000, width=2048, experts=8, top=2,
             inner=2752, limit=7.0),
        # a prompt of 2000 tokens through the delta rule (the w2048 Norelix recurrence)
        dict(name="delta_prompt_2000", kind="delta", dtype="bf16", requests=1, tokens=2000, heads=8, groups=4, dim=128,
             vdim=128, rank=16, taps=4),
        # a prompt of 2000 tokens through the gated linear recurrence (the w2048 Fanidra recurrence)
        dict(name="hgrn2_prompt_2000", kind="hgrn2", dtype="bf16", requests=1, tokens=2000, heads=16, dim=128, vdim=128),
        # a prompt of 2000 tokens through the windowed attention (the w2048 Norelix pair's left mixer)
        dict(name="grouped_prompt_2000", kind="grouped", dtype="bf16", requests=1, tokens=2000, context=0, heads=16,
             kv_heads=4, dim=64, vdim=128, window=512, keep=4),
        # prompts of 2000 tokens through the latent attention (the w2048 Pikadra mixer)
        dict(name="latent_prompt_2000", kind="latent", dtype="bf16", requests=2, tokens=2000, context=0, heads=16, rank=512,
             rot=64, window=0),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges: prompts from a few tokens to the benchmark's 2000, batches of single tokens
    from one request to 64, the presets' and designs' sizes."""
    kind = rng.choice(["step", "linear", "linear", "attention", "experts", "experts", "delta", "hgrn2", "grouped", "latent"])
    decode = rng.random() < 0.4
    batch = _spread(rng, 1, 64)
    # a prompt step: up to four requests of `tokens` in all; a decode step: a token for each request
    requests = batch if decode else rng.randint(1, 4)
    tokens = batch if decode else _spread(rng, 4 * requests, 2000)
    context = requests * _spread(rng, 8, 1024) if decode else rng.choice([0, 0, requests * rng.randint(1, 300)])
    dtype = rng.choice(["bf16", "f32"])
    if kind == "step":
        width, heads, ffn = rng.choice([(768, 12, 3072), (2048, 32, 8192)])
        if dtype == "f32":
            tokens = min(tokens, 512)
        return dict(kind=kind, dtype=dtype, requests=requests, tokens=max(tokens, requests), context=context, width=width,
                    heads=heads, ffn=ffn, layers=rng.choice([2, 4]) if width == 768 else 2, vocab=50272)
    if kind == "linear":
        k, out = rng.choice([(768, 2304), (2048, 2048), (2048, 6144), (2048, 8192), (8192, 2048), (4096, 4096), (5504, 2048),
                             (2048, 2117)])
        return dict(kind=kind, dtype=dtype, rows=_spread(rng, 1, 32) if decode else _spread(rng, 33, 1000), k=k, out=out,
                    act=rng.choice(["none", "relu", "gelu"]))
    if kind == "attention":
        heads, dim = rng.choice([(12, 64), (32, 64), (32, 80), (32, 128)])
        return dict(kind=kind, dtype="f32", requests=requests, tokens=min(tokens, 700), context=context, heads=heads, dim=dim)
    if kind == "experts":
        width, inner = rng.choice([(2048, 512), (2048, 2752), (4096, 1024)])
        return dict(kind=kind, dtype="bf16", tokens=tokens, width=width, experts=rng.choice([8, 12, 16]),
                    top=rng.choice([1, 2, 4]) if inner <= 1024 else 2, inner=inner, limit=rng.choice([0.0, 7.0]))
    if kind == "delta":
        groups = rng.choice([2, 4])
        return dict(kind=kind, dtype=dtype, requests=requests, tokens=tokens, heads=groups * rng.choice([1, 2]), groups=groups,
                    dim=rng.choice([64, 128]), vdim=rng.choice([64, 128]), rank=rng.choice([0, 16]), taps=4)
    if kind == "hgrn2":
        return dict(kind=kind, dtype=dtype, requests=requests, tokens=tokens, heads=rng.choice([4, 8, 16]),
                    dim=rng.choice([64, 128]), vdim=rng.choice([64, 128]))
    if kind == "grouped":
        kv = rng.choice([2, 4])
        return dict(kind=kind, dtype="bf16", requests=requests, tokens=tokens, context=context, heads=kv * rng.choice([1, 4]),
                    kv_heads=kv, dim=rng.choice([64, 128]), vdim=128, window=rng.choice([0, 512]), keep=rng.choice([0, 4]))
    return dict(kind=kind, dtype="bf16", requests=requests, tokens=tokens, context=context, heads=rng.choice([8, 16]), rank=512,
                rot=64, window=rng.choice([0, 512]))


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000 + salt)
    return g


def _normal(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def _ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _parts(total, n, seed):
    """``total`` cut into n ragged parts of at least one (about equal on average; the same for the same numbers)."""
    rng = random.Random(f"{total},{n},{seed}")
    weights = [rng.uniform(0.5, 1.5) for _ in range(n)]
    lens = [max(1, int(total * w / sum(weights))) for w in weights]
    lens[0] += total - sum(lens)
    return lens if lens[0] >= 1 else [total - (n - 1)] + [1] * (n - 1)


def _lengths(case):
    """(new tokens, tokens already in the cache) of each request of a case."""
    b = case["requests"]
    new = [1] * b if case["tokens"] == b else _parts(case["tokens"], b, 1)
    return new, (_parts(case["context"], b, 2) if case.get("context") else [0] * b)


class _Step:
    """The index arrays of a step, and a block table over shuffled pages."""

    def __init__(self, new, start, seed):
        b = len(new)
        self.n = sum(new)
        at = [0]
        for n in new:
            at.append(at[-1] + n)
        self.q_start, self.start_pos, self.slots = _ints(at), _ints(start), _ints(list(range(b)))
        self.positions = _ints([s + j for n, s in zip(new, start) for j in range(n)])
        self.seq = _ints([i for i, n in enumerate(new) for _ in range(n)])
        need = [-(-(n + s) // PAGE) for n, s in zip(new, start)]
        self.pages = sum(need)
        order = list(range(self.pages))
        random.Random(seed).shuffle(order)
        table, k = [[-1] * max(need) for _ in need], 0
        for i, m in enumerate(need):
            table[i][:m] = order[k:k + m]
            k += m
        self.table = table
        self.block_table = _ints(table)
        rows = ops.attention_prefill_tile_rows()
        tiles = [(i, o) for i, n in enumerate(new) for o in range(0, n, rows)]
        tiles.sort(key=lambda t: -(start[t[0]] + min(new[t[0]], t[1] + rows)))       # the longest key ranges first
        self.tiles, self.n_tiles, self.tile_rows = _ints(tiles), len(tiles), rows
        self.status = torch.zeros(1, dtype=torch.int32, device=DEV)


def _opt_weights(case, seed):
    """Random OPT parameters by checkpoint name, as float32 holding bfloat16 values."""
    g, w, f = _gen(seed), case["width"], case["ffn"]
    t = {}

    def mat(name, *shape):
        t[name] = _normal(g, *shape, std=0.02).to(torch.bfloat16).float()

    def pair(name, n, gain):
        t[name + ".weight"] = (1 + _normal(g, n, std=0.1)).to(torch.bfloat16).float()
        mat(name + ".bias", n)
    root = "model.decoder."
    mat(root + "embed_tokens.weight", case["vocab"], w)
    mat(root + "embed_positions.weight", 2050, w)
    for i in range(case["layers"]):
        p = f"{root}layers.{i}."
        for name, rows, cols in (("self_attn.q_proj", w, w), ("self_attn.k_proj", w, w), ("self_attn.v_proj", w, w),
                                 ("self_attn.out_proj", w, w), ("fc1", f, w), ("fc2", w, f)):
            mat(f"{p}{name}.weight", rows, cols)
            mat(f"{p}{name}.bias", rows)
        pair(p + "self_attn_layer_norm", w, True)
        pair(p + "final_layer_norm", w, True)
    pair(root + "final_layer_norm", w, True)
    return t


def _opt_tokens(case, seed):
    new, start = _lengths(case)
    rng = random.Random(seed)
    return [[rng.randrange(3, case["vocab"]) for _ in range(n + s)] for n, s in zip(new, start)], new, start


def _prepare_step(case, seed):
    dtype = TYPES[case["dtype"]]
    cfg = OptConfig.from_dict(dict(vocab_size=case["vocab"], hidden_size=case["width"], num_hidden_layers=case["layers"],
                                   ffn_dim=case["ffn"], num_attention_heads=case["heads"], max_position_embeddings=2048))
    mdef = build_model_def(cfg)
    raw = _opt_weights(case, seed)
    tensors = {}
    for spec in mdef.param_specs():
        if spec.tied_to is None:
            tensors[spec.name] = raw[spec.name].to(spec.storage_dtype(dtype)).contiguous()
    for spec in mdef.param_specs():
        if spec.tied_to is not None:
            tensors[spec.name] = tensors[spec.tied_to]
    model = CausalLM(mdef, tensors, dtype, torch.device(DEV, 0))
    tokens, new, start = _opt_tokens(case, seed)
    pages = sum(-(-len(t) // PAGE) for t in tokens) + len(tokens)
    engine = LLMEngine(model, page_size=PAGE, num_pages=pages, max_batch_tokens=2048, chunk_size=2048,
                       max_num_seqs=max(len(tokens), 8), max_seq_len=2048)
    slots = [engine.cache.alloc_slot() for _ in tokens]
    for slot, t, s in zip(slots, tokens, start):
        if s:
            engine.runner.step([StepEntry(slot, t[:s], 0, [])])
    entries = [StepEntry(slot, t[s:], s, [n - 1]) for slot, t, n, s in zip(slots, tokens, new, start)]
    state = dict(engine=engine, entries=entries)
    _run_step(state)                     # records the step's shape, as ``LLMEngine.warm_up`` does before requests arrive
    return state


def _run_step(state):
    engine = state["engine"]
    logits = engine.runner.step(state["entries"])
    for e in state["entries"]:           # the step's tokens are taken back, so that the same step can follow
        engine.cache.commit(e.slot, e.start_pos)
    return logits


def _prepare_linear(case, seed):
    g, dtype = _gen(seed), TYPES[case["dtype"]]
    bias = _normal(g, case["out"], std=0.02).to(torch.bfloat16).float()
    return dict(a=_normal(g, case["rows"], case["k"], dtype=dtype), w=_normal(g, case["out"], case["k"], std=0.02, dtype=dtype),
                bias=bias, bias_low=ops.lossless_bf16(bias), act=case["act"])


def _prepare_attention(case, seed):
    g, dtype = _gen(seed), TYPES[case["dtype"]]
    new, start = _lengths(case)
    st = _Step(new, start, seed)
    h, d = case["heads"], case["dim"]
    return dict(st=st, h=h, scale=d ** -0.5, q=_normal(g, st.n, h * d, dtype=dtype),
                pool=_normal(g, st.pages, 1, 2, h, PAGE, d, dtype=dtype), out=torch.empty((st.n, h * d), dtype=dtype, device=DEV))


def _expert_weights(case, seed):
    g, n, w = _gen(seed), case["inner"], case["width"]
    t = {}
    for e in range(case["experts"]):
        for key, shape in (("gate", (n, w)), ("up", (n, w)), ("down", (w, n))):
            t[f"{e}.{key}"] = _normal(g, *shape, std=0.02, dtype=TYPES[case["dtype"]])
    t["router"] = _normal(g, case["experts"], w, std=0.02).to(torch.bfloat16).float()
    return t, _normal(g, case["tokens"], w, dtype=TYPES[case["dtype"]])


def _prepare_experts(case, seed):
    t, h = _expert_weights(case, seed)
    names = [{key: f"{e}.{key}" for key in ("gate", "up", "down")} for e in range(case["experts"])]
    part = RoutedExperts(case["width"], case["inner"], case["experts"], case["top"], "silu", names, "router",
                         limit=case["limit"] or None, shift=1.0 if case["limit"] else 0.0)
    part.bind(t)
    ctx = StepContext()
    ctx.positions, ctx.n_tokens = _ints(list(range(case["tokens"]))), case["tokens"]
    return dict(part=part, h=h, ctx=ctx)


def _prepare_delta(case, seed):
    g, dtype = _gen(seed), TYPES[case["dtype"]]
    new, start = _lengths(case)
    st = _Step(new, start, seed)
    H, G, d, vd, rank, taps = (case[k] for k in ("heads", "groups", "dim", "vdim", "rank", "taps"))
    C = 2 * G * d + H * vd
    ra, rg = (rank, rank) if rank else (H, H * vd)
    n_dt = H * d if rank else H
    # decays as such models start with: rates of 1 to 16, steps of 0.001 to 0.1
    rate = torch.rand(H, generator=g, device=DEV) * 15 + 1
    step = torch.exp(torch.rand(n_dt, generator=g, device=DEV) * math.log(100.0) + math.log(0.001))
    state0 = torch.zeros((len(new), H, d, vd), device=DEV)
    return dict(st=st, dims=(H, G, d, vd), offs=(C, C + H, C + H + ra), proj=_normal(g, st.n, C + H + ra + rg),
                conv_w=_normal(g, C, taps, std=0.5), tails=torch.zeros((len(new), taps - 1, C), device=DEV),
                w_a2=_normal(g, H * d, rank, std=0.02, dtype=dtype) if rank else None,
                w_g2=_normal(g, H * vd, rank, std=0.3, dtype=dtype) if rank else None, a_log=torch.log(rate),
                dt_bias=step + torch.log(-torch.expm1(-step)), norm_w=1 + _normal(g, vd, std=0.1), state0=state0,
                state=state0.clone(), single=max(new) == 1,
                scratch=torch.empty(ops.delta_rule_scratch(st.n, H, G, d, vd), device=DEV),
                out=torch.empty((st.n, H * vd), dtype=dtype, device=DEV))


def _run_delta(s):
    st = s["st"]
    s["state"].copy_(s["state0"])        # a request starts from a cleared state
    if s["single"]:
        s["tails"].zero_()
    ops.delta_rule(s["proj"], *s["offs"], s["conv_w"], s["tails"], s["w_a2"], s["a_log"], s["dt_bias"], s["w_g2"], s["norm_w"],
                   EPS, 1.0, s["state"], True, s["single"], s["scratch"], s["out"], st.positions, st.seq, st.q_start,
                   st.slots, len(s["state0"]), *s["dims"])
    return s["out"], s["state"]


def _prepare_hgrn2(case, seed):
    g, dtype = _gen(seed), TYPES[case["dtype"]]
    new, start = _lengths(case)
    st = _Step(new, start, seed)
    H, d, vd = case["heads"], case["dim"], case["vdim"]
    state0 = _normal(g, len(new), H, d, vd, std=0.1)
    return dict(st=st, dims=(H, d, vd), proj=_normal(g, st.n, 2 * H * d + H * vd, dtype=dtype), f_bias=_normal(g, H * d, std=0.5) + 2,
                lower=torch.rand(H * d, generator=g, device=DEV) * 0.9, norm_w=1 + _normal(g, vd, std=0.1), state0=state0,
                state=state0.clone(), scratch=torch.empty(st.n * H * (vd + 2 * d), device=DEV),
                out=torch.empty((st.n, H * vd), dtype=dtype, device=DEV))


def _run_hgrn2(s):
    st, (H, d, vd) = s["st"], s["dims"]
    s["state"].copy_(s["state0"])
    ops.hgrn2_scan(s["proj"], 0, H * d, 2 * H * d, s["f_bias"], s["lower"], s["norm_w"], EPS, s["state"], s["out"], st.positions,
                   st.q_start, st.slots, len(s["state0"]), H, d, vd, scratch=s["scratch"])
    return s["out"], s["state"]


def _prepare_grouped(case, seed):
    g, dtype = _gen(seed), TYPES[case["dtype"]]
    new, start = _lengths(case)
    st = _Step(new, start, seed)
    H, G, d, vd = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
    return dict(st=st, dims=(H, G, d, vd), q=_normal(g, st.n, H * d, dtype=dtype),
                pool=_normal(g, st.pages, 1, G * PAGE * (d + vd), dtype=dtype), window=case["window"],
                keep=case["keep"] if case["window"] else 0, single=max(new) == 1,
                out=torch.empty((st.n, H * vd), dtype=dtype, device=DEV))


def _run_grouped(s):
    st, (H, G, d, vd) = s["st"], s["dims"]
    # (window, kept first keys, one more term in the denominator: a logit of zero; no gate)
    tail = (H, G, d, vd, PAGE, d ** -0.5, s["window"], s["keep"], 0.0, None, 0, 1.0)
    if s["single"]:
        return ops.gqa_attention_single(s["q"], s["pool"], 0, s["out"], st.positions, st.seq, st.slots, st.block_table, *tail,
                                        status=st.status)
    return ops.gqa_attention_tiles(s["q"], s["pool"], 0, s["out"], st.tiles, st.n_tiles, st.tile_rows, st.q_start,
                                   st.start_pos, st.slots, st.block_table, *tail, status=st.status)


def _prepare_latent(case, seed):
    g, dtype = _gen(seed), TYPES[case["dtype"]]
    new, start = _lengths(case)
    st = _Step(new, start, seed)
    H, kr, rot = case["heads"], case["rank"], case["rot"]
    hold = {}

    def scratch(n):                      # the step's scratch memory, kept from call to call
        if n not in hold:
            hold[n] = torch.empty(n, device=DEV)
        return hold[n]
    return dict(st=st, dims=(H, kr, rot), q=_normal(g, st.n, H * (kr + rot), std=0.7, dtype=dtype), window=case["window"],
                pool=_normal(g, st.pages, 1, PAGE * (kr + rot), dtype=dtype), sink=_normal(g, H),
                gates=_normal(g, st.n, H, dtype=dtype), scratch=scratch, n_seqs=len(new),
                out=torch.empty((st.n, H * kr), dtype=dtype, device=DEV))


def _run_latent(s):
    st, (H, kr, rot) = s["st"], s["dims"]
    return ops.latent_attention(s["q"], s["pool"], 0, s["out"], st.positions, st.seq, st.slots, st.block_table, H, kr, rot, PAGE,
                                192 ** -0.5, s["sink"], s["gates"], status=st.status, q_start=st.q_start,
                                start_pos=st.start_pos, n_seqs=s["n_seqs"], scratch=s["scratch"], window=s["window"])


_PREPARE = dict(step=_prepare_step, linear=_prepare_linear, attention=_prepare_attention, experts=_prepare_experts,
                delta=_prepare_delta, hgrn2=_prepare_hgrn2, grouped=_prepare_grouped, latent=_prepare_latent)


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    kind = state["kind"]
    if kind == "step":
        return _run_step(state)
    if kind == "linear":
        return ops.linear(state["a"], state["w"], state["bias"], state["act"], bias_bf16=state["bias_low"])
    if kind == "attention":
        st = state["st"]
        return ops.attention_plain(state["q"], state["pool"], 0, state["out"], st.positions, st.seq, st.slots, st.block_table,
                                   state["h"], state["scale"], 0, st.status)
    if kind == "experts":
        return state["part"].forward(state["h"], state["ctx"]).value
    return {"delta": _run_delta, "hgrn2": _run_hgrn2, "grouped": _run_grouped, "latent": _run_latent}[kind](state)


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _keys(case, window=0, keep=0):
    """(query, key) pairs that attend, and key rows read once, over the case's requests."""
    pairs = rows = 0
    for n, s in zip(*_lengths(case)):
        seen = [min(p + 1, window + keep) if window else p + 1 for p in range(s, s + n)]
        pairs += sum(seen)
        rows += min(s + n, seen[0] + n - 1)
    return pairs, rows


def work(case):
    kind, e = case["kind"], 2 if case["dtype"] == "bf16" else 4
    if kind == "linear":
        n, k, m = case["rows"], case["k"], case["out"]
        return dict(bytes=(n * k + k * m + n * m) * e + m * 4, flops=2 * n * k * m)
    if kind == "step":
        w, f, L, n = case["width"], case["ffn"], case["layers"], case["tokens"]
        pairs, rows = _keys(case)
        per = 4 * w * w + 2 * w * f
        head = case["vocab"] * w
        return dict(bytes=(L * per + head + L * 2 * w * rows + 2 * n * w) * e + case["requests"] * case["vocab"] * 4,
                    flops=2 * n * L * per + 4 * L * w * pairs + 2 * case["requests"] * head)
    if kind == "attention":
        hd = case["heads"] * case["dim"]
        pairs, rows = _keys(case)
        return dict(bytes=(2 * case["tokens"] + 2 * rows) * hd * e, flops=4 * hd * pairs)
    if kind == "experts":
        n, w, i = case["tokens"] * case["top"], case["width"], case["inner"]
        live = min(case["experts"], n)
        return dict(bytes=(live * 3 * w * i + case["tokens"] * w) * e + case["tokens"] * w * 4, flops=6 * n * w * i)
    if kind == "delta":
        n, H, G, d, vd = (case[k] for k in ("tokens", "heads", "groups", "dim", "vdim"))
        cols = 2 * G * d + H * vd + H + (2 * case["rank"] if case["rank"] else H + H * vd)
        return dict(bytes=n * cols * 4 + n * H * vd * e + 2 * case["requests"] * H * d * vd * 4, flops=7 * n * H * d * vd)
    if kind == "hgrn2":
        n, H, d, vd = (case[k] for k in ("tokens", "heads", "dim", "vdim"))
        return dict(bytes=n * H * (2 * d + 2 * vd) * e + 2 * case["requests"] * H * d * vd * 4, flops=5 * n * H * d * vd)
    if kind == "grouped":
        H, G, d, vd = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
        pairs, rows = _keys(case, case["window"], case["keep"] if case["window"] else 0)
        return dict(bytes=(case["tokens"] * H + rows * G) * (d + vd) * e, flops=2 * H * (d + vd) * pairs)
    H, kr, rot = case["heads"], case["rank"], case["rot"]
    pairs, rows = _keys(case, case["window"])
    return dict(bytes=(case["tokens"] * H * (2 * kr + rot) + rows * (kr + rot)) * e, flops=2 * H * (2 * kr + rot) * pairs)


def tolerance(case):
    """About four times the present error against the exact results, measured over listed and drawn cases.  32 bits: 1.1e-6
    for the longest products, 2.2e-6 for two layers, 4e-7 for attention and recurrences (whose sums may be ordered
    otherwise).  bfloat16: one rounding of the result is 1.7e-3, two (a product whose bias and
    activation follow it) 3e-3, probabilities rounded on the way 2.1e-3,
    a mixture's inner rows 3.5e-3, four layers 5.1e-3."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5 if case["kind"] == "step" else 5e-6}
    return {"rel": {"step": 2e-2, "experts": 1.4e-2, "grouped": 8e-3, "latent": 8e-3, "linear": 1.2e-2}.get(case["kind"], 7e-3)}


# ------------------------------------------------------------------------------------------ exact results
def _act(y, act):
    if act == "relu":
        return y.clamp(min=0)
    return 0.5 * y * (1 + torch.erf(y / math.sqrt(2.0))) if act == "gelu" else y


def _rows_of(st, pool, i, n):
    """The first n cache rows of request i: pool [pages, PAGE, ...] read through the block table."""
    pages = torch.tensor([p for p in st.table[i] if p >= 0], device=DEV)
    return pool[pages].flatten(0, 1)[:n]


def _mask(n, s, window=0, keep=0):
    p = torch.arange(s, s + n, device=DEV)[:, None]
    j = torch.arange(s + n, device=DEV)[None, :]
    ok = j <= p
    return ok & ((j > p - window) | (j < keep)) if window else ok


def _exact_step(case, seed):
    w = {k: v.double() for k, v in _opt_weights(case, seed).items()}
    tokens, new, start = _opt_tokens(case, seed)
    H, W, root = case["heads"], case["width"], "model.decoder."
    d = W // H

    def norm(x, p):
        return torch.nn.functional.layer_norm(x, (W,), w[p + ".weight"], w[p + ".bias"], EPS)

    def lin(x, p):
        return x @ w[p + ".weight"].T + w[p + ".bias"]
    out = []
    for t in tokens:
        n = len(t)
        ids = torch.tensor(t, device=DEV)
        x = w[root + "embed_tokens.weight"][ids] + w[root + "embed_positions.weight"][torch.arange(n, device=DEV) + 2]
        for i in range(case["layers"]):
            p = f"{root}layers.{i}."
            h = norm(x, p + "self_attn_layer_norm")
            q, k, v = (lin(h, f"{p}self_attn.{c}_proj").view(n, H, d).transpose(0, 1) for c in "qkv")
            a = (q @ k.transpose(1, 2) * d ** -0.5).masked_fill(~_mask(n, 0), -math.inf).softmax(-1)
            x = x + lin((a @ v).transpose(0, 1).reshape(n, W), p + "self_attn.out_proj")
            x = x + lin(lin(norm(x, p + "final_layer_norm"), p + "fc1").clamp(min=0), p + "fc2")
        out.append(norm(x[-1:], root + "final_layer_norm") @ w[root + "embed_tokens.weight"].T)
    return torch.cat(out)


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    st, h, d = s["st"], case["heads"], case["dim"]
    q, kv = s["q"].double().view(st.n, h, d), s["pool"][:, 0].permute(0, 3, 1, 2, 4)      # [pages, PAGE, k|v, heads, dim]
    out, at = [], 0
    for i, (n, c) in enumerate(zip(*_lengths(case))):
        rows = _rows_of(st, kv, i, n + c).double()
        a = torch.einsum("qhd,khd->hqk", q[at:at + n], rows[:, 0]) * s["scale"]
        a = a.masked_fill(~_mask(n, c), -math.inf).softmax(-1)
        out.append(torch.einsum("hqk,khd->qhd", a, rows[:, 1]).reshape(n, h * d))
        at += n
    return torch.cat(out)


def _exact_experts(case, seed):
    t, h = _expert_weights(case, seed)
    x = h.double()
    p = (x @ t["router"].double().T).softmax(-1)
    weight, chosen = p.topk(case["top"], dim=-1)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        token, place = (chosen == e).nonzero(as_tuple=True)
        g, u = (x[token] @ t[f"{e}.{key}"].double().T for key in ("gate", "up"))
        if case["limit"]:
            g, u = g.clamp(max=case["limit"]), u.clamp(-case["limit"], case["limit"]) + 1
        y = (g * torch.sigmoid(g) * u) @ t[f"{e}.down"].double().T
        out.index_add_(0, token, y * weight[token, place][:, None])
    return out


def _exact_delta(case, seed):
    s = _prepare_delta(case, seed)
    H, G, d, vd = s["dims"]
    C, rank, taps, silu = 2 * G * d + H * vd, case["rank"], case["taps"], torch.nn.functional.silu
    b_off, a_off, g_off = s["offs"]
    outs, states, at = [], [], 0
    for n in _lengths(case)[0]:
        rows = s["proj"][at:at + n].double()
        at += n
        past = torch.cat([torch.zeros((taps - 1, C), dtype=torch.float64, device=DEV), rows[:, :C]])
        z = silu(sum(past[j:j + n] * s["conv_w"][:, j].double() for j in range(taps)))
        q, k, v = z[:, :G * d].view(n, G, d), z[:, G * d:2 * G * d].view(n, G, d), z[:, 2 * G * d:].view(n, H, vd)
        q, k = (x * (x.square().sum(-1, keepdim=True) + 1e-6).rsqrt() for x in (q * 1, k))
        q, k = ((x * m).repeat_interleave(H // G, dim=1) for x, m in ((q, d ** -0.5), (k, 1.0)))
        beta = torch.sigmoid(rows[:, b_off:b_off + H])
        if rank:
            dt = rows[:, a_off:a_off + rank] @ s["w_a2"].double().T + s["dt_bias"].double()
            gate = rows[:, g_off:g_off + rank] @ s["w_g2"].double().T
        else:
            dt = (rows[:, a_off:a_off + H] + s["dt_bias"].double()).repeat_interleave(d, dim=1)
            gate = rows[:, g_off:g_off + H * vd]
        decay = torch.exp(-s["a_log"].double().exp()[:, None] * torch.logaddexp(dt, torch.zeros_like(dt)).view(n, H, d))
        S = torch.zeros((H, d, vd), dtype=torch.float64, device=DEV)
        o = torch.empty((n, H, vd), dtype=torch.float64, device=DEV)
        for t in range(n):
            S = S * decay[t][:, :, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = o * (o.square().mean(-1, keepdim=True) + EPS).rsqrt() * s["norm_w"].double()
        outs.append(o.view(n, H * vd) * torch.sigmoid(gate))
        states.append(S)
    return torch.cat(outs), torch.stack(states)


def _exact_hgrn2(case, seed):
    s = _prepare_hgrn2(case, seed)
    H, d, vd = s["dims"]
    outs, states, at = [], [], 0
    for i, n in enumerate(_lengths(case)[0]):
        rows = s["proj"][at:at + n].double()
        at += n
        q = torch.nn.functional.silu(rows[:, :H * d]).view(n, H, 1, d)
        lower = s["lower"].double()
        f = (lower + (1 - lower) * torch.sigmoid(rows[:, H * d:2 * H * d] + s["f_bias"].double())).view(n, H, d, 1)
        v = rows[:, 2 * H * d:].view(n, H, 1, vd)
        S = s["state0"][i].double()
        o = torch.empty((n, H, vd), dtype=torch.float64, device=DEV)
        for t in range(n):
            S = torch.baddbmm(S * f[t], 1 - f[t], v[t])
            o[t] = torch.bmm(q[t], S)[:, 0]
        outs.append((o * (o.square().mean(-1, keepdim=True) + EPS).rsqrt() * s["norm_w"].double()).view(n, H * vd))
        states.append(S)
    return torch.cat(outs), torch.stack(states)


def _exact_grouped(case, seed):
    s = _prepare_grouped(case, seed)
    st, (H, G, d, vd) = s["st"], s["dims"]
    q = s["q"].double().view(st.n, H, d)
    # a page holds its key heads [G][PAGE][d], then its value heads [G][PAGE][vd]
    cut = G * PAGE * d
    pages = len(s["pool"])
    keys = s["pool"][:, 0, :cut].reshape(pages, G, PAGE, d).transpose(1, 2)
    values = s["pool"][:, 0, cut:].reshape(pages, G, PAGE, vd).transpose(1, 2)
    out, at = [], 0
    for i, (n, c) in enumerate(zip(*_lengths(case))):
        k, v = (_rows_of(st, x, i, n + c).double().repeat_interleave(H // G, dim=1) for x in (keys, values))
        a = torch.einsum("qhd,khd->hqk", q[at:at + n], k) * d ** -0.5
        a = a.masked_fill(~_mask(n, c, s["window"], s["keep"]), -math.inf)
        a = torch.cat([a, torch.zeros_like(a[..., :1])], dim=-1).softmax(-1)[..., :-1]
        out.append(torch.einsum("hqk,khd->qhd", a, v).reshape(n, H * vd))
        at += n
    return torch.cat(out)


def _exact_latent(case, seed):
    s = _prepare_latent(case, seed)
    st, (H, kr, rot) = s["st"], s["dims"]
    q = s["q"].double().view(st.n, H, kr + rot)
    rows_all = s["pool"][:, 0].reshape(-1, PAGE, kr + rot)
    out, at = [], 0
    for i, (n, c) in enumerate(zip(*_lengths(case))):
        rows = _rows_of(st, rows_all, i, n + c).double()
        a = (q[at:at + n].transpose(0, 1) @ rows.T) * 192 ** -0.5
        a = a.masked_fill(~_mask(n, c, s["window"]), -math.inf)
        a = torch.cat([a, s["sink"].double()[:, None, None].expand(H, n, 1)], dim=-1).softmax(-1)[..., :-1]
        o = (a @ rows[:, :kr]).transpose(0, 1) * torch.sigmoid(s["gates"][at:at + n].double())[:, :, None]
        out.append(o.reshape(n, H * kr))
        at += n
    return torch.cat(out)


def exact(case, seed):
    if case["kind"] == "linear":
        s = _prepare_linear(case, seed)
        return _act(s["a"].double() @ s["w"].double().T + s["bias"].double(), case["act"])
    return {"step": _exact_step, "attention": _exact_attention, "experts": _exact_experts, "delta": _exact_delta,
            "hgrn2": _exact_hgrn2, "grouped": _exact_grouped, "latent": _exact_latent}[case["kind"]](case, seed)
