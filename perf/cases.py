"""What the engine is timed and checked on: single layers through the parts that a model is assembled from, and a whole model
through the step function.

A case names a part (``kind``), its sizes, the step's requests (``new``: the tokens each brings, ``before``: those its cache or
state already covers) and the compute type.  Sizes are those of ``bench.py`` (Qwen3-1.7B layers and the layer sizes of
``--workload designs``) or lie around them.  A step of single tokens runs as a captured graph, as the engine's decode steps do;
prompt portions and mixed steps run eagerly, with a new step context for every pass, as the engine's do.

``exact`` computes the same from the definitions, whole and in float64: it shares the inputs with ``prepare`` and nothing else.
"""

from __future__ import annotations

import math

import torch

import miniserve_b200  # noqa: F401
from miniserve_b200.cache.manager import CacheManager
from miniserve_b200.cache.storage import CacheStorage
from miniserve_b200.config.registry import resolve_architecture
from miniserve_b200.engine.step import StepEntry, StepFunction
from miniserve_b200.parts.base import FEED_FORWARDS, MIXERS, PagedLatentNeed, StateNeed
from miniserve_b200.parts.context import PagedKVView, PagedLatentView, StateView, StepContext
from miniserve_b200.parts.model import DecoderModel
from miniserve_b200.parts.spec import PartSpec

DEVICE = "cuda:0"
EPS = 1e-6
THETA = 1e6
SOFTCAP = 50.0
LIMIT = 7.0            # of the clamped gated activation
GATE_CAP = 15.0        # of the matrix memory's gates
TAPS = 4               # of the short convolutions
TAU = 16.0
FEED_FORWARD_KINDS = ("mlp", "experts")
STATE_KINDS = ("memory", "delta", "decay", "gla", "ssm")


def listed():
    return [
        # A gated feed-forward of a step that decodes one request alone: the smallest call, all latency and one read of the weights.
        dict(name="mlp_one_row", kind="mlp", dtype="bfloat16", new="1", before="0", width=2048, ff=6144),
        # The same layer in the float32 path, which is what logits of given tokens are traced with.
        dict(name="mlp_prompt_float32", kind="mlp", dtype="float32", new="389", before="0", width=2048, ff=6144),
        # Eight conversations of different lengths, each a token further: attention over a paged cache of a few thousand tokens.
        dict(name="attention_decode", kind="attention", dtype="bfloat16", new="1," * 7 + "1",
             before="4096,3011,4095,2048,1777,4001,3500,4090", width=2048, heads=16, kv_heads=8, dim=128, form="plain", page=64),
        # A prompt of odd length beside the next portion of a longer one.
        dict(name="attention_prompt", kind="attention", dtype="bfloat16", new="1777,271", before="0,1000", width=2048, heads=16,
             kv_heads=8, dim=128, form="plain", page=64),
        # Latent attention over a whole prompt, latent of 256 + 32.
        dict(name="latent_prompt", kind="latent", dtype="bfloat16", new="2048", before="0", width=2048, heads=16, dim=64, rot=32,
             vdim=64, rank=256, page=64),
        # The same decoding many requests with long contexts, what a latent cache is made for.
        dict(name="latent_decode", kind="latent", dtype="bfloat16", new="1," * 31 + "1",
             before=",".join(str(8192 - 61 * r) for r in range(32)), width=2048, heads=16, dim=64, rot=32, vdim=64, rank=256, page=64),
        # Routed experts over a prompt: the largest amount of arithmetic a layer brings.
        dict(name="experts_prompt", kind="experts", dtype="bfloat16", new="2048", before="0", width=2048, experts=16, top=4,
             expert_ff=1024, shared=0, form="silu_glu"),
        # Many small experts with a shared one in a decode step of eight requests.
        dict(name="experts_decode", kind="experts", dtype="bfloat16", new="1," * 7 + "1", before="0," * 7 + "0", width=2048, experts=60,
             top=6, expert_ff=1408, shared=2816, form="clamped_glu"),
        # Matrix memory over a prompt of odd length.
        dict(name="memory_prompt", kind="memory", dtype="bfloat16", new="2011", before="0", width=2048, heads=8, dim=128, vdim=256),
        # Delta rule over two portions of different lengths, one of which continues a sequence.
        dict(name="delta_prompt", kind="delta", dtype="bfloat16", new="1500,548", before="0,700", width=2048, heads=16, kv_heads=8,
             dim=128, vdim=128),
        # Selective state space over a prompt.
        dict(name="ssm_prompt", kind="ssm", dtype="bfloat16", new="2048", before="0", width=2048, heads=64, dim=64, state=128, groups=8),
        # A whole four-layer model decoding eight requests through the step function (captured graph), logits out.
        dict(name="model_decode", kind="model", dtype="bfloat16", new="1," * 7 + "1",
             before="2048,1024,2047,1500,777,2000,1999,1025", width=2048, heads=16, kv_heads=8, dim=128, ff=6144, layers=4,
             vocab=32000, page=64),
    ]


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    most = max(_cost(case) for case in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= most:
            return case


def _draw(rng):
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["mlp", "attention", "attention", "latent", "latent", "experts", "experts", "memory", "delta", "decay", "gla",
                       "ssm", "model"])
    dtype = "float32" if rng.random() < 0.12 and kind != "model" else "bfloat16"
    if rng.random() < 0.45:
        count = spread(1, 64)
        new = [1] * count
    else:
        count = rng.choice([1, 1, 2, 3, 5])
        total = spread(40, 512 if dtype == "float32" else 2048 if kind in STATE_KINDS + ("model",) else 4096)
        shares = [rng.uniform(0.3, 1.0) for _ in range(count)]
        new = [max(1, int(total * s / sum(shares))) for s in shares]
        if rng.random() < 0.25 and kind != "model":
            new += [1] * rng.randint(1, 8)                 # decoded tokens beside the portions
    before = [spread(16, 8192) if n == 1 or rng.random() < 0.4 else 0 for n in new]
    case = dict(kind=kind, dtype=dtype, new=",".join(map(str, new)), before=",".join(map(str, before)),
                width=rng.choice([1024, 1536, 2048, 2560]))
    if kind == "mlp":
        case.update(ff=rng.choice([2816, 4096, 6144, 10944]))
    elif kind == "attention":
        heads, kv_heads, dim = rng.choice([(16, 8, 128), (16, 4, 128), (32, 8, 64), (8, 8, 64)])
        case.update(heads=heads, kv_heads=kv_heads, dim=dim, form=rng.choice(["plain", "plain", "capped"]), page=rng.choice([16, 64]))
    elif kind == "latent":
        dim, rot, vdim, rank = rng.choice([(64, 32, 64, 256), (64, 32, 64, 256), (128, 64, 128, 512)])
        case.update(heads=rng.choice([8, 16, 16]), dim=dim, rot=rot, vdim=vdim, rank=rank, page=rng.choice([16, 64]))
    elif kind == "experts":
        experts, top, ff = rng.choice([(16, 4, 1024), (60, 6, 1408), (64, 6, 1408), (8, 2, 1536)])
        form = rng.choice(["silu_glu", "clamped_glu", "relu_square"])
        case.update(experts=experts, top=top, expert_ff=ff, shared=0 if form == "silu_glu" else 2 * ff, form=form)
    elif kind == "memory":
        heads, dim, vdim = rng.choice([(8, 128, 256), (16, 64, 128), (4, 128, 256)])
        case.update(heads=heads, dim=dim, vdim=vdim)
    elif kind == "delta":
        heads, kv_heads, dim, vdim = rng.choice([(16, 8, 128, 128), (32, 16, 64, 64), (16, 16, 128, 128)])
        case.update(heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim)
    elif kind in ("decay", "gla"):
        heads, dim, vdim = rng.choice([(16, 128, 128), (32, 64, 64)])
        case.update(heads=heads, dim=dim, vdim=vdim)
        if kind == "gla":
            case.update(rank=rng.choice([16, 32]))
    elif kind == "ssm":
        heads, dim, state, groups = rng.choice([(64, 64, 128, 8), (32, 128, 64, 4), (32, 64, 128, 1)])
        case.update(heads=heads, dim=dim, state=state, groups=groups)
    else:
        heads, kv_heads, dim = rng.choice([(16, 8, 128), (16, 4, 128), (32, 8, 64)])
        case.update(heads=heads, kv_heads=kv_heads, dim=dim, ff=rng.choice([4096, 6144]), layers=rng.choice([2, 4]), vocab=32000, page=64,
                    before=",".join(str(min(b, 2048)) for b in before))
    return case


# ------------------------------------------------------------------------------------------------------------- inputs
def _lens(case):
    return [int(n) for n in case["new"].split(",")], [int(n) for n in case["before"].split(",")]


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _part_spec(case):
    """(mixer or feed-forward spec, whether it is a feed-forward)."""
    kind, width = case["kind"], case["width"]
    if kind == "mlp":
        return PartSpec("gated_mlp", dict(hidden_size=width, intermediate_size=case["ff"]))
    if kind == "experts":
        form, shared = case["form"], case["shared"] or None
        args = dict(hidden_size=width, experts=case["experts"], top=case["top"], expert_size=case["expert_ff"], shared_size=shared,
                    activation=form)
        if form == "silu_glu":
            args.update(router_bias=False, scoring="sigmoid", normalize=1e-20, weight_scale=2.5)
        elif form == "clamped_glu":
            args.update(router_bias=False, scoring="all_softmax", limit=LIMIT, shared_limit=LIMIT)
        return PartSpec("routed_experts", args)
    position = PartSpec("rope", dict(head_dim=case["dim"], theta=THETA)) if kind == "attention" else None
    if kind == "attention":
        args = dict(hidden_size=width, num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=case["dim"], eps=EPS,
                    position=position, qk_norm=case["form"] == "plain")
        if case["form"] == "capped":
            args.update(score_softcap=SOFTCAP, sink="learned", output_gate=True, bias="qkv", scale=case["dim"] ** -0.5)
        return PartSpec("attention", args)
    if kind == "latent":
        return PartSpec("latent_attention", dict(
            hidden_size=width, num_heads=case["heads"], dim=case["dim"], rot_dim=case["rot"], vdim=case["vdim"], kv_rank=case["rank"],
            scale=(case["dim"] + case["rot"]) ** -0.5, eps=EPS, position=PartSpec("rope", dict(head_dim=case["rot"], theta=THETA))))
    if kind == "memory":
        return PartSpec("matrix_memory", dict(hidden_size=width, heads=case["heads"], head_dim=case["dim"], value_dim=case["vdim"],
                                              gate_cap=GATE_CAP, eps=EPS))
    if kind == "delta":
        return PartSpec("delta_rule", dict(hidden_size=width, heads=case["heads"], kv_heads=case["kv_heads"], head_dim=case["dim"],
                                           value_dim=case["vdim"], taps=TAPS, eps=EPS))
    if kind == "decay":
        return PartSpec("linear_attention", dict(hidden_size=width, heads=case["heads"], head_dim=case["dim"], value_dim=case["vdim"],
                                                 decay=_decays(case), eps=EPS))
    if kind == "gla":
        return PartSpec("gated_linear_attention", dict(hidden_size=width, heads=case["heads"], head_dim=case["dim"],
                                                       value_dim=case["vdim"], rank=case["rank"], tau=TAU, eps=EPS))
    return PartSpec("state_space", dict(hidden_size=width, heads=case["heads"], head_dim=case["dim"], state=case["state"],
                                        groups=case["groups"], taps=TAPS, norm_groups=case["groups"], eps=EPS))


def _decays(case):
    return [1.0 - 2.0 ** (-1 - 8 * h / case["heads"]) for h in range(case["heads"])]


class _Random:
    """Numbers from the seed alone, in the order asked for."""

    def __init__(self, seed):
        self.generator = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.randn(shape, generator=self.generator, device=DEVICE) * std + mean

    def uniform(self, low, high, *shape):
        return torch.rand(shape, generator=self.generator, device=DEVICE) * (high - low) + low

    def permutation(self, n):
        return torch.randperm(n, generator=self.generator, device=DEVICE)

    def step_bias(self, n):
        """Biases whose softplus is spread over 0.001 to 0.1, as state-space layers start out."""
        dt = torch.exp(self.uniform(math.log(1e-3), math.log(0.1), n))
        return dt + torch.log(-torch.expm1(-dt))


def _weights(case, rnd):
    """The layer's tensors by the names that the part asks for, in the types that a loader would give them."""
    kind, width, dtype = case["kind"], case["width"], _dtype(case)

    def matrix(rows, columns, gain=1.0):
        return rnd.normal(rows, columns, std=gain * columns ** -0.5).to(dtype)

    def matrix_f32(rows, columns, gain=1.0):
        return rnd.normal(rows, columns, std=gain * columns ** -0.5)

    def vector(n, mean=1.0, std=0.1):
        return rnd.normal(n, std=std, mean=mean).to(dtype)

    w = {}
    if kind == "mlp":
        w["gate_proj.weight"], w["up_proj.weight"] = matrix(case["ff"], width), matrix(case["ff"], width)
        w["down_proj.weight"] = matrix(width, case["ff"])
        return w
    if kind == "experts":
        ff, glu = case["expert_ff"], case["form"] != "relu_square"
        for e in range(case["experts"]):
            if glu:
                w[f"e{e}.gate"] = matrix(ff, width)
            w[f"e{e}.up"], w[f"e{e}.down"] = matrix(ff, width), matrix(width, ff)
        w["router"] = matrix_f32(case["experts"], width)
        if case["form"] == "relu_square":
            w["router.b"] = vector(case["experts"], 0.0)
        if case["shared"]:
            if glu:
                w["shared.gate"] = matrix(case["shared"], width)
            w["shared.up"], w["shared.down"] = matrix(case["shared"], width), matrix(width, case["shared"])
        return w
    heads, dim = case["heads"], case["dim"]
    if kind == "attention":
        kv = case["kv_heads"]
        w["q_proj.weight"], w["k_proj.weight"], w["v_proj.weight"] = matrix(heads * dim, width), matrix(kv * dim, width), matrix(kv * dim, width)
        w["o_proj.weight"] = matrix(width, heads * dim)
        if case["form"] == "plain":
            w["q_norm.weight"], w["k_norm.weight"] = vector(dim), vector(dim)
        else:
            for name, rows in (("q", heads), ("k", kv), ("v", kv)):
                w[name + "_proj.weight.b"] = vector(rows * dim, 0.0)
            w["sink"], w["g_proj.weight"] = vector(heads, 0.0, 1.0), matrix(heads, width)
        return w
    if kind == "latent":
        rank, rot, vdim = case["rank"], case["rot"], case["vdim"]
        w["q"], w["dkv"] = matrix(heads * (dim + rot), width), matrix(rank + rot, width)
        w["dkv.norm"], w["uk"], w["uv"] = vector(rank), matrix(heads * dim, rank), matrix(heads * vdim, rank)
        w["g"], w["o"] = matrix(heads, width), matrix(width, heads * vdim)
        return w
    if kind == "ssm":
        inner, channels = heads * dim, heads * dim + 2 * case["groups"] * case["state"]
        w["in"] = matrix(inner + channels + heads, width)
        w["conv"], w["conv.b"] = rnd.uniform(-0.5, 0.5, channels, TAPS).to(dtype), vector(channels, 0.0)
        w["dt_bias"], w["A_log"] = rnd.step_bias(heads).to(dtype), torch.log(rnd.uniform(1.0, 16.0, heads)).to(dtype)
        w["D"], w["norm"], w["o"] = vector(heads), vector(inner), matrix(width, inner)
        return w
    vdim = case["vdim"]
    qk_heads = case.get("kv_heads", heads)
    w["q"], w["k"], w["v"] = matrix(qk_heads * dim, width), matrix(qk_heads * dim, width), matrix(heads * vdim, width)
    w["g"], w["o"] = matrix(heads * vdim, width), matrix(width, heads * vdim)
    w["norm"] = vector(vdim if kind in ("delta", "gla") else heads * vdim)
    if kind == "memory":
        w["i"], w["f"] = matrix_f32(heads, width, 0.5), matrix_f32(heads, width, 0.5)
        w["i.b"], w["f.b"] = vector(heads, 0.0, 0.5), vector(heads, 4.0, 1.0)
    elif kind == "delta":
        for name, rows in (("q", qk_heads * dim), ("k", qk_heads * dim), ("v", heads * vdim)):
            w[name + ".conv"] = rnd.uniform(-0.5, 0.5, rows, TAPS).to(dtype)
        w["b"], w["a"] = matrix_f32(heads, width), matrix_f32(heads, width, 0.5)
        w["A_log"], w["dt_bias"] = torch.log(rnd.uniform(1.0, 16.0, heads)).to(dtype), rnd.step_bias(heads).to(dtype)
    elif kind == "gla":
        w["a1"], w["a2"] = matrix_f32(case["rank"], width), matrix_f32(heads * dim, case["rank"])
        w["a2.b"] = vector(heads * dim, 1.0, 0.5)
    return w


def _model_config(case):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=case["width"], intermediate_size=case["ff"],
                num_hidden_layers=case["layers"], num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
                head_dim=case["dim"], vocab_size=case["vocab"], max_position_embeddings=40960, rms_norm_eps=EPS, rope_theta=THETA,
                tie_word_embeddings=True, hidden_act="silu", attention_bias=False)


def _model_weights(case, rnd):
    dtype, width, dim = _dtype(case), case["width"], case["dim"]

    def matrix(rows, columns):
        return rnd.normal(rows, columns, std=columns ** -0.5).to(dtype)

    def vector(n):
        return rnd.normal(n, std=0.1, mean=1.0).to(dtype)

    w = {"model.embed_tokens.weight": matrix(case["vocab"], width), "model.norm.weight": vector(width)}
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = vector(width), vector(width)
        for name, heads in (("q", case["heads"]), ("k", case["kv_heads"]), ("v", case["kv_heads"])):
            w[p + f"self_attn.{name}_proj.weight"] = matrix(heads * dim, width)
        w[p + "self_attn.o_proj.weight"] = matrix(width, case["heads"] * dim)
        w[p + "self_attn.q_norm.weight"], w[p + "self_attn.k_norm.weight"] = vector(dim), vector(dim)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = matrix(case["ff"], width), matrix(case["ff"], width)
        w[p + "mlp.down_proj.weight"] = matrix(width, case["ff"])
    return w


def _state_size(case):
    heads, dim = case["heads"], case["dim"]
    if case["kind"] == "memory":
        return heads * (case["vdim"] + 1) * dim + heads
    if case["kind"] == "delta":
        return (TAPS - 1) * (2 * case["kv_heads"] * dim + heads * case["vdim"]) + heads * case["vdim"] * dim
    if case["kind"] == "ssm":
        return (TAPS - 1) * (heads * dim + 2 * case["groups"] * case["state"]) + heads * dim * case["state"]
    return heads * case["vdim"] * dim


def _inputs(case, seed):
    """Everything that ``prepare`` and ``exact`` share: weights, the step's rows, what caches and states hold."""
    rnd = _Random(seed)
    new, before = _lens(case)
    dtype, kind = _dtype(case), case["kind"]
    got = {"w": _model_weights(case, rnd) if kind == "model" else _weights(case, rnd)}
    if kind == "model":
        got["tokens"] = [torch.randint(0, case["vocab"], (n,), generator=rnd.generator, device=DEVICE) for n in new]
        got["old"] = [[(rnd.normal(b, case["kv_heads"], case["dim"]).to(dtype), rnd.normal(b, case["kv_heads"], case["dim"]).to(dtype))
                       for b in before] for _ in range(case["layers"])]
        return got
    got["x"] = rnd.normal(sum(new), case["width"]).to(dtype)
    if kind == "attention":
        got["old"] = [(rnd.normal(b, case["kv_heads"], case["dim"]).to(dtype), rnd.normal(b, case["kv_heads"], case["dim"]).to(dtype))
                      for b in before]
    elif kind == "latent":
        got["old"] = [rnd.normal(b, case["rank"] + case["rot"]).to(dtype) for b in before]
    elif kind in STATE_KINDS:
        got["slots"] = rnd.permutation(len(new) + 1)[:len(new)]
        states = torch.zeros((len(new) + 1, _state_size(case)), device=DEVICE)
        for r, b in enumerate(before):
            if b:
                row = rnd.normal(_state_size(case), std=0.3)
                if kind == "memory":
                    row[-case["heads"]:] = row[-case["heads"]:].abs()      # running maxima start at 0 and do not fall far
                states[got["slots"][r]] = row
        got["states"] = states
    return got


# ------------------------------------------------------------------------------------------------------ the framework
def _paging(case, rnd):
    """(pages of each request, the table [R, width], slots of the new tokens, pages in all): pages handed out in no order."""
    new, before = _lens(case)
    page = case["page"]
    counts = [(n + b + page - 1) // page for n, b in zip(new, before)]
    shuffled = rnd.permutation(sum(counts)).tolist()
    tables, at = [], 0
    for count in counts:
        tables.append(shuffled[at:at + count])
        at += count
    table = torch.full((len(new), max(counts)), sum(counts), dtype=torch.int32)
    slots = []
    for r, pages in enumerate(tables):
        table[r, :len(pages)] = torch.tensor(pages, dtype=torch.int32)
        slots += [pages[p // page] * page + p % page for p in range(before[r], before[r] + new[r])]
    return tables, table.to(DEVICE), torch.tensor(slots, dtype=torch.int32, device=DEVICE), sum(counts)


def _pages_of(rows, count, page):
    """Rows [T, ...] cut into ``count`` pages [count, page, ...]; the last one's tail is zero."""
    filled = torch.zeros((count * page,) + tuple(rows.shape[1:]), dtype=rows.dtype, device=rows.device)
    filled[:rows.shape[0]] = rows
    return filled.view((count, page) + tuple(rows.shape[1:]))


def _context_args(case, state_slots):
    new, before = _lens(case)
    starts = [0]
    for n in new:
        starts.append(starts[-1] + n)

    def ints(values):
        return torch.tensor(values, dtype=torch.int32, device=DEVICE)

    lens = [n + b for n, b in zip(new, before)]
    return dict(n_tokens=starts[-1], n_requests=len(new), token_ids=ints([0] * starts[-1]),
                positions=ints([p for n, b in zip(new, before) for p in range(b, b + n)]),
                request_of_token=ints([r for r, n in enumerate(new) for _ in range(n)]), query_start=ints(starts),
                context_lens=ints(lens), state_slots=state_slots, logit_rows=ints([0]), max_query_len=max(new),
                max_context_len=max(lens), dtype=_dtype(case), device=torch.device(DEVICE), host_query_start=starts,
                host_context_lens=lens, host_state_slots=list(range(len(new))))


def prepare(case, seed):
    if case["kind"] == "model":
        return _prepare_model(case, seed)
    inputs = _inputs(case, seed)
    new, before = _lens(case)
    spec = _part_spec(case)
    registry = FEED_FORWARDS if case["kind"] in FEED_FORWARD_KINDS else MIXERS
    part = registry.build(spec, prefix="")
    part.load(inputs["w"])
    state = dict(case=case, part=part, x=inputs["x"], cache=None, outputs=[])
    slots = inputs["slots"].to(torch.int32) if "slots" in inputs else torch.arange(len(new), dtype=torch.int32, device=DEVICE)
    state["context"] = _context_args(case, slots)
    if case["kind"] in ("attention", "latent"):
        tables, table, new_slots, pages = _paging(case, _Random(seed + 1))
        page, dtype = case["page"], _dtype(case)
        need = part.cache_need()
        if isinstance(need, PagedLatentNeed):
            pool = torch.zeros((pages + 1, page, need.rank + need.rot), dtype=dtype, device=DEVICE)
            for r, rows in enumerate(inputs["old"]):
                pool[torch.tensor(tables[r], device=DEVICE)] = _pages_of(rows, len(tables[r]), page)
            state["cache"], state["outputs"] = PagedLatentView(pool, table, new_slots, page), [pool]
        else:
            pools = [torch.zeros((pages + 1, need.num_kv_heads, page, need.head_dim), dtype=dtype, device=DEVICE) for _ in range(2)]
            for r, pair in enumerate(inputs["old"]):
                for pool, rows in zip(pools, pair):
                    pool[torch.tensor(tables[r], device=DEVICE)] = _pages_of(rows, len(tables[r]), page).transpose(1, 2)
            state["cache"], state["outputs"] = PagedKVView(pools[0], pools[1], table, new_slots, page), pools
    elif case["kind"] in STATE_KINDS:
        assert isinstance(part.cache_need(), StateNeed) and part.cache_need().shape == (inputs["states"].shape[1],)
        state["cache"], state["outputs"] = StateView(inputs["states"]), [inputs["states"]]
    if max(new) == 1:
        _capture(state)
    return state


def _forward(state, ctx):
    if state["case"]["kind"] in FEED_FORWARD_KINDS:
        return state["part"].forward(state["x"], ctx)
    return state["part"].forward(state["x"], ctx, state["cache"])


def _capture(state):
    """The step of single tokens as a graph, as the engine captures its decode steps (a warm-up first, then the capture)."""
    kept = [t.clone() for t in state["outputs"]]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        _forward(state, StepContext(**state["context"]))
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    state["graph"] = torch.cuda.CUDAGraph()
    state["captured"] = StepContext(**state["context"])
    with torch.cuda.graph(state["graph"]):
        state["y"] = _forward(state, state["captured"])
    for tensor, was in zip(state["outputs"], kept):
        tensor.copy_(was)


def _prepare_model(case, seed):
    inputs = _inputs(case, seed)
    new, before = _lens(case)
    config_dict = _model_config(case)
    architecture = resolve_architecture(config_dict)
    spec = architecture.build_spec(architecture.config_class.from_dict(config_dict))
    dtype, page = _dtype(case), case["page"]
    model = DecoderModel(spec, dtype, DEVICE)
    model.load(inputs["w"])
    longest = max(n + b for n, b in zip(new, before))
    pages = sum((n + b + page - 1) // page + 1 for n, b in zip(new, before))
    storage = CacheStorage(model.cache_groups, page, pages, len(new), dtype, torch.device(DEVICE))
    manager = CacheManager(model.cache_groups, page, pages, len(new))
    step = StepFunction(model, storage, manager, longest, use_graphs=True)
    ids = [f"r{r}" for r in range(len(new))]
    for r, rid in enumerate(ids):
        manager.admit(rid)
        storage.reset_slot(manager.requests[rid].slot, 0.0, 1.0, 0, 0)
        if before[r]:
            manager.commit(manager.prepare([(rid, before[r])]))
            table = torch.tensor(manager.requests[rid].tables[0], device=DEVICE)
            for layer in range(case["layers"]):
                for pool, rows in zip((storage.key_pools[0], storage.value_pools[0]), inputs["old"][layer][r]):
                    pool[layer, table] = _pages_of(rows, len(table), page).transpose(1, 2)
    entries = [StepEntry(rid, t.tolist(), [len(t) - 1]) for rid, t in zip(ids, inputs["tokens"])]
    if max(new) == 1:
        step.graph_for(len(new))
    return dict(case=case, manager=manager, step=step, entries=entries, before=before,
                items=[(rid, n) for rid, n in zip(ids, new)])


def run(state):
    if state["case"]["kind"] == "model":
        manager = state["manager"]
        reservation = manager.prepare(state["items"])
        logits = state["step"].run(state["entries"], reservation)
        manager.commit(reservation)
        for (rid, _), length in zip(state["items"], state["before"]):
            manager.truncate(rid, length)          # the next pass is the same step again
        return [logits]
    if "graph" in state:
        state["graph"].replay()
        return [state["y"]] + state["outputs"]
    return [_forward(state, StepContext(**state["context"]))] + state["outputs"]


# --------------------------------------------------------------------------------------------------------------- work
def work(case):
    """Weights, new rows, caches and states each read once and outputs written once; the products and the sums of the definition
    (a causal row attends to what it sees; of the experts only those that can be chosen at most)."""
    new, before = _lens(case)
    n, size, width, kind = sum(new), 4 if case["dtype"] == "float32" else 2, case["width"], case["kind"]
    seen = sum(k * b + k * (k + 1) // 2 for k, b in zip(new, before))
    rows = 2 * n * width * size
    if kind == "mlp":
        weights = 3 * width * case["ff"]
        return {"bytes": weights * size + rows, "flops": 2 * n * weights}
    if kind == "experts":
        per = (2 if case["form"] == "relu_square" else 3) * width
        used = min(case["experts"], n * case["top"])
        return {"bytes": (used * per * case["expert_ff"] + per * case["shared"]) * size + 4 * case["experts"] * width + rows,
                "flops": 2 * n * (case["top"] * per * case["expert_ff"] + per * case["shared"] + case["experts"] * width)}
    heads, dim = case["heads"], case["dim"]
    if kind == "attention":
        kv = case["kv_heads"]
        weights = width * dim * (2 * heads + 2 * kv)
        return {"bytes": (weights + 2 * kv * dim * (sum(before) + 2 * n)) * size + rows, "flops": 2 * n * weights + 4 * heads * dim * seen}
    if kind == "latent":
        rank, rot, vdim = case["rank"], case["rot"], case["vdim"]
        weights = width * (heads * (dim + rot) + rank + rot + heads * vdim) + heads * rank * (dim + vdim)
        return {"bytes": (weights + (rank + rot) * (sum(before) + 2 * n)) * size + rows,
                "flops": 2 * n * weights + 2 * heads * (2 * rank + rot) * seen}
    if kind == "model":
        layer = width * dim * (2 * heads + 2 * case["kv_heads"]) + 3 * width * case["ff"]
        weights, out = case["layers"] * layer, case["vocab"] * width
        cache = case["layers"] * 2 * case["kv_heads"] * dim * (sum(before) + 2 * n)
        return {"bytes": (weights + out + cache) * size + 4 * len(new) * case["vocab"],
                "flops": 2 * n * weights + 2 * len(new) * out + 4 * case["layers"] * heads * dim * seen}
    state = 2 * 4 * _state_size(case) * len(new)
    if kind == "ssm":
        weights = width * (3 * heads * dim + 2 * case["groups"] * case["state"] + heads)
        scan = 6 * heads * dim * case["state"]
    else:
        vdim, qk = case["vdim"], case.get("kv_heads", heads)
        weights = width * (2 * qk * dim + 3 * heads * vdim)
        scan = (8 if kind == "delta" else 5) * heads * dim * vdim
    return {"bytes": weights * size + state + rows, "flops": n * (2 * weights + scan)}


def tolerance(case):
    """About four times the distance from ``exact`` that was measured: 0.003 to 0.005 for a layer in bfloat16 (one rounding of each
    intermediate, a few in a row), 0.011 for the logits of four layers, 2e-6 in float32.  The largest differences belong to entries
    whose sums nearly cancel."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-3}
    return {"rel": 3e-2 if case["kind"] == "model" else 1.5e-2, "max": 0.4}


# ---------------------------------------------------------------------------------------------------- the definitions
def _rms(x, weight=None):
    y = x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, positions):
    """Half-split rotation of the last dimension of [T, ..., d] by the rows' positions."""
    d = x.shape[-1]
    freq = THETA ** (-2.0 * torch.arange(d // 2, dtype=torch.float64, device=x.device) / d)
    angle = positions.double()[:, None] * freq
    angle = angle.view((x.shape[0],) + (1,) * (x.dim() - 2) + (d // 2,))
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def _softmax_mix(scores, seen, values, sink=None):
    """softmax over the seen keys of scores [H, T, K], with the sink as one more key without a value; values [H, K, dv]."""
    scores = scores.masked_fill(~seen, -math.inf)
    top = scores.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink.view(-1, 1, 1))
    p = torch.exp(scores - top)
    total = p.sum(-1, keepdim=True)
    if sink is not None:
        total = total + torch.exp(sink.view(-1, 1, 1) - top)
    return (p @ values) / total


def _seen(before, n):
    keys = torch.arange(before + n, device=DEVICE)
    return keys[None, :] <= (before + torch.arange(n, device=DEVICE))[:, None]


def _exact_attention(case, w, prefix, x, old):
    """Grouped-query attention of the step's rows x (float64, [N, width]) behind each request's old keys and values."""
    new, before = _lens(case)
    heads, kv, dim = case["heads"], case["kv_heads"], case["dim"]
    capped = case.get("form") == "capped"

    def project(name, count):
        y = x @ w[prefix + name + "_proj.weight"].T
        return (y + w[prefix + name + "_proj.weight.b"] if capped else y).view(-1, count, dim)

    q, k, v = project("q", heads), project("k", kv), project("v", kv)
    if not capped:
        q, k = _rms(q, w[prefix + "q_norm.weight"]), _rms(k, w[prefix + "k_norm.weight"])
    outputs, at = [], 0
    for n, b, (old_k, old_v) in zip(new, before, old):
        rows = slice(at, at + n)
        positions = b + torch.arange(n, device=DEVICE)
        keys = torch.cat([old_k.double(), _rotate(k[rows], positions)]).transpose(0, 1).repeat_interleave(heads // kv, 0)
        values = torch.cat([old_v.double(), v[rows]]).transpose(0, 1).repeat_interleave(heads // kv, 0)
        scores = _rotate(q[rows], positions).transpose(0, 1) @ keys.transpose(1, 2) * dim ** -0.5
        if capped:
            scores = SOFTCAP * torch.tanh(scores / SOFTCAP)
        outputs.append(_softmax_mix(scores, _seen(b, n), values, w["sink"] if capped else None).transpose(0, 1))
        at += n
    y = torch.cat(outputs)
    if capped:
        y = y * torch.sigmoid(x @ w["g_proj.weight"].T)[:, :, None]
    return y.reshape(x.shape[0], heads * dim) @ w[prefix + "o_proj.weight"].T


def _exact_latent(case, w, x, old):
    new, before = _lens(case)
    heads, dim, rot, vdim, rank = case["heads"], case["dim"], case["rot"], case["vdim"], case["rank"]
    q = (x @ w["q"].T).view(-1, heads, dim + rot)
    latent = x @ w["dkv"].T
    c, k_rot = _rms(latent[:, :rank], w["dkv.norm"]), latent[:, rank:]
    outputs, at = [], 0
    for n, b, rows_before in zip(new, before, old):
        rows = slice(at, at + n)
        positions = b + torch.arange(n, device=DEVICE)
        all_c = torch.cat([rows_before[:, :rank].double(), c[rows]])
        all_rot = torch.cat([rows_before[:, rank:].double(), _rotate(k_rot[rows], positions)])
        one = []
        for h in range(heads):         # head by head: the keys of all heads at once would be large
            keys = all_c @ w["uk"].view(heads, dim, rank)[h].T
            values = all_c @ w["uv"].view(heads, vdim, rank)[h].T
            scores = q[rows, h, :dim] @ keys.T + _rotate(q[rows, h, dim:], positions) @ all_rot.T
            one.append(_softmax_mix(scores[None] * (dim + rot) ** -0.5, _seen(b, n), values[None])[0])
        outputs.append(torch.stack(one, dim=1))
        at += n
    y = torch.cat(outputs) * torch.sigmoid(x @ w["g"].T)[:, :, None]
    return y.reshape(x.shape[0], heads * vdim) @ w["o"].T


def _exact_experts(case, w, x):
    form, top = case["form"], case["top"]

    def expert(rows, prefix):
        up = rows @ w[prefix + "up"].T
        if form == "relu_square":
            hidden = torch.relu(up) ** 2
        else:
            gate = rows @ w[prefix + "gate"].T
            if form == "silu_glu":
                hidden = _silu(gate) * up
            else:
                gate, up = gate.clamp(max=LIMIT), up.clamp(-LIMIT, LIMIT)
                hidden = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        return hidden @ w[prefix + "down"].T

    z = x @ w["router"].T
    if form == "relu_square":
        z = z + w["router.b"]
    chosen, ids = torch.sort(z, dim=-1, descending=True, stable=True)
    chosen, ids = chosen[:, :top], ids[:, :top]
    if form == "relu_square":
        weights = torch.softmax(chosen, dim=-1)
    elif form == "clamped_glu":
        weights = torch.softmax(z, dim=-1).gather(1, ids)
    else:
        weights = torch.sigmoid(chosen)
        weights = 2.5 * weights / (weights.sum(-1, keepdim=True) + 1e-20)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        token, place = torch.nonzero(ids == e, as_tuple=True)
        if token.numel():
            out.index_add_(0, token, weights[token, place][:, None] * expert(x[token], f"e{e}."))
    return out + expert(x, "shared.") if case["shared"] else out


def _conv(u, weight, bias, carried):
    """Causal convolution of u [T, C] behind the carried inputs [taps - 1, C], SiLU; and the inputs to carry on."""
    line = torch.cat([carried, u])
    y = sum(line[k:k + u.shape[0]] * weight[:, k] for k in range(TAPS))
    return _silu(y if bias is None else y + bias), line[-(TAPS - 1):]


def _exact_recurrence(case, w, x, states, slots):
    """(output rows, states afterwards): every request's tokens one after the other from the state in its slot."""
    kind, heads, dim = case["kind"], case["heads"], case["dim"]
    new, _ = _lens(case)
    states = states.double().clone()
    outputs, at = [], 0
    for r, n in enumerate(new):
        rows, slot = x[at:at + n], int(slots[r])
        y, states[slot] = _exact_request(case, w, rows, states[slot])
        outputs.append(y)
        at += n
    return torch.cat(outputs) @ w["o"].T, states


def _exact_request(case, w, x, state):
    kind, heads, dim, n = case["kind"], case["heads"], case["dim"], x.shape[0]
    if kind == "ssm":
        size, groups, inner = case["state"], case["groups"], heads * dim
        channels = inner + 2 * groups * size
        proj = x @ w["in"].T
        z, dt = proj[:, :inner], torch.nn.functional.softplus(proj[:, inner + channels:] + w["dt_bias"])
        conv, carried = _conv(proj[:, inner:inner + channels], w["conv"], w["conv.b"], state[:(TAPS - 1) * channels].view(TAPS - 1, channels))
        u = conv[:, :inner].view(n, heads, dim)
        b = conv[:, inner:inner + groups * size].view(n, groups, size).repeat_interleave(heads // groups, 1)
        c = conv[:, inner + groups * size:].view(n, groups, size).repeat_interleave(heads // groups, 1)
        keep = torch.exp(-torch.exp(w["A_log"]) * dt)
        s, y = state[(TAPS - 1) * channels:].view(heads, dim, size).clone(), []
        for t in range(n):
            s = keep[t, :, None, None] * s + (dt[t, :, None] * u[t])[:, :, None] * b[t, :, None, :]
            y.append((s @ c[t, :, :, None])[:, :, 0] + w["D"][:, None] * u[t])
        v = (torch.stack(y).reshape(n, inner) * _silu(z)).view(n, groups, inner // groups)
        return _rms(v).reshape(n, inner) * w["norm"], torch.cat([carried.reshape(-1), s.reshape(-1)])
    vdim, qk = case["vdim"], case.get("kv_heads", heads)
    q, k, v = x @ w["q"].T, x @ w["k"].T, x @ w["v"].T
    gate = x @ w["g"].T
    carried = None
    if kind == "delta":
        channels = 2 * qk * dim + heads * vdim
        weight = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]])
        conv, carried = _conv(torch.cat([q, k, v], dim=1), weight, None, state[:(TAPS - 1) * channels].view(TAPS - 1, channels))
        state = state[(TAPS - 1) * channels:]
        q, k, v = conv[:, :qk * dim], conv[:, qk * dim:2 * qk * dim], conv[:, 2 * qk * dim:]
    elif kind == "decay":
        q, k, v = _silu(q), _silu(k), _silu(v)
    q, k, v = q.view(n, qk, dim), k.view(n, qk, dim), v.view(n, heads, vdim)
    if kind == "delta":
        q, k = (part / torch.sqrt(part.pow(2).sum(-1, keepdim=True) + 1e-6) for part in (q, k))
        q, k = q.repeat_interleave(heads // qk, 1), k.repeat_interleave(heads // qk, 1)
        beta = torch.sigmoid(x @ w["b"].T)
        keep = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))
    if kind != "decay":
        q = q * dim ** -0.5
    y = []
    if kind == "memory":
        matrices = heads * (vdim + 1) * dim
        s, m = state[:matrices].view(heads, vdim + 1, dim).clone(), state[matrices:].clone()
        i = GATE_CAP * torch.tanh((x @ w["i"].T + w["i.b"]) / GATE_CAP)
        f = torch.nn.functional.logsigmoid(GATE_CAP * torch.tanh((x @ w["f"].T + w["f.b"]) / GATE_CAP))
        ones = torch.cat([v, torch.ones_like(v[:, :, :1])], dim=2)
        for t in range(n):
            top = torch.maximum(f[t] + m, i[t])
            s = torch.exp(f[t] + m - top)[:, None, None] * s + torch.exp(i[t] - top)[:, None, None] * ones[t, :, :, None] * k[t, :, None, :]
            m = top
            o = (s @ q[t, :, :, None])[:, :, 0]
            y.append(o[:, :vdim] / (torch.maximum(o[:, vdim].abs(), torch.exp(-m)) + 1e-6)[:, None])
        after = torch.cat([s.reshape(-1), m])
        return (_rms(torch.stack(y)).reshape(n, heads * vdim) * w["norm"]) * torch.sigmoid(gate), after
    s = state.view(heads, vdim, dim).clone()
    if kind == "decay":
        keep = torch.tensor(_decays(case), dtype=torch.float64, device=DEVICE).expand(n, heads)[:, :, None, None]
    elif kind == "gla":
        keep = torch.sigmoid(x @ w["a1"].T @ w["a2"].T + w["a2.b"]).pow(1.0 / TAU).view(n, heads, 1, dim)
    else:
        keep = keep[:, :, None, None]
    for t in range(n):
        s = keep[t] * s
        add = v[t]
        if kind == "delta":
            add = beta[t, :, None] * (v[t] - (s @ k[t, :, :, None])[:, :, 0])
        s = s + add[:, :, None] * k[t, :, None, :]
        y.append((s @ q[t, :, :, None])[:, :, 0])
    y = torch.stack(y)
    after = s.reshape(-1) if carried is None else torch.cat([carried.reshape(-1), s.reshape(-1)])
    if kind == "decay":
        return _rms(y.reshape(n, heads * vdim), w["norm"]) * torch.sigmoid(gate), after
    return _rms(y, w["norm"]).reshape(n, heads * vdim) * _silu(gate), after


def _exact_model(case, w, tokens, old):
    new, _ = _lens(case)
    stream = w["model.embed_tokens.weight"][torch.cat(tokens)]
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}."
        h = _rms(stream, w[p + "input_layernorm.weight"])
        stream = stream + _exact_attention(case, w, p + "self_attn.", h, old[layer])
        h = _rms(stream, w[p + "post_attention_layernorm.weight"])
        hidden = _silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)
        stream = stream + hidden @ w[p + "mlp.down_proj.weight"].T
    ends = torch.tensor(new, device=DEVICE).cumsum(0) - 1
    return _rms(stream[ends], w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T


def exact(case, seed):
    inputs = _inputs(case, seed)
    w = {name: tensor.double() for name, tensor in inputs["w"].items()}
    kind = case["kind"]
    if kind == "model":
        return [_exact_model(case, w, inputs["tokens"], inputs["old"])]
    x = inputs["x"].double()
    if kind == "mlp":
        return [(_silu(x @ w["gate_proj.weight"].T) * (x @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T]
    if kind == "experts":
        return [_exact_experts(case, w, x)]
    if kind == "attention":
        return [_exact_attention(case, w, "", x, inputs["old"]), None, None]
    if kind == "latent":
        return [_exact_latent(case, w, x, inputs["old"]), None]
    return list(_exact_recurrence(case, w, x, inputs["states"], inputs["slots"]))
