"""What the framework is timed on: a whole model that serves requests, and the layers its decoders are made of, each through
the entry point a program calls (`Engine.step`; a registered part's `forward` on a step and its cache lines).

The ranges: layers of the widths 2,048, 3,072 and 4,096 that the presets and `bench.py` use (and some odd ones), prompts of 1 to
4 sequences with together 16 to about 2,700 tokens, decoding with 1 to 64 sequences over 100 to 3,000 cached positions, head
sizes from 48 to 128 lanes, bfloat16 and, for the dense decoder's layers, the 32-bit path.

A layer case is a dict: "kind" names the part, "lengths" the new tokens of every sequence, "cached" how many positions every
sequence holds already, the rest are the part's sizes.  Its outputs are the part's output and the cache lines it has written.
"""
import math

import torch

from burn_lm_b200.config.presets import preset
from burn_lm_b200.engine.engine import Engine, StepEntry, Workspace
from burn_lm_b200.model import Model, plan_of
from burn_lm_b200.cache.cache import CacheView
from burn_lm_b200.parts.base import Runtime, StepContext
from burn_lm_b200.parts.attention import AttentionSpec
from burn_lm_b200.parts.feed_forward import SwiGLUSpec
from burn_lm_b200.parts.gated_delta import GatedDeltaSpec
from burn_lm_b200.parts.hgrn2 import Hgrn2Spec
from burn_lm_b200.parts.latent_attention import LatentAttentionSpec
from burn_lm_b200.parts.mamba2 import Mamba2Spec
from burn_lm_b200.parts.moe import RoutedMoESpec
from burn_lm_b200.parts.position import RotarySpec
from burn_lm_b200.parts.sigmoid_attention import SigmoidAttentionSpec
from burn_lm_b200.parts.sink_attention import SinkAttentionSpec
from burn_lm_b200.parts.wkv import WkvSpec
from burn_lm_b200.plan import PartPlan
from burn_lm_b200.registry import part_class

PAGE = 64
EPS = 1e-6
DEV = "cuda"


# ---- the cases -----------------------------------------------------------------------------------------------------------
def listed():
    return [
        # a batch of eight chats on the 1B decoder: their prompts in one step, then 24 tokens each (the headline workload)
        dict(name="requests_1b", kind="requests", preset="llama3_2_1b", seqs=8, prompt=512, steps=24),
        # one layer's feed-forward for eight decoding sequences: the smallest call there is
        dict(name="swiglu_decode8", kind="swiglu", width=2048, inner=8192, lengths="1x8", cached=512, dtype="bfloat16"),
        # the 32-bit path (what the trace runner's --dtype float32 serves): a prompt through a feed-forward
        dict(name="swiglu_float32", kind="swiglu", width=2048, inner=8192, lengths="317", cached=0, dtype="float32"),
        # the dense decoder's attention over a packed batch of unequal prompts
        dict(name="attention_prompts", kind="attention", width=2048, heads=32, kv=8, dim=64, lengths="1000,611,37,400", cached=0, dtype="bfloat16"),
        # windowed attention with kept first tokens and a sink, a prompt longer than the window (8B-sized layer)
        dict(name="sink_prompt", kind="sink", width=4096, heads=32, kv=8, dim=128, vdim=128, window=1024, keep=64, lengths="2048", cached=0),
        # attention without a softmax whose heads are mixed: a prompt, and decoding a full batch
        dict(name="sigmoid_prompt", kind="sigmoid", width=2048, heads=32, kv=8, dim=64, vdim=64, lengths="1536", cached=0),
        dict(name="sigmoid_decode", kind="sigmoid", width=2048, heads=32, kv=8, dim=64, vdim=64, lengths="1x64", cached=1087),
        # the recurrent mixers' prompts: a state-space scan, the gated delta rule over two prompts, a decay per key channel
        dict(name="mamba2_prompt", kind="mamba2", width=2048, heads=64, vdim=64, state=128, groups=8, lengths="2048", cached=0),
        dict(name="delta_prompts", kind="delta", width=2048, heads=16, qk_heads=8, dim=128, vdim=128, lengths="1501,500", cached=0),
        dict(name="wkv_prompt", kind="wkv", width=4096, heads=32, dim=128, lengths="2048", cached=0),
        # attention over a cached latent, decoding with long contexts
        dict(name="latent_decode", kind="latent", width=4096, heads=32, dim=64, rot=64, vdim=128, rank=512, lengths="1x32", cached=2500),
        # a prompt through a mixture of gated experts
        dict(name="experts_prompt", kind="experts", width=2048, inner=4096, experts=8, top=2, lengths="1800", cached=0),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _prompts(rng, most):
    """Lengths of one to four prompts of together at most `most` tokens."""
    total, n = _spread(rng, 16, most), rng.choice((1, 1, 2, 3, 4))
    cuts = sorted(rng.randint(1, max(1, total - 1)) for _ in range(n - 1))
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]) if b > a)


def draw(rng):
    kind = rng.choice(("swiglu", "attention", "sink", "sigmoid", "mamba2", "delta", "wkv", "hgrn2", "latent", "experts", "requests"))
    if kind == "requests":
        return dict(kind=kind, preset="llama3_2_1b", seqs=rng.choice((1, 2, 3, 5, 8)), prompt=_spread(rng, 16, 500), steps=rng.randint(4, 20))
    width = rng.choice((2048, 2048, 3072, 4096, 1536, 2304))
    if rng.random() < 0.6:
        case = dict(kind=kind, width=width, lengths=_prompts(rng, 2700), cached=0)
    else:
        case = dict(kind=kind, width=width, lengths="1x%d" % _spread(rng, 1, 64), cached=_spread(rng, 100, 3000))
    heads = width // 64
    if kind == "swiglu":
        case.update(inner=8 * rng.randint(width // 4, width // 2), dtype=rng.choice(("bfloat16", "bfloat16", "float32")))
        if case["dtype"] == "float32":
            case["lengths"] = str(_spread(rng, 1, 600))
            case["cached"] = 0
    elif kind == "attention":
        case.update(heads=24 if width == 3072 else 32, kv=8, dim=128 if width >= 3072 else 64, dtype="bfloat16")
    elif kind == "sink":
        case.update(heads=32, kv=rng.choice((4, 8)), dim=rng.choice((64, 96, 128)), vdim=rng.choice((64, 80, 128)),
                    window=rng.choice((256, 1000, 1024, 2048)), keep=rng.choice((0, 4, 64, 70)))
    elif kind == "sigmoid":
        case.update(heads=rng.choice((16, 24, 32)), kv=8, dim=rng.choice((48, 64, 128)), vdim=rng.choice((64, 128)))
    elif kind == "mamba2":
        case.update(heads=heads, vdim=64, state=rng.choice((64, 100, 128)), groups=rng.choice((1, 4)))
    elif kind == "delta":
        case.update(heads=16, qk_heads=rng.choice((8, 16)), dim=rng.choice((64, 100, 128)), vdim=rng.choice((64, 96, 128)))
    elif kind == "wkv":
        case.update(heads=heads, dim=64) if rng.random() < 0.5 else case.update(heads=width // 128, dim=128)
    elif kind == "hgrn2":
        case.update(heads=width // 128, dim=rng.choice((64, 128)), vdim=rng.choice((64, 128)))
    elif kind == "latent":
        case.update(heads=rng.choice((16, 32)), dim=64, rot=rng.choice((32, 64)), vdim=rng.choice((64, 128)), rank=rng.choice((256, 384, 512)))
    elif kind == "experts":
        case.update(width=min(width, 2304), inner=8 * rng.randint(128, 512), experts=rng.choice((6, 8, 16)), top=2)
    return case


# ---- what a case is made of ----------------------------------------------------------------------------------------------
def _lengths(case):
    parts = [p.split("x") for p in case["lengths"].split(",")]         # "500,37" or "1x64": 64 sequences of one token
    return [int(p[0]) for p in parts for _ in range(int(p[1]) if len(p) > 1 else 1)]


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


class _Draws:
    """Tensors one after another from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed * 7919 + 11)

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.float32):
        t = torch.empty(shape, dtype=torch.float32, device=DEV)
        return t.normal_(mean, std, generator=self.g).to(dtype)

    def uniform(self, shape, lo, hi):
        return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=self.g)

    def matrix(self, rows, cols, dtype=torch.bfloat16):
        return self.normal((rows, cols), std=cols ** -0.5, dtype=dtype)


def _weights(case, d):
    """The part's stored tensors by role, bfloat16 matrices with rows of about unit gain and 32-bit vectors."""
    c, kind, w = case, case["kind"], case["width"]
    if kind == "swiglu":
        return dict(gate=d.matrix(c["inner"], w), up=d.matrix(c["inner"], w), down=d.matrix(w, c["inner"]))
    if kind == "attention":
        q, kv = c["heads"] * c["dim"], c["kv"] * c["dim"]
        return dict(q=d.matrix(q, w), k=d.matrix(kv, w), v=d.matrix(kv, w), o=d.matrix(w, q))
    if kind == "sink":
        q, k, v, o = c["heads"] * c["dim"], c["kv"] * c["dim"], c["kv"] * c["vdim"], c["heads"] * c["vdim"]
        return dict(q=d.matrix(q, w), k=d.matrix(k, w), v=d.matrix(v, w), o=d.matrix(w, o), g=d.matrix(c["heads"], w),
                    q_norm=d.normal((q,), 0.1, 1.0), k_norm=d.normal((k,), 0.1, 1.0))
    if kind == "sigmoid":
        q, k, v, o = c["heads"] * c["dim"], c["kv"] * c["dim"], c["kv"] * c["vdim"], c["heads"] * c["vdim"]
        return dict(q=d.matrix(q, w), k=d.matrix(k, w), v=d.matrix(v, w), o=d.matrix(w, o), q_bias=d.normal((q,), 0.1),
                    k_bias=d.normal((k,), 0.1), v_bias=d.normal((v,), 0.1), talk=d.normal((c["heads"], c["heads"]), c["heads"] ** -0.5),
                    head_bias=d.normal((c["heads"],), 1.0, -3.0))
    if kind == "mamba2":
        inner, gn = c["heads"] * c["vdim"], c["groups"] * c["state"]
        dt = torch.exp(d.uniform((c["heads"],), math.log(0.001), math.log(0.1)))        # the steps state-space layers start from
        return dict({"in": d.matrix(2 * inner + 2 * gn + c["heads"], w)}, conv=d.normal((inner + 2 * gn, 4), 0.5),
                    conv_bias=d.normal((inner + 2 * gn,), 0.1), dt_bias=torch.log(torch.expm1(dt)),
                    A_log=torch.log(d.uniform((c["heads"],), 1.0, 16.0)), D=d.normal((c["heads"],), 0.1, 1.0),
                    norm=d.normal((inner,), 0.1, 1.0), o=d.matrix(w, inner))
    if kind == "delta":
        qk, vw, rank = c["qk_heads"] * c["dim"], c["heads"] * c["vdim"], 128
        return dict(q=d.matrix(qk, w), k=d.matrix(qk, w), v=d.matrix(vw, w), b=d.matrix(c["heads"], w), q_conv=d.normal((qk, 4), 0.5),
                    k_conv=d.normal((qk, 4), 0.5), v_conv=d.normal((vw, 4), 0.5), A_log=d.normal((c["heads"],), 0.5),
                    norm=d.normal((c["vdim"],), 0.1, 1.0), a1=d.matrix(rank, w), a2=d.matrix(c["heads"] * c["dim"], rank),
                    dt_bias=d.normal((c["heads"] * c["dim"],), 1.0, -3.0), g1=d.matrix(rank, w), g2=d.matrix(vw, rank), o=d.matrix(w, vw))
    if kind == "wkv":
        hk, rank = c["heads"] * c["dim"], 64
        mus = {"mu_" + m: d.uniform((w,), 0.0, 1.0) for m in "rkvgw"}
        return dict(mus, r=d.matrix(hk, w), k=d.matrix(hk, w), v=d.matrix(hk, w), g=d.matrix(hk, w), w1=d.matrix(rank, w),
                    w2=d.matrix(hk, rank), w0=d.uniform((hk,), -6.0, 0.0), u=d.normal((c["heads"], c["dim"]), 0.5),
                    norm=d.normal((hk,), 0.1, 1.0), o=d.matrix(w, hk))
    if kind == "hgrn2":
        kw, vw = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        return dict(q=d.matrix(kw, w), f=d.matrix(kw, w), f_bias=d.normal((kw,), 1.0), lower=d.uniform((kw,), 0.0, 0.97),
                    v=d.matrix(vw, w), norm=d.normal((c["vdim"],), 0.1, 1.0), o=d.matrix(w, vw))
    if kind == "latent":
        q, vw = c["heads"] * (c["dim"] + c["rot"]), c["heads"] * c["vdim"]
        return dict(q=d.matrix(q, w), dkv=d.matrix(c["rank"] + c["rot"], w), c_norm=d.normal((c["rank"],), 0.1, 1.0),
                    uk=d.matrix(c["heads"] * c["dim"], c["rank"]), uv=d.matrix(vw, c["rank"]), g=d.matrix(vw, w), o=d.matrix(w, vw))
    if kind == "experts":
        out = dict(router=d.matrix(c["experts"], w, torch.float32) * 2.0)
        for e in range(c["experts"]):
            out.update({f"gate{e}": d.matrix(c["inner"], w), f"up{e}": d.matrix(c["inner"], w), f"down{e}": d.matrix(w, c["inner"])})
        return out
    raise ValueError(kind)


def _spec(c):
    w, kind = c["width"], c["kind"]
    if kind == "swiglu":
        return "feed_forward", "swiglu", SwiGLUSpec(w, c["inner"])
    if kind == "attention":
        return "mixer", "attention", AttentionSpec(w, c["heads"], c["kv"], c["dim"], PartPlan("rotary", RotarySpec(c["dim"], 500000.0)))
    if kind == "sink":
        return "mixer", "sink_attention", SinkAttentionSpec(w, c["heads"], c["kv"], c["dim"], c["vdim"], c["dim"] ** -0.5, c["window"], c["keep"],
                                                            qk_norm_eps=EPS)
    if kind == "sigmoid":
        return "mixer", "sigmoid_attention", SigmoidAttentionSpec(w, c["heads"], c["kv"], c["dim"], c["vdim"], c["dim"] ** -0.5, softcap=30.0,
                                                                  rotary_dim=c["dim"], rotary_base=500000.0)
    if kind == "mamba2":
        return "mixer", "mamba2", Mamba2Spec(w, c["heads"], c["vdim"], c["state"], c["groups"], 4, c["groups"], EPS)
    if kind == "delta":
        return "mixer", "gated_delta", GatedDeltaSpec(w, c["heads"], c["qk_heads"], c["dim"], c["vdim"], 4, EPS)
    if kind == "wkv":
        return "mixer", "wkv", WkvSpec(w, c["heads"], c["dim"], EPS)
    if kind == "hgrn2":
        return "mixer", "hgrn2", Hgrn2Spec(w, c["heads"], c["dim"], c["vdim"], EPS)
    if kind == "latent":
        return "mixer", "latent_attention", LatentAttentionSpec(w, c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"], (c["dim"] + c["rot"]) ** -0.5,
                                                                c["rot"], 500000.0, EPS)
    if kind == "experts":
        return "feed_forward", "routed_moe", RoutedMoESpec(w, c["experts"], c["top"], c["inner"], correction=False)
    raise ValueError(kind)


def _state_rows(n):
    """Rows of a recurrent state as it lies in the cache: eight row groups times a power of two."""
    rn = 1
    while 8 * rn < n:
        rn *= 2
    return 8 * rn


def _state_sizes(c):
    """(floats of the carried inputs, heads, rows, columns) of a recurrent part's state."""
    kind = c["kind"]
    if kind == "mamba2":
        return 3 * (c["heads"] * c["vdim"] + 2 * c["groups"] * c["state"]), c["heads"], c["state"], c["vdim"]
    if kind == "delta":
        return 3 * (2 * c["qk_heads"] * c["dim"] + c["heads"] * c["vdim"]), c["heads"], c["dim"], c["vdim"]
    if kind == "wkv":
        return c["width"], c["heads"], c["dim"], c["dim"]
    return 0, c["heads"], c["dim"], c["vdim"]


def _lines(c, d):
    """The cache lines of a case as its sequences hold them: (pool, block table, state).  Pages of 64 positions in a shuffled
    order: a page's keys [kv head][64][lanes], then its values; for a latent [64][lanes].  States twice a sequence, the copy
    chosen by whether the position is even."""
    lens, kind = _lengths(c), c["kind"]
    pool = table = state = None
    if kind in ("attention", "sink", "sigmoid", "latent"):
        each = -(-(c["cached"] + max(lens)) // PAGE)
        n = each * len(lens)
        g = torch.Generator()
        g.manual_seed(n)
        table = torch.randperm(n, generator=g).to(torch.int32).reshape(len(lens), each).to(DEV)
        if kind == "latent":
            shape = (n, PAGE, c["rank"] + c["rot"])
        elif c.get("vdim", c["dim"]) == c["dim"]:
            shape = (n, 2, c["kv"], PAGE, c["dim"])
        else:
            shape = (n, c["kv"] * PAGE * (c["dim"] + c["vdim"]))
        pool = d.normal(shape, dtype=_dtype(c)) if c["cached"] else torch.zeros(shape, dtype=_dtype(c), device=DEV)
    elif kind in ("mamba2", "delta", "wkv", "hgrn2"):
        hist, heads, rows, cols = _state_sizes(c)
        padded = _state_rows(rows)
        state = torch.zeros((len(lens), 2, hist + heads * padded * cols), dtype=torch.float32, device=DEV)
        if c["cached"]:
            state[:, :, :hist] = d.normal((len(lens), 2, hist))
            lanes = state[:, :, hist:].view(len(lens), 2, heads, padded // 8, cols, 8)
            lanes.copy_(d.normal(tuple(lanes.shape), 0.3))
            row = torch.arange(padded, device=DEV).view(padded // 8, 1, 8)
            lanes *= (row < rows)
    return pool, table, state


def _rows(c, d):
    """The layer's input rows: what a norm in front of it gives."""
    n = sum(_lengths(c))
    return d.normal((n, c["width"]), dtype=torch.float32 if c["kind"] == "wkv" else _dtype(c))


def _step(c):
    lens, cached = _lengths(c), c["cached"]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return StepContext(
        n_tokens=cu[-1], n_seqs=len(lens), max_q_len=max(lens), max_kv_len=cached + max(lens), tokens=i32([0] * cu[-1]),
        token_seq=i32([s for s, n in enumerate(lens) for _ in range(n)]), token_pos=i32([cached + t for n in lens for t in range(n)]),
        cu_seqlens=i32(cu), slot_of_seq=i32(list(range(len(lens)))), start_pos=i32([cached] * len(lens)), want_rows=None, n_want=0,
        workspace=Workspace(torch.device(DEV)))


def _part(c, weights):
    family, kind, spec = _spec(c)
    cls = part_class(family, kind)
    names = {r: r for r in cls.roles}
    if c["kind"] == "experts":
        names.update(gate="gate{}", up="up{}", down="down{}")
    dt = _dtype(c)
    part = cls(spec, names, Runtime(dt, torch.device(DEV)))
    part.bind({k: v.to(dt) if v.dtype == torch.bfloat16 else v for k, v in weights.items()})
    if hasattr(part, "prepare"):
        part.prepare(-(-(c["cached"] + max(_lengths(c))) // PAGE) * PAGE)
    return part


def prepare(case, seed):
    if case["kind"] == "requests":
        seqs, prompt, steps = case["seqs"], case["prompt"], case["steps"]
        _, _, plan = plan_of(preset(case["preset"]))
        model = Model(plan, Runtime(torch.bfloat16, torch.device(DEV)))
        model.bind(_request_weights(preset(case["preset"]), seed))
        engine = Engine(model, seqs * (-(-(prompt + steps) // PAGE) * PAGE), max_seqs=seqs, max_seq_len=prompt + steps)
        prompts, fed = _request_tokens(case, seed, engine.vocab_size)
        return dict(case=case, engine=engine, prompts=prompts, fed=fed)
    d = _Draws(seed)
    weights = _weights(case, d)
    x = _rows(case, d)
    pool, table, state = _lines(case, d)
    view = CacheView("kv" if pool is not None else "state", True, pool=pool, block_table=table, state=state,
                     window=case.get("window"), keep_first=case.get("keep", 0))
    return dict(case=case, part=_part(case, weights), x=x, step=_step(case), view=view)


def _request_tokens(case, seed, vocab):
    """(prompts, the tokens fed after them step by step): what a recorded conversation brings."""
    g = torch.Generator()
    g.manual_seed(seed)
    t = torch.randint(0, vocab, (case["seqs"], case["prompt"] + case["steps"]), generator=g).tolist()
    return [r[:case["prompt"]] for r in t], [[r[case["prompt"] + i] for r in t] for i in range(case["steps"])]


def _request_weights(p, seed):
    """The dense decoder's stored tensors by name, bfloat16 N(0, 0.02) as its presets are benchmarked with."""
    d, w = _Draws(seed), p["hidden_size"]
    q, kv, inner = p["num_attention_heads"] * p["head_dim"], p["num_key_value_heads"] * p["head_dim"], p["intermediate_size"]
    m = lambda rows, cols: d.normal((rows, cols), 0.02, dtype=torch.bfloat16)
    norm = lambda: d.normal((w,), 0.1, 1.0, dtype=torch.bfloat16)
    out = {"model.embed_tokens.weight": m(p["vocab_size"], w), "model.norm.weight": norm()}
    for i in range(p["num_hidden_layers"]):
        at = f"model.layers.{i}."
        out.update({at + "input_layernorm.weight": norm(), at + "post_attention_layernorm.weight": norm(),
                    at + "self_attn.q_proj.weight": m(q, w), at + "self_attn.k_proj.weight": m(kv, w),
                    at + "self_attn.v_proj.weight": m(kv, w), at + "self_attn.o_proj.weight": m(w, q),
                    at + "mlp.gate_proj.weight": m(inner, w), at + "mlp.up_proj.weight": m(inner, w),
                    at + "mlp.down_proj.weight": m(w, inner)})
    return out


def run(state):
    if "engine" in state:
        # a batch of requests from its prompts to its last token: a logits row for every token that was asked for
        engine = state["engine"]
        slots = [engine.acquire() for _ in state["prompts"]]
        out = [engine.step([StepEntry(s, p, (len(p) - 1,)) for s, p in zip(slots, state["prompts"])])]
        for tokens in state["fed"]:
            out.append(engine.step([StepEntry(s, (t,), (0,)) for s, t in zip(slots, tokens)]).clone())
        for s in slots:
            engine.release(s)
        return out
    part, step, view = state["part"], state["step"], state["view"]
    step.memo.clear()
    if part.family == "feed_forward":
        return [part.forward(state["x"], step)]
    out = part.forward(state["x"], step, view)
    return [out, view.pool if view.pool is not None else view.state]


# ---- the least a pass can do ---------------------------------------------------------------------------------------------
def _pairs(c):
    """(query, key) pairs that are seen."""
    total = 0
    for n in _lengths(c):
        for i in range(c["cached"], c["cached"] + n):
            seen = i + 1
            if "window" in c:
                seen = min(seen, c["window"] + c["keep"])
            total += seen
    return total


def work(case):
    c, kind = case, case["kind"]
    if kind == "requests":
        p = preset(c["preset"])
        w, layers, kvw = p["hidden_size"], p["num_hidden_layers"], p["num_key_value_heads"] * p["head_dim"]
        layer = 2 * w * w + 2 * w * kvw + 3 * w * p["intermediate_size"]
        head, tokens = w * p["vocab_size"], c["seqs"] * c["prompt"]
        kv = 4 * layers * kvw
        after = c["seqs"] * c["steps"]
        cached = c["seqs"] * sum(c["prompt"] + t for t in range(c["steps"]))
        logits = 4 * p["vocab_size"] * c["seqs"] * (c["steps"] + 1)
        pairs = c["seqs"] * c["prompt"] * (c["prompt"] + 1) / 2 + cached
        return {"bytes": 2 * (layers * layer + head) * (c["steps"] + 1) + kv * (tokens + after + cached) + logits,
                "flops": 2.0 * layers * layer * (tokens + after) + 2.0 * head * (after + c["seqs"]) + 4.0 * layers * w * pairs}
    n, w = sum(_lengths(c)), c["width"]
    size = 4 if _dtype(c) == torch.float32 else 2
    if kind == "swiglu":
        m = 3 * w * c["inner"]
        return {"bytes": size * (m + 2 * n * w), "flops": 2.0 * n * m}
    if kind == "experts":
        m, used = 3 * w * c["inner"], min(c["experts"], n * c["top"])
        return {"bytes": 2 * (used * m + n * w) + 4 * (c["experts"] * w + n * w), "flops": 2.0 * n * (c["top"] * m + c["experts"] * w)}
    if kind in ("attention", "sink", "sigmoid"):
        vd = c.get("vdim", c["dim"])
        m = w * (c["heads"] * (c["dim"] + vd) + c["kv"] * (c["dim"] + vd) + (c["heads"] if kind == "sink" else 0))
        seen = sum(min(c["cached"] + k, c.get("window", 1 << 30) + k + c.get("keep", 0)) for k in _lengths(c))
        mix = 2.0 * c["heads"] ** 2 if kind == "sigmoid" else 0.0
        return {"bytes": 2 * (m + n * w + seen * c["kv"] * (c["dim"] + vd)) + (4 if kind == "sigmoid" else 2) * n * w,
                "flops": 2.0 * n * m + _pairs(c) * (2.0 * c["heads"] * (c["dim"] + vd) + mix)}
    if kind == "latent":
        lanes = c["rank"] + c["rot"]
        m = w * (c["heads"] * (c["dim"] + c["rot"] + 2 * c["vdim"]) + lanes)
        up = c["heads"] * c["rank"] * (c["dim"] + c["vdim"])
        seen = sum(c["cached"] + k for k in _lengths(c))
        if max(_lengths(c)) == 1:
            attend = 2.0 * n * up + _pairs(c) * 2.0 * c["heads"] * (lanes + c["rank"])
        else:
            attend = 2.0 * seen * up + _pairs(c) * 2.0 * c["heads"] * (c["dim"] + c["rot"] + c["vdim"])
        return {"bytes": 2 * (m + up + n * w + seen * lanes) + 4 * n * w, "flops": 2.0 * n * m + attend}
    hist, heads, rows, cols = _state_sizes(c)
    width = sum(t.numel() for k, t in _weight_shapes(c).items() if len(t.shape) == 2 and min(t.shape) > 4)
    states = 4 * len(_lengths(c)) * (hist + heads * rows * cols) * (2 if c["cached"] else 1)
    ops = {"mamba2": 4.0, "delta": 6.0, "wkv": 4.0, "hgrn2": 4.0}[kind]
    return {"bytes": 2 * width + (4 if kind == "wkv" else 2) * n * w + 4 * n * w + states, "flops": 2.0 * n * width + ops * n * heads * rows * cols}


class _Shapes:
    """Stands in for _Draws where only the shapes are wanted."""

    def normal(self, shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.empty(shape, device="meta")

    def uniform(self, shape, lo, hi):
        return torch.empty(shape, device="meta")

    def matrix(self, rows, cols, dtype=torch.bfloat16):
        return torch.empty((rows, cols), device="meta")


def _weight_shapes(c):
    return _weights(c, _Shapes())


def tolerance(case):
    """About four times what is seen against `exact`: 0.0016 to 0.004 from the rounding of 16-bit operands and outputs, 2e-6
    from 32-bit sums, and 0.017 to 0.02 where a whole model carries the former through sixteen layers."""
    if case["kind"] == "requests":
        return {"rel": 7e-2, "max": 0.5}
    if case.get("dtype") == "float32":
        return {"rel": 8e-6, "max": 8e-5}
    return {"rel": 1.5e-2, "max": 0.15}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------
def _rotate(x, pos, dims, base, halves=True):
    """x [n, heads, lanes]: the first `dims` lanes turn, lane i with lane i + dims / 2 (or neighbours)."""
    half = dims // 2
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(half)], dtype=torch.float64, device=DEV)
    a = pos.to(torch.float64)[:, None, None] * f
    co, si = torch.cos(a), torch.sin(a)
    out = x.clone()
    u, v = (x[..., :half], x[..., half:dims]) if halves else (x[..., 0:dims:2], x[..., 1:dims:2])
    one, two = (slice(0, half), slice(half, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., one] = u * co - v * si
    out[..., two] = v * co + u * si
    return out


def _unit(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(x):
    return x * torch.sigmoid(x)


def _paged(pool, table, c, lanes_k, lanes_v, heads):
    """float64 views of the pages: (keys [pages, heads, 64, lanes_k], values)."""
    flat = pool.to(torch.float64).reshape(pool.shape[0], -1)
    k = flat[:, :heads * PAGE * lanes_k].view(-1, heads, PAGE, lanes_k)
    v = flat[:, heads * PAGE * lanes_k:].view(-1, heads, PAGE, lanes_v) if lanes_v else None
    return flat, k, v


def _bounds(c):
    at, out = 0, []
    for s, n in enumerate(_lengths(c)):
        out.append((s, at, n))
        at += n
    return out


def _exact_attention(c, w, x, pool, table):
    kind, H, G, dk = c["kind"], c["heads"], c["kv"], c["dim"]
    dv = c.get("vdim", dk)
    pos = torch.cat([torch.arange(c["cached"], c["cached"] + n, device=DEV) for n in _lengths(c)])
    q, k, v = x @ w["q"].T, x @ w["k"].T, x @ w["v"].T
    if kind == "sigmoid":
        q, k, v = q + w["q_bias"], k + w["k_bias"], v + w["v_bias"]
    if kind == "sink":
        q, k = _unit(q) * w["q_norm"], _unit(k) * w["k_norm"]
    q, k, v = q.view(-1, H, dk), k.view(-1, G, dk), v.view(-1, G, dv)
    if kind != "sink":
        q, k = _rotate(q, pos, dk, 500000.0), _rotate(k, pos, dk, 500000.0)
    stored = slice(None)
    if kind == "attention" and _dtype(c) == torch.bfloat16:
        # the dense decoder keeps a head's lanes in groups of eight, each followed by its partners of the rotation
        half = dk // 2
        stored = torch.tensor([(8 * (p // 16) + p % 16) if p % 16 < 8 else (half + 8 * (p // 16) + p % 16 - 8) for p in range(dk)], device=DEV)
        q, k = q[..., stored], k[..., stored]
    flat, pk, pv = _paged(pool, table, c, dk, dv, G)
    for s, at, n in _bounds(c):
        p = pos[at:at + n]
        pages = table[s, (p // PAGE)].long()
        pk[pages, :, p % PAGE] = k[at:at + n]
        pv[pages, :, p % PAGE] = v[at:at + n]
    out = torch.empty((x.shape[0], H, dv), dtype=torch.float64, device=DEV)
    scale = dk ** -0.5
    for s, at, n in _bounds(c):
        total = c["cached"] + n
        pages = table[s, :-(-total // PAGE)].long()
        keys = pk[pages].transpose(1, 2).reshape(-1, G, dk)[:total]
        vals = pv[pages].transpose(1, 2).reshape(-1, G, dv)[:total]
        for lo in range(0, n, 256):                      # some query rows at a time
            hi = min(n, lo + 256)
            qs, i = q[at + lo:at + hi], pos[at + lo:at + hi, None]
            j = torch.arange(total, device=DEV)[None, :]
            seen = j <= i
            if kind == "sink":
                seen = seen & ((i - j < c["window"]) | (j < c["keep"]))
            sc = torch.einsum("ngpd,tgd->gpnt", qs.view(-1, G, H // G, dk), keys).reshape(H, hi - lo, total) * scale
            if kind == "sigmoid":
                wt = torch.where(seen, torch.sigmoid(30.0 * torch.tanh(sc / 30.0) + w["head_bias"][:, None, None]), 0.0)
                wt = torch.einsum("hg,gnt->hnt", w["talk"], wt)
            else:
                sc = torch.where(seen, sc, -math.inf)
                if kind == "sink":
                    m = torch.clamp(sc.amax(-1, keepdim=True), min=0.0)
                    e = torch.exp(sc - m)
                    wt = e / (torch.exp(-m) + e.sum(-1, keepdim=True))
                else:
                    wt = torch.softmax(sc, -1)
            out[at + lo:at + hi] = torch.einsum("gpnt,tgd->ngpd", wt.view(G, H // G, hi - lo, total), vals).reshape(hi - lo, H, dv)
    if kind == "sink":
        out = out * torch.sigmoid(x @ w["g"].T)[:, :, None]
    return [out.reshape(-1, H * dv) @ w["o"].T, flat.view(pool.shape)]


def _exact_latent(c, w, x, pool, table):
    H, dk, dr, dv, R = c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"]
    pos = torch.cat([torch.arange(c["cached"], c["cached"] + n, device=DEV) for n in _lengths(c)])
    q, down = (x @ w["q"].T).view(-1, H, dk + dr), x @ w["dkv"].T
    lat = _unit(down[:, :R]) * w["c_norm"]
    kr = _rotate(down[:, None, R:], pos, dr, 500000.0, halves=False)[:, 0]
    qr = _rotate(q[..., dk:], pos, dr, 500000.0, halves=False)
    flat = pool.to(torch.float64)
    for s, at, n in _bounds(c):
        p = pos[at:at + n]
        flat[table[s, p // PAGE].long(), p % PAGE] = torch.cat([lat, kr], 1)[at:at + n]
    uk, uv = w["uk"].view(H, dk, R), w["uv"].view(H, dv, R)
    ql = torch.einsum("nhd,hdr->nhr", q[..., :dk], uk)
    out = torch.empty((x.shape[0], H, dv), dtype=torch.float64, device=DEV)
    for s, at, n in _bounds(c):
        total = c["cached"] + n
        rows = flat[table[s, :-(-total // PAGE)].long()].reshape(-1, R + dr)[:total]
        for lo in range(0, n, 256):
            hi = min(n, lo + 256)
            sl = slice(at + lo, at + hi)
            sc = (torch.einsum("nhr,tr->hnt", ql[sl], rows[:, :R]) + torch.einsum("nhr,tr->hnt", qr[sl], rows[:, R:])) * (dk + dr) ** -0.5
            seen = torch.arange(total, device=DEV)[None, :] <= pos[sl, None]
            p = torch.softmax(torch.where(seen, sc, -math.inf), -1)
            out[sl] = torch.einsum("hnr,hdr->nhd", torch.einsum("hnt,tr->hnr", p, rows[:, :R]), uv)
    out = out.reshape(-1, H * dv) * torch.sigmoid(x @ w["g"].T)
    return [out @ w["o"].T, flat]


def _convolved(rows, taps, carried):
    """silu-less causal convolution of one sequence's rows behind its carried inputs."""
    k = taps.shape[1]
    padded = torch.cat([carried, rows])
    return sum(padded[j:j + rows.shape[0]] * taps[:, j] for j in range(k)), padded[rows.shape[0]:]


def _exact_recurrent(c, w, x, state):
    kind, (hist, H, R, V) = c["kind"], _state_sizes(c)
    padded, start = _state_rows(R), c["cached"]
    new = state.to(torch.float64)
    lens = _lengths(c)
    n_most = max(lens)
    qs, ks, vs, decays, betas, gates = [], [], [], [], [], []
    for s, at, n in _bounds(c):
        rows, end = x[at:at + n], (start + n) & 1
        carried = new[s, start & 1, :hist].clone()
        if kind == "mamba2":
            inner, gn, G = H * V, c["groups"] * R, c["groups"]
            p = rows @ w["in"].T
            xbc, left = _convolved(p[:, inner:2 * inner + 2 * gn], w["conv"], carried.view(3, -1))
            xbc = _silu(xbc + w["conv_bias"])
            dt = torch.nn.functional.softplus(p[:, 2 * inner + 2 * gn:] + w["dt_bias"])
            per = H // G
            ks.append(xbc[:, inner:inner + gn].view(n, G, R).repeat_interleave(per, 1) * dt[..., None])
            qs.append(xbc[:, inner + gn:].view(n, G, R).repeat_interleave(per, 1))
            vs.append(xbc[:, :inner].view(n, H, V))
            decays.append(torch.exp(-torch.exp(w["A_log"]) * dt)[..., None].expand(n, H, R))
            gates.append(p[:, :inner])
        elif kind == "delta":
            qk, per = c["qk_heads"] * R, H // c["qk_heads"]
            taps = torch.cat([w["q_conv"], w["k_conv"], w["v_conv"]])
            cv, left = _convolved(torch.cat([rows @ w["q"].T, rows @ w["k"].T, rows @ w["v"].T], 1), taps, carried.view(3, -1))
            cv = _silu(cv)
            one = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
            qs.append(one(cv[:, :qk].view(n, -1, R)).repeat_interleave(per, 1) * R ** -0.5)
            ks.append(one(cv[:, qk:2 * qk].view(n, -1, R)).repeat_interleave(per, 1))
            vs.append(cv[:, 2 * qk:].view(n, H, V))
            betas.append(torch.sigmoid(rows @ w["b"].T))
            a = ((rows @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(n, H, R)
            decays.append(torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a)))
            gates.append((rows @ w["g1"].T) @ w["g2"].T)
        elif kind == "wkv":
            prev = torch.cat([carried[None], rows[:-1]])
            mix = {m: rows + (prev - rows) * w["mu_" + m] for m in "rkvgw"}
            left = rows[-1]
            qs.append((mix["r"] @ w["r"].T).view(n, H, R))
            ks.append((mix["k"] @ w["k"].T).view(n, H, R))
            vs.append((mix["v"] @ w["v"].T).view(n, H, V))
            decays.append(torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["w1"].T) @ w["w2"].T + w["w0"])).view(n, H, R))
            gates.append(mix["g"] @ w["g"].T)
        else:
            f = w["lower"] + (1.0 - w["lower"]) * torch.sigmoid(rows @ w["f"].T + w["f_bias"])
            qs.append(_silu(rows @ w["q"].T).view(n, H, R))
            decays.append(f.view(n, H, R))
            ks.append(1.0 - decays[-1])
            vs.append((rows @ w["v"].T).view(n, H, V))
            left = carried
        new[s, end, :hist] = left.reshape(-1)
    # all sequences walk together, token by token (S [sequences, heads, rows, columns])
    pad = lambda ts, fill=0.0: torch.stack([torch.nn.functional.pad(t, (0,) * (2 * t.dim() - 1) + (n_most - t.shape[0],), value=fill) for t in ts], 1)
    live = torch.tensor([[t < n for n in lens] for t in range(n_most)], device=DEV)
    q, k, v, dec = pad(qs), pad(ks), pad(vs), pad([d.contiguous() for d in decays], 1.0)
    beta = pad(betas) if betas else None
    lanes = new[:, :, hist:].view(len(lens), 2, H, padded // 8, V, 8)
    S = lanes[:, start & 1].permute(0, 1, 2, 4, 3).reshape(len(lens), H, padded, V)[:, :, :R].clone()
    if start == 0:
        S.zero_()
    y = torch.empty((n_most, len(lens), H, V), dtype=torch.float64, device=DEV)
    u = w["u"].double() if kind == "wkv" else None
    for t in range(n_most):
        if kind == "wkv":
            kv = k[t][..., None] * v[t][:, :, None]
            y[t] = torch.einsum("shrv,shr->shv", S + u[..., None] * kv, q[t])
            S = dec[t][..., None] * S + kv
        else:
            S = dec[t][..., None] * S
            add = v[t] if beta is None else beta[t][..., None] * (v[t] - torch.einsum("shrv,shr->shv", S, k[t]))
            S = S + k[t][..., None] * add[:, :, None]
            y[t] = torch.einsum("shrv,shr->shv", S, q[t])
    S = torch.nn.functional.pad(S, (0, 0, 0, padded - R)).view(len(lens), H, padded // 8, 8, V).permute(0, 1, 2, 4, 3)
    for s, n in enumerate(lens):
        lanes[s, (start + n) & 1] = S[s]
    del live
    o = torch.cat([y[:n, s] for s, n in enumerate(lens)])
    gate = torch.cat(gates) if gates else None
    flat = o.reshape(-1, H * V)
    if kind == "mamba2":
        flat = (flat + (torch.cat(vs) * w["D"][:, None]).reshape(-1, H * V)) * _silu(gate)
        flat = _unit(flat.view(flat.shape[0], c["groups"], -1)).reshape(-1, H * V) * w["norm"]
    elif kind == "delta":
        flat = (_unit(o) * w["norm"]).reshape(-1, H * V) * torch.sigmoid(gate)
    elif kind == "wkv":
        flat = _unit(o).reshape(-1, H * V) * w["norm"] * _silu(gate)
    else:
        flat = (_unit(o) * w["norm"]).reshape(-1, H * V)
    return [flat @ w["o"].T, new]


def _exact_experts(c, w, x):
    s = torch.softmax(x @ w["router"].T, -1)
    top, ids = torch.topk(s, c["top"], -1)
    top = top / (top.sum(-1, keepdim=True) + 1e-20)
    out = torch.zeros_like(x)
    for e in range(c["experts"]):
        row, place = (ids == e).nonzero(as_tuple=True)
        h = x[row]
        out[row] += top[row, place][:, None] * ((_silu(h @ w[f"gate{e}"].double().T) * (h @ w[f"up{e}"].double().T)) @ w[f"down{e}"].double().T)
    return [out]


def _exact_requests(case, seed):
    """The dense decoder over whole sequences, every logits row a request asks for."""
    p = preset(case["preset"])
    w = _request_weights(p, seed)
    prompts, fed = _request_tokens(case, seed, p["vocab_size"])
    H, G, dk = p["num_attention_heads"], p["num_key_value_heads"], p["head_dim"]
    tokens = torch.tensor([a + [f[s] for f in fed] for s, a in enumerate(prompts)], device=DEV)
    B, T = tokens.shape
    pos = torch.arange(T, device=DEV)
    rs, half = p["rope_scaling"], dk // 2
    freq = []
    for i in range(half):
        f = p["rope_theta"] ** (-2.0 * i / dk)
        turn, orig = 2.0 * math.pi / f, rs["original_max_position_embeddings"]
        if turn > orig / rs["low_freq_factor"]:
            f = f / rs["factor"]
        elif turn >= orig / rs["high_freq_factor"]:
            a = (orig / turn - rs["low_freq_factor"]) / (rs["high_freq_factor"] - rs["low_freq_factor"])
            f = (1.0 - a) * f / rs["factor"] + a * f
        freq.append(f)
    ang = pos.double()[:, None] * torch.tensor(freq, dtype=torch.float64, device=DEV)
    co, si = torch.cos(ang)[None, :, None], torch.sin(ang)[None, :, None]
    turned = lambda t: torch.cat([t[..., :half] * co - t[..., half:] * si, t[..., half:] * co + t[..., :half] * si], -1)
    rms = lambda t, g: t / torch.sqrt((t * t).mean(-1, keepdim=True) + p["rms_norm_eps"]) * g.double()
    x = w["model.embed_tokens.weight"].double()[tokens]
    seen = pos[None, :] <= pos[:, None]
    for i in range(p["num_hidden_layers"]):
        m = lambda name, h: h @ w[f"model.layers.{i}.{name}.weight"].double().T
        h = rms(x, w[f"model.layers.{i}.input_layernorm.weight"])
        q = turned(m("self_attn.q_proj", h).view(B, T, H, dk))
        k = turned(m("self_attn.k_proj", h).view(B, T, G, dk)).repeat_interleave(H // G, 2)
        v = m("self_attn.v_proj", h).view(B, T, G, dk).repeat_interleave(H // G, 2)
        o = torch.empty((B, T, H, dk), dtype=torch.float64, device=DEV)
        for b in range(B):
            sc = torch.einsum("thd,shd->hts", q[b], k[b]) * dk ** -0.5
            o[b] = torch.einsum("hts,shd->thd", torch.softmax(torch.where(seen, sc, -math.inf), -1), v[b])
        x = x + m("self_attn.o_proj", o.reshape(B, T, H * dk))
        h = rms(x, w[f"model.layers.{i}.post_attention_layernorm.weight"])
        x = x + m("mlp.down_proj", _silu(m("mlp.gate_proj", h)) * m("mlp.up_proj", h))
    h = rms(x[:, case["prompt"] - 1:], w["model.norm.weight"])
    table = w["model.embed_tokens.weight"]
    logits = torch.cat([h @ table[lo:lo + 16384].double().T for lo in range(0, table.shape[0], 16384)], -1)
    return [logits[:, t] for t in range(case["steps"] + 1)]


def exact(case, seed):
    if case["kind"] == "requests":
        return _exact_requests(case, seed)
    d = _Draws(seed)
    weights = _weights(case, d)
    x = _rows(case, d).double()
    pool, table, state = _lines(case, d)
    w = weights if case["kind"] == "experts" else {k: v.double() for k, v in weights.items()}
    if case["kind"] == "experts":
        w = dict(weights, router=weights["router"].double())
        return _exact_experts(case, w, x)
    if case["kind"] == "swiglu":
        return [(_silu(x @ w["gate"].T) * (x @ w["up"].T)) @ w["down"].T]
    if case["kind"] == "latent":
        return _exact_latent(case, w, x, pool, table)
    if state is not None:
        return _exact_recurrent(case, w, x, state)
    return _exact_attention(case, w, x, pool, table)
