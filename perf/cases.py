"""The work that serving a model consists of, as cases that can be timed and compared.

A pass is a call or two of :class:`eredu_b200.runtime.engine.Engine` on one of four models, in the three forms in which requests
reach it:

* ``prefill``: whole prompts, from admission to the logits that choose their first tokens;
* ``turn``: some new tokens behind a context that is already cached - the next message of a chat, or a prompt whose beginning
  another request has brought;
* ``decode``: steps of a batch that is being decoded, one token per sequence and step, captured in a CUDA graph.

The models have the widths, heads, vocabularies and formats of the configurations in :mod:`eredu_b200.models.config`: Llama-3-8B,
Llama-3-70B with 4-bit weights (groups of 64), Qwen3-30B-A3B and the 16-layer draft model. All layers of a model are alike, so the
three large ones keep eight of them; the draft model is whole. Weights are random and made from the seed.
"""
from __future__ import annotations

import dataclasses
import random
from types import SimpleNamespace
from zlib import crc32

import torch

from eredu_b200.models import config
from eredu_b200.models.llama import build_from_tensors
from eredu_b200.models.moe import make_moe_factory
from eredu_b200.ops import SamplingParams
from eredu_b200.ops.quant import make_quantizer
from eredu_b200.runtime.engine import Engine

LAYERS = 8
MODELS = {
    "draft": config.draft_llama_16l(),
    "8b": dataclasses.replace(config.llama3_8b(), num_hidden_layers=LAYERS),
    "70b-4bit": dataclasses.replace(config.llama3_70b(), num_hidden_layers=LAYERS),
    "moe": dataclasses.replace(config.qwen3_30b_a3b(), num_hidden_layers=LAYERS),
}
BITS, GROUP = 4, 64
STEPS = 4           # decode steps of a pass
BUDGET = 128        # tokens a decoding request may still produce: its pages are reserved when it is admitted


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # speculative decoding's drafter between two verifications: the smallest steps there are
        dict(name="draft decode", model="draft", form="decode", batch=1, context=512, new=0),
        # one user, and a full decode batch, of the model most requests go to
        dict(name="8b decode 1", model="8b", form="decode", batch=1, context=2048, new=0),
        dict(name="8b decode 32", model="8b", form="decode", batch=32, context=2048, new=0),
        # time to the first token: one long prompt, and the short ones of all lengths that arrive together
        dict(name="8b prompt", model="8b", form="prefill", batch=1, context=0, new=2048),
        dict(name="8b prompts ragged", model="8b", form="prefill", batch=5, context=0, new=333),
        # the next message of a chat
        dict(name="8b turn", model="8b", form="turn", batch=1, context=4096, new=45),
        # the model that is served in 4 bits because of its size: one user, a small batch, a prompt
        dict(name="70b decode 1", model="70b-4bit", form="decode", batch=1, context=2048, new=0),
        dict(name="70b decode 8", model="70b-4bit", form="decode", batch=8, context=1024, new=0),
        dict(name="70b prompt", model="70b-4bit", form="prefill", batch=1, context=0, new=4096),
        # sparse experts: a token that reads 8 of 128 of them, a batch that reads nearly all, a prompt
        dict(name="moe decode 1", model="moe", form="decode", batch=1, context=1024, new=0),
        dict(name="moe decode 32", model="moe", form="decode", batch=32, context=1024, new=0),
        dict(name="moe prompt", model="moe", form="prefill", batch=1, context=0, new=1024),
    ]


# tokens of context over the batch, and of a batch of prompts: what a drawn case may cost
CONTEXT_TOKENS = {"draft": 65536, "8b": 65536, "70b-4bit": 16384, "moe": 32768}
PROMPT_TOKENS = {"draft": 8192, "8b": 8192, "70b-4bit": 4096, "moe": 8192}


def draw(rng):
    def spread(low, high):
        return min(high, int(low * (high / low) ** rng.random() + rng.random()))

    model, form = rng.choice(list(MODELS)), rng.choice(["decode", "decode", "prefill", "turn"])
    if form == "decode":
        batch = spread(1, 32)
        return dict(model=model, form=form, batch=batch, context=spread(16, min(8000, CONTEXT_TOKENS[model] // batch)), new=0)
    if form == "prefill":
        batch = spread(1, 8)
        return dict(model=model, form=form, batch=batch, context=0, new=spread(4, PROMPT_TOKENS[model] // batch))
    batch = spread(1, 4)
    return dict(model=model, form=form, batch=batch, context=spread(64, min(7600, CONTEXT_TOKENS[model] // batch)), new=spread(2, 384))


def lengths(case):
    """(cached tokens, new tokens) of every sequence: the first has as many as the case says, the others between half of that and all."""
    rng = random.Random(f"{case['batch']} {case['context']} {case['new']}")
    part = lambda n, first: n if first or n < 2 else rng.randint(n // 2, n)     # noqa: E731
    new = STEPS if case["form"] == "decode" else case["new"]
    return [(part(case["context"], i == 0), new if case["form"] == "decode" else part(new, i == 0)) for i in range(case["batch"])]


# ------------------------------------------------------------------------------------------ inputs
def tokens(case, seed):
    """Token ids of every sequence, cached ones first."""
    g = torch.Generator().manual_seed(seed)
    vocab = MODELS[case["model"]].vocab_size
    return [torch.randint(0, vocab, (old + new,), generator=g).tolist() for old, new in lengths(case)]


def shapes(cfg):
    H, D, V = cfg.hidden_size, cfg.head_dim, cfg.vocab_size
    out = {"model.embed_tokens.weight": (V, H), "model.norm.weight": (H,), "lm_head.weight": (V, H)}
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        out.update({p + "input_layernorm.weight": (H,), p + "post_attention_layernorm.weight": (H,),
                    p + "self_attn.q_proj.weight": (cfg.num_attention_heads * D, H),
                    p + "self_attn.k_proj.weight": (cfg.num_key_value_heads * D, H),
                    p + "self_attn.v_proj.weight": (cfg.num_key_value_heads * D, H),
                    p + "self_attn.o_proj.weight": (H, cfg.num_attention_heads * D)})
        if cfg.qk_norm:
            out.update({p + "self_attn.q_norm.weight": (D,), p + "self_attn.k_norm.weight": (D,)})
        if cfg.num_experts:
            E, I = cfg.num_experts, cfg.moe_intermediate_size
            out.update({p + "mlp.gate.weight": (E, H), p + "mlp.experts.gate_up_proj": (E, 2 * I, H), p + "mlp.experts.down_proj": (E, H, I)})
        else:
            I = cfg.intermediate_size
            out.update({p + "mlp.gate_proj.weight": (I, H), p + "mlp.up_proj.weight": (I, H), p + "mlp.down_proj.weight": (H, I)})
    return out


# Standard deviation of a matrix times the root of its input width. Attention then sees some of the cached tokens and not their average
# (scores of 2), the experts of a token weigh differently, and a layer adds a third of what is there to the stream, as in trained models.
GAINS = {"q_proj": 1.4, "k_proj": 1.4, "o_proj": 0.4, "gate": 4.0, "down_proj": 0.5}


def weights(cfg, seed):
    """``get(name)``: the bf16 tensor of that name on the GPU, the same one at every call; ``has(name)``."""
    table = shapes(cfg)

    def get(name):
        g = torch.Generator(device="cuda").manual_seed(seed * 1000003 + crc32(name.encode()))
        t = torch.randn(table[name], generator=g, dtype=torch.bfloat16, device="cuda")
        kind = name.removesuffix(".weight").rpartition(".")[2]
        if kind.endswith("norm"):
            return t.mul_(0.1).add_(1.4 if kind in ("q_norm", "k_norm") else 1.0)
        return t if kind == "embed_tokens" else t.mul_(GAINS.get(kind, 1.0) / table[name][-1] ** 0.5)

    return get, table.__contains__


# ------------------------------------------------------------------------------------------ passes
GREEDY = SamplingParams(temperature=0.0)


def prepare(case, seed):
    cfg = MODELS[case["model"]]
    quantizer = None
    if case["model"] == "70b-4bit":
        quantizer = make_quantizer(None, SimpleNamespace(quantization=SimpleNamespace(bits=BITS, group_size=GROUP, mode="affine"),
                                                         native_gguf=False))
    model = build_from_tensors(cfg, *weights(cfg, seed), "cuda", torch.bfloat16, moe_factory=make_moe_factory() if cfg.num_experts else None,
                               quantizer=quantizer)
    ids, sizes = tokens(case, seed), lengths(case)
    eng = Engine(model, max_batch=case["batch"], max_seq_len=max(len(t) for t in ids) + BUDGET, prefill_chunk=8192)
    state = {"case": case, "engine": eng, "ids": ids}
    # a decoded token's logits stay in the engine; a program that scores tokens looks at what the head returns
    head = model.logits

    def logits(*args, **kwargs):
        state["logits"] = head(*args, **kwargs)
        return state["logits"]

    model.logits = logits
    if case["form"] == "prefill":
        return state
    seqs = state["sequences"] = [eng.new_sequence(t[:old], GREEDY, max_new_tokens=BUDGET if case["form"] == "decode" else new)
                                 for t, (old, new) in zip(ids, sizes)]
    first = eng.prefill(seqs)
    if case["form"] == "turn":
        state["entries"] = [(s, t[old:], [new - 1]) for s, t, (old, new) in zip(seqs, ids, sizes)]
        return state
    eng.start_decode(seqs, first)
    decoding = eng._decode_state
    state["begin"] = {k: decoding[k].clone() for k in ("positions", "seq_lens", "slots", "rows")}
    # the tokens of each step are given, so that a pass does not hang on which of two nearly equal logits is the larger
    state["steps"] = [torch.tensor([t[old + i] for t, (old, _) in zip(ids, sizes)], dtype=torch.int32).pin_memory() for i in range(STEPS)]
    eng.decode_step(host_tokens=state["steps"][0], sync=False)      # captures the graph, as the first step of a batch does
    return state


def run(state):
    """Logits [sequences, vocabulary] behind the last token of every sequence. Those of a decode pass depend on its earlier steps through
    the keys and values that these have written."""
    eng, case = state["engine"], state["case"]
    if case["form"] == "prefill":
        seqs = [eng.new_sequence(t, GREEDY, max_new_tokens=BUDGET) for t in state["ids"]]
        eng.prefill(seqs)
        for s in seqs:
            eng.release(s)
        return state["logits"]
    if case["form"] == "turn":
        out = eng.forward_tokens(state["entries"])
        for s, new, _ in state["entries"]:
            s.kv_len -= len(new)        # back to where the message began
        return out
    for name, t in state["begin"].items():
        eng._decode_state[name].copy_(t)
    for step in state["steps"]:
        eng.decode_step(host_tokens=step, sync=False)
    return state["logits"]


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    cfg = MODELS[case["model"]]
    H, D, V, L = cfg.hidden_size, cfg.head_dim, cfg.vocab_size, cfg.num_hidden_layers
    nq, nkv, B = cfg.num_attention_heads, cfg.num_key_value_heads, case["batch"]
    attention = H * D * (2 * nq + 2 * nkv)
    size = BITS / 8 + 4 / GROUP if case["model"] == "70b-4bit" else 2
    spans, passes = lengths(case), STEPS if case["form"] == "decode" else 1
    bytes_ = flops = 0.0
    for step in range(passes):
        part = [(old + step, 1) for old, _ in spans] if case["form"] == "decode" else spans
        T = sum(new for _, new in part)
        if cfg.num_experts:
            expert, k, E = 3 * H * cfg.moe_intermediate_size, cfg.num_experts_per_tok, cfg.num_experts
            used, read = attention + k * expert + E * H, attention + E * H + E * (1 - (1 - k / E) ** T) * expert
        else:
            used = read = attention + 3 * H * cfg.intermediate_size
        cached = sum(old + new for old, new in part)
        pairs = sum(new * old + new * (new + 1) / 2 for old, new in part)
        flops += L * (2 * T * used + 4 * nq * D * pairs) + 2 * B * V * H
        bytes_ += L * (read * size + 4 * nkv * D * cached) + 2 * V * H + 2 * T * H + 4 * B * V
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # bf16 activations through 8 or 16 layers are 0.008 to 0.017 from exact() (2-norm over the logits)
    return {"rel": 0.03, "max": 0.2}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def affine(w):
    """The numbers that 4 bits keep of ``w``, group by group: multiples of a bf16 scale from a bf16 extreme on, zero among them."""
    x = w.float().view(w.shape[0], -1, GROUP)
    low, high = x.amin(-1), x.amax(-1)
    bins = 2 ** BITS - 1
    scale = ((high - low) / bins).clamp_min(1e-7)
    scale = torch.where(low.abs() > high.abs(), scale, -scale)
    edge = torch.where(low.abs() > high.abs(), low, high)
    zero = torch.round(edge / scale)
    scale = torch.where(zero != 0, edge / zero.where(zero != 0, torch.ones_like(zero)), scale).bfloat16().float()[..., None]
    base = torch.where(zero == 0, torch.zeros_like(edge), edge).bfloat16().float()[..., None]
    code = torch.round((x - base) / scale).clamp(0, bins)
    return (code.double() * scale.double() + base.double()).view(w.shape)


def exact(case, seed):
    cfg = MODELS[case["model"]]
    get, _ = weights(cfg, seed)
    ids = tokens(case, seed)
    H, D, L = cfg.hidden_size, cfg.head_dim, cfg.num_hidden_layers
    nq, nkv = cfg.num_attention_heads, cfg.num_key_value_heads
    count = [len(t) for t in ids]
    start = [sum(count[:i]) for i in range(len(ids))]
    at = torch.cat([torch.arange(n) for n in count]).cuda().double()
    angle = at[:, None] * torch.tensor([cfg.rope_theta ** (-2 * i / D) for i in range(D // 2)], dtype=torch.float64, device="cuda")
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def matrix(name):
        w = get(name)
        return affine(w) if case["model"] == "70b-4bit" else w.double()

    def norm(x, name):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.rms_norm_eps) * get(name).double()

    def turned(x):
        a, b = x.chunk(2, -1)
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    def feed(x, p):
        if not cfg.num_experts:
            gate, up, down = (matrix(p + f"mlp.{n}_proj.weight") for n in ("gate", "up", "down"))
            return torch.cat([(torch.nn.functional.silu(part @ gate.t()) * (part @ up.t())) @ down.t() for part in x.split(8192)])
        top, which = torch.topk(torch.softmax(x @ matrix(p + "mlp.gate.weight").t(), -1), cfg.num_experts_per_tok)
        top = top / top.sum(-1, keepdim=True)
        gate_up, down = get(p + "mlp.experts.gate_up_proj"), get(p + "mlp.experts.down_proj")
        out = torch.zeros_like(x)
        for e in range(cfg.num_experts):
            row, k = (which == e).nonzero(as_tuple=True)
            gate, up = (x[row] @ gate_up[e].double().t()).chunk(2, -1)
            out.index_add_(0, row, top[row, k, None] * ((torch.nn.functional.silu(gate) * up) @ down[e].double().t()))
        return out

    table = get("model.embed_tokens.weight")
    h = torch.cat([table[torch.tensor(t, device="cuda")] for t in ids]).double()
    del table
    last = torch.tensor([s + n - 1 for s, n in zip(start, count)], device="cuda")
    for i in range(L):
        p = f"model.layers.{i}."
        x = norm(h, p + "input_layernorm.weight")
        q, k, v = ((x @ matrix(p + f"self_attn.{n}_proj.weight").t()).view(len(x), -1, D) for n in "qkv")
        if cfg.qk_norm:
            q, k = norm(q, p + "self_attn.q_norm.weight"), norm(k, p + "self_attn.k_norm.weight")
        q, k = turned(q), turned(k)
        mixed = torch.empty_like(q)
        for s, n in zip(start, count):
            for head in range(nkv):
                key, value = k[s:s + n, head], v[s:s + n, head]
                mine = slice(head * (nq // nkv), (head + 1) * (nq // nkv))
                for a in range(0, n, 1024):
                    b = min(n, a + 1024)
                    score = q[s + a:s + b, mine].transpose(0, 1) @ key[:b].t() / D ** 0.5
                    late = torch.arange(b, device="cuda") > torch.arange(a, b, device="cuda")[:, None]
                    mixed[s + a:s + b, mine] = (torch.softmax(score.masked_fill(late, float("-inf")), -1) @ value[:b]).transpose(0, 1)
        mixed = mixed.view(len(x), -1)
        if i == L - 1:
            mixed, h = mixed[last], h[last]
        h = h + mixed @ matrix(p + "self_attn.o_proj.weight").t()
        h = h + feed(norm(h, p + "post_attention_layernorm.weight"), p)
    return norm(h, "model.norm.weight") @ get("lm_head.weight").double().t()
