"""Workloads that the engine's speed is judged by.

A case is a model (the widths of the presets, fewer layers where layers repeat), how the engine is called, and sizes:

  call "generate"  Engine.generate: every row decodes `new` tokens behind its prompt, one captured step per token.  run() is
                   the retry of a call that prepare() made: agents resubmit identical prompts up to two times, so a dense
                   model finds the prompts' pages in its prefix cache and computes the part of a page that is left; layer
                   stacks keep no prefix and compute the prompts again.  Rows are forced through given tokens, so that every
                   pass runs every row to the end over the same tokens whatever its random logits favour: a dense model's under
                   the game's vote grammar through "{" and blanks, which it allows without end, a stack's through tokens of
                   their own (rows choose experts of their own).
  call "replay"    Engine.open / step / close_sequence: `join` sequences are admitted per step (0: all at once), prompts
                   come in portions of at most `portion` tokens (0: whole) beside the single tokens of the sequences that
                   are through, `new` of them each.  Logits are wanted behind the
                   last `want` tokens of a prompt's last portion, and behind single tokens.

Prompts are ragged, 0.8 to 1.2 times `prompt`.  Weights, prompts and fed tokens come from the seed.  Matrices are
N(0, 1 / inputs), those that write to the residual stream smaller by sqrt(2 * layers), so that a stream of unit size passes
through layers which each change a part of it, as in a trained model.
"""
import dataclasses
import math

import numpy as np
import torch

from byzantine_consensus_llm_agents_b200 import model as M
from byzantine_consensus_llm_agents_b200 import stack as S
from byzantine_consensus_llm_agents_b200.engine import Engine, Request
from byzantine_consensus_llm_agents_b200.tokenizer import get_tokenizer

PAGE = 16
STACK_VOCAB = 32768
VOTE = {"type": "object", "properties": {"decision": {"type": "string", "enum": ["stop", "continue"]}},
        "required": ["decision"], "additionalProperties": False}
# layer stacks at widths of 1-2B and 8B class models; feed-forwards that make a layer a dense model's size
STACKS = {
    "bekopel-2k": lambda n: S.bekopel_preset("bekopel-2k", n, 2048, 7424, STACK_VOCAB, heads=16),
    "bekopel-4k": lambda n: S.bekopel_preset("bekopel-4k", n, 4096, 14592, STACK_VOCAB),
    "lerazen-2k": lambda n: S.lerazen_preset("lerazen-2k", n, 2048, 9216, STACK_VOCAB, heads=16),
    "lerazen-2k-experts": lambda n: S.lerazen_preset("lerazen-2k-experts", n, 2048, 9216, STACK_VOCAB, heads=16, experts=64, top=8,
                                                     expert_ff=768),
    "merulorn-2k": lambda n: S.merulorn_preset("merulorn-2k", n, 2048, 11520, STACK_VOCAB, heads=16),
    "merulorn-4k": lambda n: S.merulorn_preset("merulorn-4k", n, 4096, 23680, STACK_VOCAB),
    "vosolorn-2k": lambda n: S.vosolorn_preset("vosolorn-2k", n, 2048, 5632, STACK_VOCAB, heads=16),
    "vosolorn-2k-experts": lambda n: S.vosolorn_preset("vosolorn-2k-experts", n, 2048, 5632, STACK_VOCAB, heads=16, experts=64, top=8,
                                                       expert_ff=960),
}


def _case(name, model, layers, call, rows, prompt, new, portion=0, join=0, want=1, dtype="bfloat16"):
    return dict(name=name, model=model, layers=layers, call=call, rows=rows, prompt=prompt, new=new, portion=portion, join=join,
                want=want, dtype=dtype)


def listed():
    return [
        # one agent asks again (the reference's sequential retries) on the smallest preset: launches and latency
        _case("agent-0.6b", "qwen3-0.6b", 28, "generate", 1, 700, 48),
        # the headline game: ten agents' call on the default model's layers
        _case("agents-14b", "qwen3-14b", 6, "generate", 10, 1650, 48),
        # the agent-count sweep's largest step
        _case("agents-8b-64", "qwen3-8b", 6, "generate", 64, 900, 24),
        # the first prompts of a round in one launch
        _case("prompts-14b", "qwen3-14b", 4, "replay", 7, 1770, 0),
        # sequences that arrive one by one, prompts in portions, single tokens beside them: the step interface as served
        _case("portions-8b", "qwen3-8b", 6, "replay", 6, 700, 3, portion=256, join=1),
        # prompts of each layer-stack design, many and one at a time
        _case("bekopel-prompts", "bekopel-2k", 8, "replay", 8, 1536, 0, want=16),
        _case("lerazen-experts-prompts", "lerazen-2k-experts", 4, "replay", 5, 1300, 0, want=16),
        _case("merulorn-one-prompt", "merulorn-2k", 8, "replay", 1, 2999, 1, portion=2048, want=16),
        # calls of each design, prompts and decoding together
        _case("bekopel-call", "bekopel-2k", 8, "generate", 8, 500, 64),
        _case("merulorn-call", "merulorn-2k", 8, "generate", 8, 1024, 64),
        _case("vosolorn-experts-call", "vosolorn-2k-experts", 4, "generate", 32, 300, 48),
        # replay in float32, the mode for comparing logits
        _case("lerazen-float32", "lerazen-2k", 4, "replay", 2, 410, 2, dtype="float32"),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["dense", "dense", "dense", "stack", "stack", "stack", "stack", "float32"])
    if kind == "float32":
        return _draw("lerazen-2k", 4, "replay", log(1, 4), log(40, 400), rng.randint(0, 3), 0, 0, 4, "float32")
    if kind == "dense":
        model, layers = rng.choice([("qwen3-0.6b", 28), ("qwen3-8b", 6), ("qwen3-14b", 4), ("mistral-22b", 3)])
    else:
        model, layers = rng.choice([("bekopel-2k", 8), ("bekopel-4k", 4), ("lerazen-2k", 8), ("lerazen-2k-experts", 4), ("merulorn-2k", 8),
                                    ("merulorn-4k", 4), ("vosolorn-2k", 8), ("vosolorn-2k-experts", 4)])
    if rng.random() < 0.5:
        rows = log(1, 64)
        most = (40000 if kind == "dense" else 10000) // rows
        return _draw(model, layers, "generate", rows, log(60, min(1700, most)), log(12, 48), 0, 0, 1, "bfloat16")
    rows = log(1, 8)
    prompt = log(100, min(3000, 11000 // rows))
    portion = rng.choice([0, log(60, prompt)])
    return _draw(model, layers, "replay", rows, prompt, rng.randint(0, 4), max(portion, prompt // 12) if portion else 0, rng.choice([0, 1, 2]),
                 1 if kind == "dense" else 16, "bfloat16")


def _draw(*a):
    c = _case("", *a[:6], portion=a[6], join=a[7], want=a[8], dtype=a[9])
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------ the work of a pass
def _config(case):
    if case["model"] in STACKS:
        return dataclasses.replace(STACKS[case["model"]](case["layers"]), act_dtype=case["dtype"], max_pos=4096)
    return dataclasses.replace(M.PRESETS[case["model"]], n_layers=case["layers"], max_pos=4096)


def _lengths(case):
    return [max(1, int(case["prompt"] * (0.8 + 0.4 * ((i + 1) * 0.618034 % 1.0)))) for i in range(case["rows"])]


def _schedule(case):
    """Steps of a replay: lists of (row, first token, tokens, how many of the last ones' logits are wanted)."""
    lens, at, steps = _lengths(case), [0] * case["rows"], []
    ends = [n + case["new"] for n in lens]
    while any(a < e for a, e in zip(at, ends)):
        step = []
        for r in range(case["rows"]):
            if at[r] == ends[r] or case["join"] and r >= case["join"] * (len(steps) + 1):
                continue
            n = 1 if at[r] >= lens[r] else min(case["portion"] or lens[r], lens[r] - at[r])
            step.append((r, at[r], n, min(n, case["want"]) if at[r] + n >= lens[r] else 0))
            at[r] += n
        steps.append(step)
    return steps


def _passes(case):
    """What a pass computes, launch by launch: lists of (row, first token, tokens, wanted)."""
    if case["call"] == "replay":
        return _schedule(case)
    lens = _lengths(case)
    keep = [(n - 1) // PAGE * PAGE if case["model"] not in STACKS else 0 for n in lens]
    return [[(r, k, n - k, 1) for r, (n, k) in enumerate(zip(lens, keep))]] + \
        [[(r, n + t, 1, 1) for r, n in enumerate(lens)] for t in range(case["new"] - 1)]


def _dense_shapes(c):
    d, hd, out = c.d_model, c.head_dim, {"model.embed_tokens.weight": (c.vocab, c.d_model), "model.norm.weight": (c.d_model,)}
    if not c.tie_embeddings:
        out["lm_head.weight"] = (c.vocab, d)
    for i in range(c.n_layers):
        shapes = {"input_layernorm": (d,), "post_attention_layernorm": (d,), "self_attn.q_proj": (c.n_heads * hd, d),
                  "self_attn.k_proj": (c.n_kv_heads * hd, d), "self_attn.v_proj": (c.n_kv_heads * hd, d),
                  "self_attn.o_proj": (d, c.n_heads * hd), "mlp.gate_proj": (c.d_ff, d), "mlp.up_proj": (c.d_ff, d),
                  "mlp.down_proj": (d, c.d_ff)}
        if c.qk_norm:
            shapes.update({"self_attn.q_norm": (hd,), "self_attn.k_norm": (hd,)})
        out.update({f"model.layers.{i}.{n}.weight": s for n, s in shapes.items()})
    return out


def _shapes(cfg):
    return cfg.tensor_shapes() if isinstance(cfg, S.StackConfig) else _dense_shapes(cfg)


def work(case):
    cfg, steps = _config(case), _passes(case)
    stack, size = isinstance(cfg, S.StackConfig), 4 if case["dtype"] == "float32" else 2
    matrices = [(n, s[0] * s[1]) for n, s in _shapes(cfg).items() if len(s) == 2 and not n.startswith(("embed", "pos", "head", "model.emb",
                                                                                                       "lm_head"))]
    plain = sum(k for n, k in matrices if ".mlp.e" not in n)
    experts = sum(k for n, k in matrices if ".mlp.e" in n)
    moe = next((l.mlp for l in cfg.layers if isinstance(l.mlp, S.MoeMlp)), None) if stack else None
    share = moe.top / moe.experts if moe else 0.0
    if stack:       # (window, blocks of, query-key and value products of a pair of tokens, cached numbers of a token) of attention layers
        att = []
        for m in cfg.mixers(S.LatentAttention, S.GroupedAttention):
            row = m.cache_row if isinstance(m, S.LatentAttention) else m.kv_heads * (m.dim + m.vdim)
            att.append((m.window, getattr(m, "pool", 0), m.heads * (m.dim + getattr(m, "rot_dim", 0) + m.vdim), row))
        state = cfg.state_bytes_per_row
        recur = sum(m.heads * m.dim * m.dim * 9 for m in cfg.mixers(S.GeneralDelta)) + \
            sum(m.heads * m.vdim * m.state * 6 for m in cfg.mixers(S.StateSpace)) + \
            sum(m.heads * m.vdim * m.dim * 6 for m in cfg.mixers(S.MatrixMemory))
    else:
        att = [(0, 0, 2 * cfg.n_heads * cfg.head_dim, 2 * cfg.n_kv_heads * cfg.head_dim)] * cfg.n_layers
        state = recur = 0
    nbytes = flops = 0.0
    for step in steps:
        T, want = sum(e[2] for e in step), sum(e[3] for e in step)
        used = 1.0 - (1.0 - share) ** T if moe else 0.0
        nbytes += 2.0 * (plain + used * experts) + (2.0 * cfg.vocab * cfg.d_model if want else 0) + want * cfg.vocab * 4.0
        flops += 2.0 * T * (plain + share * experts + recur / 2) + 2.0 * want * cfg.vocab * cfg.d_model
        for _, a, n, _ in step:
            nbytes += 2.0 * state
            for window, pool, pair, row in att:
                seen = lambda p: min(p, window or p) + (max(0, p - window) // pool if pool else 0)
                nbytes += size * row * (seen(a + n) + n)
                flops += 2.0 * pair * n * (seen(a + 1) + seen(a + n)) / 2
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------ inputs
def _tensors(cfg, seed):
    """The checkpoint, name -> tensor on the GPU: bf16 matrices, fp32 vectors."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    stack = isinstance(cfg, S.StackConfig)
    out = {}
    for n, s in _shapes(cfg).items():
        leaf = n.rsplit(".", 1)[-1]
        noise = lambda std, mean=0.0: torch.empty(s, device="cuda").normal_(mean, std, generator=g)
        if len(s) == 2 and leaf != "conv":
            std = s[1] ** -0.5
            if n in ("embed", "pos", "model.embed_tokens.weight"):
                std = 1.0 / cfg.embed_scale if stack else 1.0
                std *= 0.3 if n == "pos" else 1.0
            if leaf == "router":        # a choice that is clear, and experts that together change the stream less than a feed-forward does
                std *= 2.0
            if ".mlp.e" in n and leaf == "down":
                std /= 8.0
            if leaf in ("o", "down") or n.endswith(("o_proj.weight", "down_proj.weight")):
                std *= (2 * cfg.n_layers) ** -0.5
            out[n] = torch.empty(s, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)
        elif leaf == "act":
            out[n] = torch.tensor([1.0, 0.5, 0.25, 0.0], device="cuda") + noise(0.05)
        elif leaf == "vmix":
            out[n] = torch.tensor(0.5, device="cuda")
        elif leaf == "conv":
            out[n] = noise(s[1] ** -0.5)
        elif leaf == "dt_bias":         # steps around 0.02
            out[n] = noise(0.5, -4.0)
        elif leaf == "A_log":           # decay rates around 1 to 8
            out[n] = noise(0.7, 1.0)
        elif leaf == "w0":              # channels that forget at once and channels that hardly forget
            out[n] = noise(2.0, -3.0)
        elif n.endswith(".f.b"):        # memories of a few dozen tokens and more
            out[n] = torch.linspace(3.0, 6.0, s[0], device="cuda")
        elif n.endswith(("ls1", "ls2", "norm1b", "norm2b")):      # what a sublayer's output is scaled by
            out[n] = noise(0.05, 0.3)
        elif "norm" in n:
            offset = cfg.norm_offset if stack and ".mix." not in n else 0.0
            out[n] = noise(0.1, 1.0 - offset)
        else:                           # biases, sinks, skips
            out[n] = noise(0.1, 1.0 if leaf == "D" else 0.0)
    return out


def _tokens(case, cfg, seed):
    """Every row's tokens: a prompt and what is fed behind it (no stop tokens, which are the last ones)."""
    rng, feed = np.random.default_rng(seed), []
    if case["call"] == "generate" and case["model"] not in STACKS:
        tk = get_tokenizer("qwen3", cfg.vocab)
        feed = tk.encode("{", False) + tk.encode(" ", False) * (case["new"] - 1)
    return [rng.integers(0, cfg.vocab, n).tolist() + (feed or rng.integers(0, cfg.vocab // 2, case["new"]).tolist()) for n in _lengths(case)]


def prepare(case, seed):
    cfg = _config(case)
    weights = _tensors(cfg, seed)
    dev = torch.device("cuda:0")
    w = S.StackWeights.from_tensors(cfg, weights.__getitem__, dev) if isinstance(cfg, S.StackConfig) \
        else M.Weights.from_hf_state_dict(cfg, weights, dev)
    del weights
    lens = _lengths(case)
    longest = max(lens) + case["new"]
    blocks = -(-longest // PAGE) + 1
    generate = case["call"] == "generate"
    launch = max(sum(e[2] for e in step) for step in _passes(case))
    if generate:        # the first attempt computes whole prompts
        launch = sum(lens)
    engine = Engine(cfg, w, get_tokenizer("qwen3", cfg.vocab) if generate else None, max_model_len=blocks * PAGE, max_rows=case["rows"],
                    prefill_tokens=min(16384, -(-launch // 128) * 128), kv_pages=case["rows"] * blocks + 8, logit_rows=128 if case["want"] > 1 else 0)
    tokens = _tokens(case, cfg, seed)
    state = dict(engine=engine, rows=case["rows"], vocab=cfg.vocab)
    if generate:
        schema = None if case["model"] in STACKS else VOTE
        state["requests"] = [Request("", schema, 0.3, case["new"], forced=t[n:], prompt_ids=t[:n]) for t, n in zip(tokens, lens)]
        engine.generate(state["requests"])
    else:
        state["steps"] = [[(r, tokens[r][a:a + n], list(range(n - want, n))) for r, a, n, want in step] for step in _schedule(case)]
    return state


def run(state):
    engine = state["engine"]
    if "requests" in state:
        results = engine.generate(state["requests"])
        return {"tokens": np.array([r.token_ids for r in results]), "logits": engine.buf["logits"][:state["rows"], :state["vocab"]]}
    live = [None] * state["rows"]
    out = []
    for step in state["steps"]:
        work_items = []
        for r, tokens, want in step:
            if live[r] is None:
                live[r] = engine.open()
            work_items.append((live[r], tokens, want))
        out.append(engine.step(work_items))
    for seq in live:
        engine.close_sequence(seq)
    return {"logits": torch.cat(out)}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    # measured against 64 bits: dense models 2e-3, the designs up to 8e-3; with experts more, where another rounding chooses another
    # expert for a token
    if "experts" in case["model"]:
        return {"rel": 3e-2, "max": 5e-1}
    return {"rel": 2e-2, "max": 2e-1} if case["model"] in STACKS else {"rel": 1e-2, "max": 6e-2}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps, w=None):
    y = x * (x.square().mean(-1, keepdim=True) + eps).rsqrt()
    return y if w is None else y * w


def _turn(x, pos, dims, base, pairs, back=False):
    """Rotates the first `dims` of the last axis of x [rows, tokens, heads, n]: entry i with dims / 2 + i, or pairs of neighbours."""
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    a = pos.double()[:, None, None] * f * (-1.0 if back else 1.0)
    c, s, y = a.cos(), a.sin(), x.clone()
    i, j = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    y[..., i], y[..., j] = x[..., i] * c - x[..., j] * s, x[..., j] * c + x[..., i] * s
    return y


def _attend(q, k, v, scale, window=0, bias=None, sink=None, pool=0):
    """q [rows, tokens, heads, n], k and v with fewer heads; one row and key head at a time."""
    B, n, H, _ = q.shape
    G = k.shape[2]
    i, j = torch.arange(n, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
    hidden = (j > i) | (i - j >= (window or n))
    if pool:
        m = n // pool
        k, v = (torch.cat([x, x[:, :m * pool].unflatten(1, (m, pool)).mean(2)], 1) for x in (k, v))
        b = torch.arange(m, device=q.device)[None]
        hidden = torch.cat([hidden, b * pool + pool - 1 > i - window], 1)
    out = q.new_empty(B, n, H, v.shape[3])
    for r in range(B):
        for g in range(G):
            h = slice(g * H // G, (g + 1) * H // G)
            s = torch.einsum("ihd,jd->hij", q[r, :, h], k[r, :, g]) * scale
            if bias is not None:
                s = s - bias[h, None, None] * (i - j)
            s = s.masked_fill_(hidden, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = torch.maximum(top, sink[h, None, None])
            p = (s - top).exp_()
            den = p.sum(-1, keepdim=True) + (0.0 if sink is None else (sink[h, None, None] - top).exp())
            out[r, :, h] = torch.einsum("hij,jd->ihd", p / den, v[r, :, g])
    return out


def _lin(x, w):
    return x @ w.double().T


def _dense(cfg, w, x, pos):
    hd = cfg.head_dim
    f = lambda n: w[n].double()
    for i in range(cfg.n_layers):
        p = f"model.layers.{i}."
        h = _rms(x, cfg.rms_eps, f(p + "input_layernorm.weight"))
        q, k, v = (_lin(h, w[f"{p}self_attn.{c}_proj.weight"]).unflatten(-1, (-1, hd)) for c in "qkv")
        if cfg.qk_norm:
            q, k = _rms(q, cfg.rms_eps, f(p + "self_attn.q_norm.weight")), _rms(k, cfg.rms_eps, f(p + "self_attn.k_norm.weight"))
        q, k = (_turn(t, pos, hd, cfg.rope_theta, False) for t in (q, k))
        x = x + _lin(_attend(q, k, v, hd ** -0.5).flatten(2), w[p + "self_attn.o_proj.weight"])
        h = _rms(x, cfg.rms_eps, f(p + "post_attention_layernorm.weight"))
        x = x + _lin(torch.nn.functional.silu(_lin(h, w[p + "mlp.gate_proj.weight"])) * _lin(h, w[p + "mlp.up_proj.weight"]),
                     w[p + "mlp.down_proj.weight"])
    return _rms(x, cfg.rms_eps, f("model.norm.weight"))


def _latent(m, w, h, pos, eps, caches, i):
    q = _lin(h, w["q"]).unflatten(-1, (m.heads, -1))
    q = torch.cat([q[..., :m.dim], _turn(q[..., m.dim:], pos, m.rot.dims, m.rot.base, m.rot.pairs)], -1)
    if m.kv_from is None:
        c = _lin(h, w["dkv"])
        caches[i] = _rms(c[..., :m.kv_rank], eps, w["dkv.norm"]), _turn(c[..., None, m.kv_rank:], pos, m.rot.dims, m.rot.base, m.rot.pairs)
    latent, kr = caches[i if m.kv_from is None else m.kv_from]
    k = torch.cat([_lin(latent, w["uk"]).unflatten(-1, (m.heads, -1)), kr.expand(-1, -1, m.heads, -1)], -1)
    v = _lin(latent, w["uv"]).unflatten(-1, (m.heads, -1))
    return _lin(_attend(q, k, v, m.scale, m.window, sink=w["sink"]).flatten(2), w["o"])


def _delta(m, w, h, eps):
    split = lambda t: t.unflatten(-1, (m.heads, m.dim))
    r, k, v = (split(_lin(h, w[n])) for n in "rkv")
    decay = split((-math.exp(-0.5) * (_lin(_lin(h, w["w1"]).tanh(), w["w2"]) + w["w0"]).sigmoid()).exp())
    u = k * (k.square().sum(-1, keepdim=True) + 1e-6).rsqrt()
    gone = split((_lin(h, w["a"]) + w["a.b"]).sigmoid()) * u
    st, out = h.new_zeros(h.shape[0], m.heads, m.dim, m.dim), torch.empty_like(r)
    for t in range(h.shape[1]):
        seen = u[:, t, :, None] @ st
        st = decay[:, t, :, :, None] * st - gone[:, t, :, :, None] * seen + k[:, t, :, :, None] * v[:, t, :, None]
        out[:, t] = (r[:, t, :, None] @ st)[:, :, 0]
    return _lin(_rms(out, eps).flatten(2) * w["norm"] * _lin(h, w["g"]).sigmoid(), w["o"])


def _state_space(m, w, h, eps):
    n, gn = m.out_dim, m.groups * m.state
    z, x, step = _lin(h, w["in"]).split([n, n + 2 * gn, m.heads], -1)
    x = torch.nn.functional.conv1d(torch.nn.functional.pad(x.mT, (m.conv - 1, 0)), w["conv"][:, None], w["conv.b"], groups=n + 2 * gn).mT
    x, b, c = torch.nn.functional.silu(x).split([n, gn, gn], -1)
    x = x.unflatten(-1, (m.heads, m.vdim))
    b, c = (t.unflatten(-1, (m.groups, m.state)).repeat_interleave(m.heads // m.groups, 2) for t in (b, c))
    step = torch.logaddexp(step + w["dt_bias"], step.new_zeros(()))
    keep = (-w["A_log"].exp() * step).exp()
    st, out = h.new_zeros(h.shape[0], m.heads, m.vdim, m.state), torch.empty_like(x)
    for t in range(h.shape[1]):
        st = keep[:, t, :, None, None] * st + (step[:, t, :, None] * x[:, t])[..., None] * b[:, t, :, None]
        out[:, t] = (st @ c[:, t, :, :, None])[..., 0]
    y = (out + w["D"][:, None] * x).flatten(2) * torch.nn.functional.silu(z)
    return _lin(_rms(y.unflatten(-1, (m.norm_groups, -1)), eps).flatten(2) * w["norm"], w["o"])


def _memory(m, w, h, eps):
    q, k, v = (_lin(h, w[n]).unflatten(-1, (m.heads, -1)) for n in "qkv")
    cap = lambda n: m.gate_cap * ((_lin(h, w[n]) + w[n + ".b"]) / m.gate_cap).tanh()
    gi, gf = cap("i"), torch.nn.functional.logsigmoid(cap("f"))
    B, H = h.shape[0], m.heads
    st, norm, top, out = h.new_zeros(B, H, m.vdim, m.dim), h.new_zeros(B, H, m.dim), h.new_zeros(B, H), torch.empty_like(v)
    for t in range(h.shape[1]):
        new = torch.maximum(gf[:, t] + top, gi[:, t])
        keep, add, top = (gf[:, t] + top - new).exp(), (gi[:, t] - new).exp(), new
        kt, qt = add[..., None] * k[:, t], q[:, t] * m.dim ** -0.5
        st = keep[..., None, None] * st + v[:, t, :, :, None] * kt[:, :, None]
        norm = keep[..., None] * norm + kt
        den = torch.maximum((norm * qt).sum(-1).abs(), (-top).exp()) + 1e-6
        out[:, t] = (st @ qt[..., None])[..., 0] / den[..., None]
    return _lin(_rms(out, eps).flatten(2) * w["norm"] * _lin(h, w["g"]).sigmoid(), w["o"])


def _grouped(m, w, h, pos, eps, first):
    """(output, values before they are mixed with those of the first such layer)"""
    add = lambda n: w[n + ".b"] if n + ".b" in w else 0.0
    q, k, v = (_lin(h, w[n]) + add(n) for n in "qkv")
    raw = v
    if m.v_mix and first is not None:
        v = (1 - w["vmix"]) * v + w["vmix"] * first
    if m.qk_norm:
        q, k = _rms(q, eps, w["q.norm"]), _rms(k, eps, w["k.norm"])
    q, k, v = q.unflatten(-1, (m.heads, -1)), k.unflatten(-1, (m.kv_heads, -1)), v.unflatten(-1, (m.kv_heads, -1))
    if m.head_norm:
        q, k = _rms(q, eps, w["q.norm"]), _rms(k, eps, w["k.norm"])
    if m.rot:
        q, k = (_turn(t, pos, m.rot.dims, m.rot.base, m.rot.pairs) for t in (q, k))
    if m.v_rot:
        v = _turn(v, pos, m.v_rot.dims, m.v_rot.base, True)
    if m.temp_coef:
        q = q * (1 + m.temp_coef * (((pos + 1) / m.temp_every).floor() + 1).log())[:, None, None]
    slopes = 2.0 ** (-8.0 * torch.arange(1, m.heads + 1, dtype=torch.float64, device=h.device) / m.heads) if m.slopes else None
    o = _attend(q, k, v, m.scale, m.window, slopes, pool=m.pool)
    if m.v_rot:
        o = _turn(o, pos, m.v_rot.dims, m.v_rot.base, True, back=True)
    if m.gate:
        o = o * _lin(h, w["g"]).sigmoid()[..., None]
    return _lin(o.flatten(2), w["o"]) + add("o"), raw


def _clamped(g, u, f):
    g, u = g.clamp(max=f.limit), u.clamp(-f.limit, f.limit)
    return g * (f.alpha * g).sigmoid() * (u + 1)


def _feed_forward(f, w, h, eps):
    if isinstance(f, S.DenseMlp):
        u = _lin(h, w["up"])
        if f.act == "poly_norm":
            a, b, c, e = w["act"].double()
            y = a * _rms(u, eps) + b * _rms(u ** 2, eps) + c * _rms(u ** 3, eps) + e
        elif f.act == "relu2":
            y = u.clamp(min=0) ** 2
        elif f.act == "clamped_glu":
            y = _clamped(_lin(h, w["gate"]), u, f)
        else:
            y = torch.nn.functional.gelu(_lin(h, w["gate"]), approximate="tanh") * u
        return _lin(y, w["down"])
    x = h.flatten(0, 1)
    logits = _lin(x, w["router"]) + (0.0 if f.glu else w["router.b"])
    best = logits.topk(f.top, -1)
    weight = best.values.sigmoid() if f.glu else best.values.softmax(-1)
    out = torch.zeros_like(x)
    if f.shared:
        out += _lin(torch.nn.functional.gelu(_lin(x, w["shared.up"])), w["shared.down"])
    for e in range(f.experts):
        t, c = (best.indices == e).nonzero(as_tuple=True)
        xe, s = x[t], weight[t, c][:, None]
        if f.glu:
            y = _lin(_clamped(_lin(xe * s, w[f"e{e}.gate"]), _lin(xe * s, w[f"e{e}.up"]), f), w[f"e{e}.down"])
        else:
            y = s * _lin(torch.nn.functional.gelu(_lin(xe, w[f"e{e}.up"])), w[f"e{e}.down"])
        out.index_add_(0, t, y)
    return out.view_as(h)


def _stack(cfg, w, x, pos):
    eps, caches, first = cfg.rms_eps, {}, None
    norm = lambda t, n: _rms(t, eps, w[n].double() + (cfg.norm_offset if ".mix." not in n else 0.0))
    x = x * cfg.embed_scale
    if cfg.embed_norm:
        x = norm(x, "embed.norm")
    if cfg.learned_pos:
        x = x + w["pos"].double()[pos]
    if cfg.sinusoid_pos:
        a = pos.double()[:, None] * 10000.0 ** (-2.0 * torch.arange(cfg.d_model // 2, dtype=torch.float64, device=x.device) / cfg.d_model)
        x = x + torch.stack([a.sin(), a.cos()], -1).flatten(1)
    for i, l in enumerate(cfg.layers):
        part = lambda p: {n[len(p):]: t if t.dim() == 2 and t.dtype == torch.bfloat16 else t.double() for n, t in w.items() if n.startswith(p)}
        h, y = norm(x, f"l{i}.norm1") if l.pre_norm else x, 0.0
        for side, m in zip(("mix.left.", "mix.right.") if len(l.mixers) == 2 else ("mix.",), l.mixers):
            v = part(f"l{i}.{side}")
            if isinstance(m, S.LatentAttention):
                o = _latent(m, v, h, pos, eps, caches, i)
            elif isinstance(m, S.GeneralDelta):
                o = _delta(m, v, h, eps)
            elif isinstance(m, S.StateSpace):
                o = _state_space(m, v, h, eps)
            elif isinstance(m, S.MatrixMemory):
                o = _memory(m, v, h, eps)
            else:
                o, raw = _grouped(m, v, h, pos, eps, first)
                first = raw if first is None else first
            y = y + o * (1.0 if len(l.mixers) == 1 else l.mixer.left_scale if "left" in side else l.mixer.right_scale)
        after = lambda t, k: norm(t, f"l{i}.norm{k}" + ("b" if l.pre_norm else "")) * (w[f"l{i}.ls{k}"].double() if l.layer_scale else 1.0) \
            if l.post_norm and not l.parallel else t
        if l.parallel:
            x = x + y + (_feed_forward(l.mlp, part(f"l{i}.mlp."), h, eps) if l.mlp else 0.0)
            continue
        x = x + after(y, 1)
        if l.mlp:
            x = x + after(_feed_forward(l.mlp, part(f"l{i}.mlp."), norm(x, f"l{i}.norm2") if l.pre_norm else x, eps), 2)
    return norm(x, "final.norm") * cfg.logit_scale


def exact(case, seed):
    cfg = _config(case)
    w = _tensors(cfg, seed)
    tokens = _tokens(case, cfg, seed)
    n = max(len(t) for t in tokens)
    ids = torch.tensor([t + [0] * (n - len(t)) for t in tokens], device="cuda")
    pos = torch.arange(n, device="cuda")
    stack = isinstance(cfg, S.StackConfig)
    embed = w["embed" if stack else "model.embed_tokens.weight"]
    head = w.get("head" if stack else "lm_head.weight", embed)
    wanted = [[(r, p) for r, a, n, want in step for p in range(a + n - want, a + n)] for step in _passes(case)]
    wanted = sum(wanted, []) if case["call"] == "replay" else wanted[-1]
    got = {}
    for r0 in range(0, case["rows"], 8):
        y = (_stack if stack else _dense)(cfg, w, embed[ids[r0:r0 + 8]].double(), pos)
        got.update({(r, p): y[r - r0, p] for r, p in wanted if r0 <= r < r0 + 8})
    x = torch.stack([got[e] for e in wanted])
    logits = torch.cat([_lin(x, head[v:v + 16384]) for v in range(0, cfg.vocab, 16384)], 1)
    return {"tokens": None, "logits": logits} if case["call"] == "generate" else {"logits": logits}
