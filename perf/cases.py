"""What this library is used for, as cases that can be timed and checked.

A pass is one piece of work of a user's program on an engine that it holds: take slots, run the
requests through the public entry points (``Engine.step``, ``DecodeSession``), give the slots back.
Sizes are those of the presets, of the benchmark and of the tests.  Three kinds of work:

``answer``  what ``Engine.generate`` runs: the prompts of a batch in one step, then one token a
            sequence and step through a decode session, the host's tokens in and the selected
            tokens out.  The tokens that go in are given by the case and not the selected ones: two
            correct implementations in 16 bits select different tokens at near ties, and everything
            after such a place would have to differ.
``score``   the logits at every place of some texts (likelihoods), in one step.
``replay``  what ``bin/trace_run`` drives: requests that go on in later steps with a chunk of new
            tokens behind what the cache holds, and with single tokens, through ``Engine.step``.

The results are the logits at the wanted places and, of ``answer``, the logit that each selected
token has.  ``exact`` computes them from the same weights and tokens in float64 with plain torch
operations over whole sequences, without a cache.  Of the designs beside GPT-2 one stands here that
has no routed experts (which experts a token takes is decided by comparisons that rounding to 16 bits
may turn over, so results of two correct implementations would not be close everywhere).
"""
from __future__ import annotations

import json
import math
from dataclasses import dataclass
from pathlib import Path

import torch

import nimbus_infer_rs_b200
from nimbus_infer_rs_b200 import Engine
from nimbus_infer_rs_b200.config.registry import resolve_architecture
from nimbus_infer_rs_b200.engine.decode import DecodeSession
from nimbus_infer_rs_b200.engine.model import PRECISIONS, Model, Runtime
from nimbus_infer_rs_b200.weights.loader import TensorDict, load_params

PRESETS = Path(nimbus_infer_rs_b200.__file__).resolve().parent / "config" / "presets"
PAGE = 64            # tokens of a cache page: what a sequence holds counts in whole pages
CHUNK = 1 << 24      # numbers of a float64 block of scores or logits


def _case(name, work, preset, dtype, batch, shortest, longest, new=0, turn=0):
    """``batch`` texts of ``shortest`` to ``longest`` tokens, then (``replay``) ``turn`` more tokens
    each, then ``new`` single tokens each."""
    return {"name": name, "work": work, "preset": preset, "dtype": dtype, "batch": batch,
            "shortest": shortest, "longest": longest, "new": new, "turn": turn}


def listed():
    return [
        # a single short request: latency and launches
        _case("one short answer", "answer", "gpt2", "bfloat16", 1, 13, 13, new=12),
        # the protocol of the command line's `bench` and of the published CPU figures
        _case("one answer, 128 + 64", "answer", "gpt2", "bfloat16", 1, 128, 128, new=62),
        # a small batch of chats near the model's full context: the benchmark's headline
        _case("eight long chats", "answer", "gpt2", "bfloat16", 8, 731, 960, new=48),
        # many short unequal requests
        _case("64 short answers", "answer", "gpt2", "bfloat16", 64, 9, 201, new=32),
        # prompts alone (first tokens, rankings by the last place): the benchmark's prefill
        _case("two whole prompts", "answer", "gpt2", "bfloat16", 2, 1024, 1024),
        # unequal prompts of a larger model
        _case("medium, eight prompts", "answer", "gpt2-medium", "bfloat16", 8, 32, 1000, new=8),
        # likelihoods of every token of a text
        _case("scores of a text", "score", "gpt2", "bfloat16", 1, 997, 997),
        # conversations that go on: a chunk behind a cached context, then single tokens by step
        _case("conversations go on", "replay", "gpt2", "bfloat16", 5, 211, 618, new=16, turn=77),
        # the largest model, a full batch
        _case("xl, 64 requests", "answer", "gpt2-xl", "bfloat16", 64, 97, 128, new=24),
        # true 32-bit: a batch of answers, and prompts
        _case("32-bit answers", "answer", "gpt2", "float32", 8, 99, 401, new=24),
        _case("32-bit prompts", "answer", "gpt2", "float32", 2, 1000, 1024),
        # another design: differential and latent attention on several streams
        _case("streams, eight answers", "answer", "bumulix-2k", "bfloat16", 8, 203, 700, new=24),
    ]


def _between(rng, lo, hi):
    """A whole number from ``lo`` to ``hi``, spread evenly over its logarithm."""
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng):
    work = rng.choice(("answer", "answer", "answer", "replay", "score"))
    preset = rng.choice(("gpt2", "gpt2", "gpt2", "gpt2-medium", "gpt2-xl", "bumulix-2k"))
    dtype = "float32" if preset == "gpt2" and rng.random() < 0.3 else "bfloat16"
    longest = _between(rng, 8, 900)
    shortest = _between(rng, max(1, longest // 8), longest)
    rows = {"gpt2": 16384, "gpt2-medium": 8192, "gpt2-xl": 4096, "bumulix-2k": 8192}[preset]
    batch = _between(rng, 1, max(1, min(64, rows // (2 if dtype == "float32" else 1) // longest)))
    if work == "score":     # every place's logits come back
        batch, new = max(1, min(batch, 2048 // longest)), 0
    else:
        new = _between(rng, 4, 48)
    turn = _between(rng, 2, 70) if work == "replay" else 0
    c = _case("", work, preset, dtype, batch, shortest, longest, new=new, turn=turn)
    return {k: v for k, v in c.items() if k != "name"}


# ------------------------------------------------------------------------------------- inputs
def _config(preset):
    obj = json.loads((PRESETS / f"{preset}.json").read_text())
    return {k: v for k, v in obj.items() if k not in ("_about", "random_weights")}


def _lengths(case):
    """The texts' lengths, from the shortest to the longest in unequal steps, in a mixed order."""
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    steps = [lo + (hi - lo) * i // (n - 1) for i in range(n)]
    return [steps[i * 7 % n] for i in range(n)] if n % 7 else steps[::-1]


def _vocab(cfg):
    return cfg["vocab"] if "vocab" in cfg else cfg["vocab_size"]


def _texts(case, cfg, seed):
    """Every request's tokens: its text, its turn and its single tokens behind one another."""
    g = torch.Generator().manual_seed(int(seed) * 2 + 1)
    return [torch.randint(0, _vocab(cfg), (n + case["turn"] + case["new"],), generator=g).tolist()
            for n in _lengths(case)]


class _Values:
    """Random tensors on the GPU, drawn one after another from one seed."""

    def __init__(self, seed, dtype):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) * 2)
        self.dtype = dtype

    def matrix(self, *shape, std):
        return (torch.randn(*shape, generator=self.g, device="cuda") * std).to(self.dtype)

    def vector(self, n, std, mean=0.0):
        return torch.randn(n, generator=self.g, device="cuda") * std + mean


def _gpt2_tensors(cfg, v):
    """Under the names of published GPT-2 files; linear weights stand ``(in, out)``."""
    d, m = cfg["n_embd"], cfg.get("n_inner") or 4 * cfg["n_embd"]
    t = {"wte.weight": v.matrix(cfg["vocab_size"], d, std=0.02),
         "wpe.weight": v.matrix(cfg["n_positions"], d, std=0.02)}
    for i in range(cfg["n_layer"]):
        p = f"h.{i}."
        for name, a, b in (("attn.c_attn", d, 3 * d), ("attn.c_proj", d, d), ("mlp.c_fc", d, m),
                           ("mlp.c_proj", m, d)):
            t[f"{p}{name}.weight"] = v.matrix(a, b, std=0.02)
            t[f"{p}{name}.bias"] = v.vector(b, 0.02)
        for name in ("ln_1", "ln_2"):
            t[f"{p}{name}.weight"], t[f"{p}{name}.bias"] = v.vector(d, 0.1, 1.0), v.vector(d, 0.02)
    t["ln_f.weight"], t["ln_f.bias"] = v.vector(d, 0.1, 1.0), v.vector(d, 0.02)
    return t


def _bumulix_tensors(cfg, v):
    """Under the names of a Bumulix weight file; linear weights stand ``(out, in)``."""
    D, S = cfg["width"], cfg["streams"]

    def mat(n_out, n_in):
        return v.matrix(n_out, n_in, std=n_in ** -0.5)

    t = {"embed": v.matrix(cfg["vocab"], D, std=1.0)}
    for i, layer in enumerate(cfg["layers"]):
        m, p, x = layer["mixer"], f"l{i}.", f"l{i}.mix."
        for q in (1, 2):
            t[f"{p}norm{q}"], t[f"{p}ls{q}"] = v.vector(D, 0.1), v.vector(D, 0.1, 1.0)
            t[f"{p}hc{q}.in"], t[f"{p}hc{q}.out"] = v.vector(S, 0.1, 1.0 / S), v.vector(S, 0.1, 1.0)
            t[f"{p}hc{q}.mix"] = torch.eye(S, device="cuda") + v.vector(S * S, 0.1).view(S, S)
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "attention":
            t[x + "q"], t[x + "k"] = mat(H * 2 * d, D), mat(m["kv_heads"] * 2 * d, D)
            t[x + "v"] = mat(m["kv_heads"] * dv, D)
            for name in ("lq1", "lk1", "lq2", "lk2"):
                t[x + name] = v.vector(d, 0.1)
        else:
            R, Q, dr = m["kv_rank"], m["q_rank"], m["rot_dim"]
            t[x + "dq"], t[x + "uq"], t[x + "dkv"] = mat(Q, D), mat(H * (d + dr), Q), mat(R + dr, D)
            t[x + "dq.norm"], t[x + "dkv.norm"] = v.vector(Q, 0.1, 1.0), v.vector(R, 0.1, 1.0)
            t[x + "uk"], t[x + "uv"], t[x + "g"] = mat(H * d, R), mat(H * dv, R), mat(H * dv, D)
        t[x + "o"] = mat(D, H * dv)
        t[p + "mlp.up"], t[p + "mlp.down"] = mat(layer["mlp"]["ff"], D), mat(D, layer["mlp"]["ff"])
    t["final.norm"] = v.vector(D, 0.1)
    return t


def _tensors(case, cfg, seed):
    make = _bumulix_tensors if "streams" in cfg else _gpt2_tensors
    return make(cfg, _Values(seed, PRECISIONS[case["dtype"]]))


@dataclass
class State:
    case: dict
    engine: Engine
    texts: list            # the tokens of each request
    lengths: list          # how many of them are its text
    logits: torch.Tensor | None   # [1 + new, batch, vocab]: where the logits of an answer are kept


def prepare(case, seed):
    """A model in memory, loaded through the by-name plan that a weight file takes, a cache with
    room for the requests, and the requests' tokens on the host."""
    cfg = _config(case["preset"])
    arch = resolve_architecture(cfg)
    config = arch.config_cls.from_json(cfg)
    source = TensorDict(_tensors(case, cfg, seed))
    rt = Runtime(torch.device("cuda:0"), PRECISIONS[case["dtype"]])
    spec = arch.build_spec(config)
    model = Model(spec, rt)
    plan = arch.weight_plan(config, spec, set(source.names()))
    model.bind(load_params(model.param_specs(), plan, source, precision=rt.precision, device=rt.device))
    texts, lengths = _texts(case, cfg, seed), _lengths(case)
    pages = sum(-(-(len(t) + 1) // PAGE) for t in texts)
    if "streams" in cfg:       # what bounds a sequence is the cache
        pages = max(pages, -(-2048 // PAGE))
    engine = Engine(model, config, cache_tokens=pages * PAGE, n_slots=case["batch"])
    kept = None
    if case["work"] == "answer":
        kept = torch.empty((1 + case["new"], case["batch"], _vocab(cfg)), device="cuda")
    return State(case, engine, texts, lengths, kept)


# ------------------------------------------------------------------------------------- a pass
def run(state):
    slots = [state.engine.alloc_slot() for _ in state.texts]
    try:
        return {"answer": _answer, "score": _score, "replay": _replay}[state.case["work"]](state, slots)
    finally:
        for s in slots:
            state.engine.free_slot(s)


def _answer(state, slots):
    """The prompts' step and the decode steps behind it, as ``Engine.generate`` takes them."""
    engine, new, out = state.engine, state.case["new"], state.logits
    out[0] = engine.step([(s, t[:n], [n - 1]) for s, t, n in zip(slots, state.texts, state.lengths)])
    if not new:
        return {"logits": out}
    fed = [[t[n + k] for t, n in zip(state.texts, state.lengths)] for k in range(new)]
    session = DecodeSession(engine, slots, fed[0])
    selected = []
    try:
        for k in range(new):
            session.step(fed[k])
            selected.append(session.read_tokens())
            out[1 + k] = session.logits
    finally:
        session.close()
    at = torch.tensor(selected, device=out.device)
    return {"logits": out, "selected": out[1:].gather(2, at[:, :, None])[:, :, 0]}


def _score(state, slots):
    return {"logits": state.engine.step([(s, t, range(len(t))) for s, t in zip(slots, state.texts)])}


def _replay(state, slots):
    """Text, turn and single tokens, each a step; the logits of every step's last places."""
    engine, case = state.engine, state.case
    at = list(state.lengths)
    out = [engine.step([(s, t[:n]) for s, t, n in zip(slots, state.texts, at)])]
    for size in [case["turn"]] + [1] * case["new"]:
        out.append(engine.step([(s, t[n:n + size]) for s, t, n in zip(slots, state.texts, at)]))
        at = [n + size for n in at]
    return {"logits": out}


# ------------------------------------------------------------------------------------- its work
def _layer_sizes(cfg):
    """Per layer: the numbers of its matrices; what a (query, key) pair costs (multiply-adds); the
    numbers it keeps of a token; how far back it sees."""
    if "streams" not in cfg:
        d, m = cfg["n_embd"], cfg.get("n_inner") or 4 * cfg["n_embd"]
        hd = cfg["n_head"] * (cfg.get("head_dim") or d // cfg["n_head"])
        return [(4 * d * hd + 2 * d * m, 2 * hd, 2 * hd, 1 << 30)] * cfg["n_layer"]
    D, out = cfg["width"], []
    for layer in cfg["layers"]:
        m = layer["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "attention":
            G = m["kv_heads"]
            out.append((D * (2 * H * d + 2 * G * d + G * dv + H * dv) + 2 * D * layer["mlp"]["ff"],
                        H * 2 * (d + dv), G * (2 * d + dv), m["mask"]["size"]))
        else:
            R, Q, dr = m["kv_rank"], m["q_rank"], m["rot_dim"]
            out.append((D * (Q + R + dr + 2 * H * dv) + Q * H * (d + dr) + R * H * (d + dv)
                        + 2 * D * layer["mlp"]["ff"], H * (d + dr + dv), R + dr, 1 << 30))
    return out


def _steps(case):
    """Every step of a pass: (tokens before it, tokens in it, rows wanted) per request."""
    lengths = _lengths(case)
    steps = [[(0, n, n if case["work"] == "score" else 1) for n in lengths]]
    at = lengths
    for size in ([case["turn"]] if case["turn"] else []) + [1] * case["new"]:
        steps.append([(n, size, 1) for n in at])
        at = [n + size for n in at]
    return steps


def work(case):
    """Per step: every weight once (a step needs the tokens of the one before it, and the weights of
    all layers do not stay on the chip between two), the cached keys and values its tokens see read
    and the new ones written once, the wanted logits written; twice the multiply-adds as flops."""
    cfg = _config(case["preset"])
    size, V = (2 if case["dtype"] == "bfloat16" else 4), _vocab(cfg)
    D = cfg.get("width") or cfg["n_embd"]
    nbytes = flops = 0
    for step in _steps(case):
        rows, wanted = sum(s[1] for s in step), sum(s[2] for s in step)
        nbytes += V * D * size + wanted * V * 4 + rows * (D * size + 4)
        flops += 2 * wanted * V * D
        for weights, pair, kept, window in _layer_sizes(cfg):
            nbytes += weights * size
            flops += 2 * rows * weights
            for before, n, _ in step:
                first = max(0, before + 1 - window)
                nbytes += (before - first + n) * kept * size
                pairs = sum(min(before + j + 1, window) for j in range(n))
                flops += 2 * pairs * pair
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the results are off ``exact`` by: 1.5e-6 in 32-bit, 0.005 in 16-bit
    (2-norm; single logits by a few times that, of the results' root mean square)."""
    return {"rel": 1e-5, "max": 1e-4} if case["dtype"] == "float32" else {"rel": 2e-2, "max": 0.1}


# ------------------------------------------------------------------------------------- in 64 bits
def exact(case, seed):
    cfg = _config(case["preset"])
    forward = _bumulix_logits if "streams" in cfg else _gpt2_logits
    weights, texts, lengths = _tensors(case, cfg, seed), _texts(case, cfg, seed), _lengths(case)
    rows = []                       # of each request: the places whose logits are wanted
    for text, n in zip(texts, lengths):
        if case["work"] == "score":
            rows.append(list(range(n)))
        else:
            first = [n - 1] + ([n - 1 + case["turn"]] if case["turn"] else [])
            rows.append(first + [first[-1] + 1 + k for k in range(case["new"])])
    got = [forward(weights, cfg, torch.tensor(t, device="cuda"), torch.tensor(r, device="cuda"))
           for t, r in zip(texts, rows)]
    if case["work"] == "score":
        return {"logits": torch.cat(got)}
    logits = torch.stack(got, 1)    # [places, batch, vocab]
    if case["work"] == "replay":
        return {"logits": list(logits)}
    return {"logits": logits} | ({"selected": logits[1:].amax(2)} if case["new"] else {})


def _softmax_rows(q, k, v, scale, window=1 << 30):
    """q [H, T, d], k [H, T, d], v [H, T, dv]: causal softmax attention, a block of rows at a time."""
    H, T, _ = q.shape
    out, rows = [], max(1, CHUNK // (H * T))
    j = torch.arange(T, device=q.device)
    for r in range(0, T, rows):
        s = q[:, r:r + rows] @ k.transpose(1, 2) * scale
        i = torch.arange(r, min(T, r + rows), device=q.device)[:, None]
        out.append(s.masked_fill((j > i) | (i - j >= window), -math.inf).softmax(-1) @ v)
    return torch.cat(out, 1)


def _gpt2_logits(W, cfg, tokens, rows):
    d, H, eps = cfg["n_embd"], cfg["n_head"], cfg["layer_norm_epsilon"]

    def norm(x, p):
        c = x - x.mean(-1, keepdim=True)
        return c / (c.square().mean(-1, keepdim=True) + eps).sqrt() * W[p + "weight"].double() \
            + W[p + "bias"].double()

    def linear(x, p):
        return x @ W[p + "weight"].double() + W[p + "bias"].double()

    T = tokens.numel()
    x = W["wte.weight"][tokens].double() + W["wpe.weight"][:T].double()
    for i in range(cfg["n_layer"]):
        p = f"h.{i}."
        q, k, v = linear(norm(x, p + "ln_1."), p + "attn.c_attn.").view(T, 3, H, d // H).permute(1, 2, 0, 3)
        a = _softmax_rows(q, k, v, (d // H) ** -0.5)
        x = x + linear(a.transpose(0, 1).reshape(T, d), p + "attn.c_proj.")
        z = linear(norm(x, p + "ln_2."), p + "mlp.c_fc.")
        z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
        x = x + linear(z, p + "mlp.c_proj.")
    return norm(x[rows], "ln_f.") @ W["wte.weight"].double().T


def _bumulix_logits(W, cfg, tokens, rows):
    eps, m_res, S = cfg["norm"]["eps"], cfg["residual_mult"], cfg["streams"]
    T = tokens.numel()

    def w(name):
        return W[name].double()

    def unit(x):
        return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()

    def heads(x, n):
        return x.view(T, n, -1).transpose(0, 1)

    def turned(x, rot):
        """Pairs (i, i + dims / 2) turned by position; slow ones slowed, both scaled."""
        dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
        rates = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
        at = [dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base))
              for t in (sc["fast"], sc["slow"])]
        lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
        r = ((torch.arange(dims // 2, device=x.device) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        rates = rates / sc["factor"] * r + rates * (1.0 - r)
        size = 0.1 * math.log(sc["factor"]) + 1.0
        ang = torch.arange(T, device=x.device)[:, None] * rates
        c, s = size * ang.cos(), size * ang.sin()
        a, b = x[..., :dims // 2], x[..., dims // 2:dims]
        return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)

    def differential(x, p, m):
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        q = (x @ w(p + "q").T).view(T, H, 2, d).permute(2, 1, 0, 3)
        k = (x @ w(p + "k").T).view(T, G, 2, d).permute(2, 1, 0, 3).repeat_interleave(H // G, 1)
        v = heads(x @ w(p + "v").T, G).repeat_interleave(H // G, 0)
        a, b = (_softmax_rows(q[i], k[i], v, m["scale"], m["mask"]["size"]) for i in (0, 1))
        lam = (w(p + "lq1") * w(p + "lk1")).sum().exp() - (w(p + "lq2") * w(p + "lk2")).sum().exp() + m["diff"]
        return unit(a - lam * b) * (1.0 - m["diff"])

    def latent(x, p, m):
        H, d, R = m["heads"], m["dim"], m["kv_rank"]
        q = heads(unit(x @ w(p + "dq").T) * w(p + "dq.norm") @ w(p + "uq").T, H)
        down = x @ w(p + "dkv").T
        c = unit(down[:, :R]) * w(p + "dkv.norm")
        k = torch.cat([heads(c @ w(p + "uk").T, H), turned(down[:, R:], m["rot"]).expand(H, T, -1)], -1)
        q = torch.cat([q[..., :d], turned(q[..., d:], m["rot"])], -1)
        o = _softmax_rows(q, k, heads(c @ w(p + "uv").T, H), m["scale"])
        return o * heads((x @ w(p + "g").T).sigmoid(), H)

    def feed_forward(x, p):
        z = x @ w(p + "up").T
        return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3))) @ w(p + "down").T

    xs = w("embed")[tokens].expand(S, T, -1)
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        for q in (1, 2):
            h = unit(torch.einsum("s,std->td", w(f"{p}hc{q}.in"), xs)) * (1.0 + w(f"{p}norm{q}"))
            if q == 1:
                mix = differential if layer["type"] == "attention" else latent
                y = mix(h, p + "mix.", layer["mixer"]).transpose(0, 1).reshape(T, -1) @ w(p + "mix.o").T
            else:
                y = feed_forward(h, p + "mlp.")
            xs = torch.einsum("st,snd->tnd", w(f"{p}hc{q}.mix"), xs) \
                + m_res * w(f"{p}hc{q}.out")[:, None, None] * (y * w(f"{p}ls{q}"))
    x = unit(xs.sum(0)[rows]) * (1.0 + w("final.norm"))
    cap = cfg["logit_softcap"]
    return cap * torch.tanh(x @ w("embed").T / cap)
