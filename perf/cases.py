"""The work by which this engine's speed is judged: steps of its step function on random weights of its sample
configurations, and one closed loop of the engine.

A case names a configuration, what is run on it and its sizes.  ``prepare`` builds the engine with weights drawn from the
seed and brings the requests to the state that the call finds them in; ``run`` is the call; ``exact`` states the same models
plainly in 64 bits, from the published rule for the weights to the logits, without the package.

Kinds of call:

* ``decode``: one token for every live request;
* ``prefill``: one step with whole new prompts, which leave afterwards; the logits of each prompt's last token;
* ``mixed``: a new prompt in two portions, each beside one token of every live request;
* ``replay``: given tokens fed through the step function, first a prompt with the logits of all its places, then two single
  tokens;
* ``generate``: ``Engine.generate``, prompts to greedily chosen tokens.
"""
from __future__ import annotations

import hashlib
import json
import math
import os

import numpy as np
import torch

from infurnace_b200.engine import Engine, EngineOptions, SamplingParams, StepEntry

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PAGE = 16              # tokens of a page
BUDGET = 2048          # tokens of a step
ROOM = 128             # decoded tokens after which a request starts over from its prompt
# Layers of a model that are run where those it has would be too many: with random weights of the larger model's sizes
# two correct bfloat16 engines part by 3.5 % of the logits after its 36 layers, and by 1.7 % after these.
LAYERS = {"qwen3-8b": 8}

TINY = dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=2, hidden_size=64, num_attention_heads=4,
            num_key_value_heads=2, head_dim=16, intermediate_size=128, vocab_size=256, rope_theta=10000.0, rms_norm_eps=1e-6,
            tie_word_embeddings=True, max_position_embeddings=128)


def _config(case):
    if case["model"] == "tiny":
        return dict(TINY)
    with open(os.path.join(ROOT, "configs", case["model"] + ".json"), encoding="utf-8") as f:
        cfg = json.load(f)
    if case["model"] in LAYERS:
        cfg["num_hidden_layers"] = LAYERS[case["model"]]
    return cfg


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    def case(name, model, kind, requests=1, shortest=0, longest=0, tokens=0, dtype="bfloat16"):
        """``requests`` live requests or new prompts of ``shortest`` to ``longest`` tokens; ``tokens``: of the prompt that
        comes in portions or is replayed, or those to generate."""
        return dict(name=name, model=model, kind=kind, dtype=dtype, requests=requests, shortest=shortest, longest=longest,
                    tokens=tokens)
    return [
        # the smallest use: three short prompts generated from by a toy model in 32-bit arithmetic
        case("generate-tiny-fp32", "tiny", "generate", 3, 1, 33, 16, dtype="float32"),
        # one chat: every token waits for the one before
        case("decode-0.6b-1", "qwen3-0.6b", "decode", 1, 301, 301),
        # a few long contexts, the setting that the benchmark quotes
        case("decode-0.6b-8-long", "qwen3-0.6b", "decode", 8, 3967, 3967),
        # a full batch of short chats (prompts of 128 tokens, up to 256 generated)
        case("decode-0.6b-64", "qwen3-0.6b", "decode", 64, 129, 383),
        # time to the first token of a short question
        case("prefill-0.6b-131", "qwen3-0.6b", "prefill", 1, 131, 131),
        # a document
        case("prefill-0.6b-2048", "qwen3-0.6b", "prefill", 1, 2048, 2048),
        # serving: portions of a prompt beside requests that decode
        case("mixed-0.6b-15", "qwen3-0.6b", "mixed", 15, 77, 1500, 803),
        # checking against another implementation in 32-bit arithmetic: logits at every place
        case("replay-0.6b-fp32", "qwen3-0.6b", "replay", 1, 0, 0, 193, dtype="float32"),
        # layers of the larger model, a small batch
        case("decode-8b-8", "qwen3-8b", "decode", 8, 411, 1024),
        # layers of the larger model, a document
        case("prefill-8b-2048", "qwen3-8b", "prefill", 1, 2048, 2048),
        # a recurrence and chunk-local attention with mixed heads: prompts of uneven length in one step
        case("prefill-kafunex-3", "kafunex-s", "prefill", 3, 147, 1215),
        # and decoding
        case("decode-kafunex-8", "kafunex-s", "decode", 8, 100, 900),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    c = dict(model="qwen3-0.6b", dtype="bfloat16", requests=1, shortest=0, longest=0, tokens=0)
    c["kind"] = rng.choice(["decode", "decode", "prefill", "prefill", "mixed", "replay", "generate"])
    if c["kind"] == "generate":
        c.update(model="tiny", dtype="float32", requests=rng.randint(1, 4), tokens=rng.randint(4, 32))
        c["longest"] = rng.randint(8, 64)
        c["shortest"] = rng.randint(1, c["longest"])
    elif c["kind"] == "replay":
        c.update(dtype="float32", tokens=_log(rng, 17, 193))
    elif c["kind"] == "mixed":
        c.update(requests=_log(rng, 1, 40), longest=_log(rng, 64, 2000), tokens=_log(rng, 64, 1800))
        c["shortest"] = rng.randint(16, c["longest"])
    else:
        c["model"] = rng.choice(["qwen3-0.6b", "qwen3-0.6b", "qwen3-8b", "kafunex-s"])
        large = c["model"] == "qwen3-8b"
        if c["kind"] == "decode":
            c["requests"] = _log(rng, 1, 16 if large else 64)
            c["longest"] = _log(rng, 64, min(4000, (8192 if large else 32768) // c["requests"]))
            c["shortest"] = rng.randint(c["longest"] // 4, c["longest"])
        else:
            total = _log(rng, 64, 1900)
            c["requests"] = rng.randint(1, min(8, total // 32))
            c["longest"] = max(2, 2 * total // (c["requests"] + 1) if c["requests"] > 1 else total)
            c["shortest"] = max(1, (2 * total) // c["requests"] - c["longest"]) if c["requests"] > 1 else total
            if c["shortest"] > c["longest"]:
                c["shortest"], c["longest"] = c["longest"], c["shortest"]
    return c


def _lengths(case):
    """The lengths of the case's requests, from the shortest to the longest in equal steps."""
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    return [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)] if lo else []


def _tokens(vocab, seed, n, what):
    """``n`` uniform token ids; ``what`` numbers the sequence."""
    return np.random.RandomState((seed * 1000003 + what) % (1 << 32)).randint(0, vocab, n).tolist()


def _portions(case):
    """Where the prompt of a mixed case is cut."""
    first = case["tokens"] * 5 // 9
    return first, case["tokens"] - first


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


# ------------------------------------------------------------------------------------------------ the calls
def prepare(case, seed):
    cfg = _config(case)
    vocab, lengths, kind = _vocab(cfg), _lengths(case), case["kind"]
    live = kind in ("decode", "mixed")
    longest = [n + 2 * ROOM + 2 if live else n + case["tokens"] for n in lengths] + [case["tokens"] + 2]
    options = EngineOptions(dtype=case["dtype"], page_size=PAGE, num_pages=sum(-(-n // PAGE) for n in longest),
                            max_num_seqs=max(1, case["requests"] + (kind == "mixed")), max_num_batched_tokens=BUDGET,
                            max_model_len=-(-max(longest) // PAGE) * PAGE)
    engine = Engine.from_random(cfg, seed, options)
    runner = engine.runner
    prompts = [_tokens(vocab, seed, n, i) for i, n in enumerate(lengths)]
    s = dict(kind=kind, engine=engine, runner=runner, prompts=prompts, lengths=lengths)
    if kind == "generate":
        s["sampling"] = SamplingParams(max_tokens=case["tokens"])
    if kind == "prefill":
        s["entries"] = [StepEntry("p%d" % i, p, [len(p) - 1]) for i, p in enumerate(prompts)]
    if kind in ("mixed", "replay"):
        s["new"] = _tokens(vocab, seed, case["tokens"] + 2, 9999)
        s["cut"] = _portions(case)[0]
        s["all"] = list(range(case["tokens"]))
    if live:
        s["rids"] = ["r%d" % i for i in range(len(prompts))]
        s["next"] = np.random.RandomState(seed % (1 << 32)).randint(0, vocab, (2 * ROOM, len(prompts))).tolist()
        s["step"] = 0
        todo = []                                       # the contexts are prefilled in steps of the token budget
        for rid, p in zip(s["rids"], prompts):
            runner.cache.add_request(rid)
            at = 0
            while at < len(p):
                n = min(len(p) - at, BUDGET - sum(len(e.tokens) for e in todo))
                todo.append(StepEntry(rid, p[at:at + n]))
                at += n
                if sum(len(e.tokens) for e in todo) == BUDGET:
                    runner.step(todo)
                    todo = []
        if todo:
            runner.step(todo)
    return s


def _singles(s):
    """The next token of every live request.  After ``ROOM`` steps the requests start over at the length of their prompts,
    on pages that still hold keys and values."""
    if s["step"] >= ROOM:
        cache, s["step"] = s["runner"].cache, 0
        for rid, n in zip(s["rids"], s["lengths"]):
            cache.free_request(rid)
            cache.add_request(rid)
            cache.allocate(rid, n)
            cache.commit(rid, n)
    row = s["next"][s["step"]]
    s["step"] += 1
    return [StepEntry(rid, [t], [0]) for rid, t in zip(s["rids"], row)]


def run(s):
    kind, runner = s["kind"], s["runner"]
    if kind == "decode":
        return runner.step(_singles(s))
    if kind == "prefill":
        for e in s["entries"]:
            runner.cache.add_request(e.request_id)
        logits = runner.step(s["entries"])
        for e in s["entries"]:
            runner.cache.free_request(e.request_id)
        return logits
    if kind == "mixed":
        new, cut = s["new"][:-2], s["cut"]
        runner.cache.add_request("new")
        first = runner.step(_singles(s) + [StepEntry("new", new[:cut])]).clone()
        second = runner.step(_singles(s) + [StepEntry("new", new[cut:], [len(new) - cut - 1])])
        runner.cache.free_request("new")
        return [first, second]
    if kind == "replay":
        new = s["new"]
        runner.cache.add_request("new")
        out = [runner.step([StepEntry("new", new[:-2], s["all"])]).clone()]
        out += [runner.step([StepEntry("new", [t], [0])]).clone() for t in new[-2:]]
        runner.cache.free_request("new")
        return out
    return [np.array(tokens) for tokens in s["engine"].generate(s["prompts"], s["sampling"])]


# ------------------------------------------------------------------------------------------------ what a call cannot do without
def _sequences(case):
    """(tokens a request held before, new tokens, places whose logits are wanted) of every request in a call."""
    kind, lengths = case["kind"], _lengths(case)
    if kind == "decode":
        return [(n, 1, 1) for n in lengths]
    if kind == "prefill":
        return [(0, n, 1) for n in lengths]
    if kind == "mixed":
        a, b = _portions(case)
        return [(n, 2, 2) for n in lengths] + [(0, a + b, 1)]
    if kind == "replay":
        return [(0, case["tokens"] + 2, case["tokens"] + 2)]
    return [(0, n + case["tokens"] - 1, case["tokens"]) for n in lengths]


def work(case):
    cfg, size = _config(case), 2 if case["dtype"] == "bfloat16" else 4
    W, V = cfg.get("hidden_size") or cfg["width"], _vocab(cfg)
    seqs = _sequences(case)
    new, wanted = sum(s[1] for s in seqs), sum(s[2] for s in seqs)
    flops = 2.0 * wanted * W * V
    params, kept = W * V, 0
    if "layers" in cfg:
        for layer in cfg["layers"]:
            m = layer["mixer"]
            h = m["heads"] * m["dim"]
            if layer["type"] == "attention":
                g = m["kv_heads"] * m["dim"]
                matrices = W * (3 * h + g)
                chunk = m["mask"]["size"]
                pairs = sum(p % chunk + 1 for before, n, _ in seqs for p in range(before, before + n))
                flops += 4.0 * pairs * h
                kept += sum(before % chunk + n for before, n, _ in seqs) * g * size
            else:
                v = m["heads"] * m["vdim"]
                matrices = W * (2 * h + 2 * v)
                flops += 4.0 * new * h * m["vdim"]
                kept += 2 * len(seqs) * h * m["vdim"] * 4
            matrices += 2 * W * layer["mlp"]["ff"]
            params += matrices
            flops += 2.0 * new * matrices
    else:
        L, d = cfg["num_hidden_layers"], cfg["head_dim"]
        h, g, f = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d, cfg["intermediate_size"]
        matrices = W * (2 * h + 2 * g + 3 * f)
        params += L * matrices
        flops += 2.0 * new * L * matrices
        flops += 4.0 * L * h * sum(n * before + n * (n + 1) / 2 for before, n, _ in seqs)
        kept += sum(before + n for before, n, _ in seqs) * L * 2 * g * size
    return {"bytes": float(params * size + kept + new * (W * size + 8) + wanted * V * 4), "flops": float(flops)}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"
    # four times the distances from ``exact`` that were measured: 2.5e-6 in 32-bit arithmetic, 0.004 for the small recurrent
    # model, 0.0075 and 0.017 for the others
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.016, "max": 0.2} if case["model"] == "kafunex-s" else {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------------------------------------ the models in 64 bits
class _Weights:
    """The random tensors of a model: element i of a tensor is mean + std * z_i, z_i the centred sum of the twelve 16-bit
    parts of three words of a 64-bit mixer at counters 3i, 3i + 1 and 3i + 2, rounded to bfloat16."""

    def __init__(self, seed):
        self.seed = seed

    def __call__(self, name, *shape, mean=None, std=None):
        if mean is None:
            mean, std = (1.0, 0.1) if len(shape) <= 1 else (0.0, 0.02)
        start = int.from_bytes(hashlib.sha256(("%d:%s" % (self.seed, name)).encode()).digest()[:8], "little")

        def signed(v):
            return v - (1 << 64) if v >> 63 else v

        def shifted(z, k):
            return (z >> k) & ((1 << (64 - k)) - 1)
        count = int(np.prod(shape)) if shape else 1
        out = torch.empty(count, dtype=torch.bfloat16, device="cuda")
        for a in range(0, count, 1 << 25):
            i = torch.arange(a, min(count, a + (1 << 25)), device="cuda") * 3
            total = torch.zeros_like(i)
            for j in range(3):
                z = (i + j) * signed(0x9E3779B97F4A7C15) + signed(start)
                z = (z ^ shifted(z, 30)) * signed(0xBF58476D1CE4E5B9)
                z = (z ^ shifted(z, 27)) * signed(0x94D049BB133111EB)
                z = z ^ shifted(z, 31)
                total += (z & 0xFFFF) + (shifted(z, 16) & 0xFFFF) + (shifted(z, 32) & 0xFFFF) + shifted(z, 48)
            one = torch.tensor([mean, std], dtype=torch.float32, device="cuda")
            out[a:a + i.numel()] = one[0] + one[1] * ((total - 393210).float() / 65536.0)
        return out.view(shape).double()


def _rms(v, eps):
    return v / torch.sqrt(v.pow(2).mean(-1, keepdim=True) + eps)


def _causal(q, k, v, scale, bias=None, visible=None):
    """Softmax attention of one sequence: q [T, H, d], k and v [T, G, d]."""
    T, H, _ = q.shape
    rep = H // k.shape[1]
    vis = torch.ones(T, T, dtype=torch.bool, device=q.device).tril() if visible is None else visible
    out = []
    for g in range(k.shape[1]):
        a = torch.einsum("thd,sd->hts", q[:, g * rep:(g + 1) * rep], k[:, g]) * scale
        out.append(torch.einsum("hts,sd->thd", a.masked_fill_(~vis, -math.inf).softmax(-1), v[:, g]))
    return torch.cat(out, dim=1)


def _qwen3(cfg, w, ids):
    """The final rows [T, W] of sequences of token ids, and the head's matrix."""
    W, d, eps = cfg["hidden_size"], cfg["head_dim"], cfg["rms_norm_eps"]
    H, G, F, V = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"], cfg["vocab_size"]
    table = w("model.embed_tokens.weight", V, W)
    xs = [table[i] for i in ids]
    head = table if cfg["tie_word_embeddings"] else None
    del table
    freq = cfg["rope_theta"] ** (-torch.arange(0, d, 2, device="cuda").double() / d)

    def turn(v):
        ang = torch.arange(v.shape[0], device="cuda").double()[:, None, None] * freq
        a, b = v[..., :d // 2], v[..., d // 2:]
        return torch.cat((a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()), dim=-1)
    for layer in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % layer
        n1, n2 = w(p + "input_layernorm.weight", W), w(p + "post_attention_layernorm.weight", W)
        wq, wk = w(p + "self_attn.q_proj.weight", H * d, W).t(), w(p + "self_attn.k_proj.weight", G * d, W).t()
        wv, wo = w(p + "self_attn.v_proj.weight", G * d, W).t(), w(p + "self_attn.o_proj.weight", W, H * d).t()
        qn, kn = w(p + "self_attn.q_norm.weight", d), w(p + "self_attn.k_norm.weight", d)
        gate, up = w(p + "mlp.gate_proj.weight", F, W).t(), w(p + "mlp.up_proj.weight", F, W).t()
        down = w(p + "mlp.down_proj.weight", W, F).t()
        for i, x in enumerate(xs):
            T = x.shape[0]
            h = _rms(x, eps) * n1
            q, k = turn(_rms((h @ wq).view(T, H, d), eps) * qn), turn(_rms((h @ wk).view(T, G, d), eps) * kn)
            x = x + _causal(q, k, (h @ wv).view(T, G, d), d ** -0.5).reshape(T, H * d) @ wo
            h = _rms(x, eps) * n2
            xs[i] = x + (torch.nn.functional.silu(h @ gate) * (h @ up)) @ down
    n = w("model.norm.weight", W)
    return [_rms(x, eps) * n for x in xs], head if head is not None else w("lm_head.weight", V, W)


def _kafunex(cfg, w, ids):
    W, V, eps = cfg["width"], cfg["vocab"], cfg["norm"]["eps"]
    table = w("embed", V, W)
    half = 10000.0 ** (-2.0 * torch.arange(W // 2, device="cuda").double() / W)

    def place(T):
        ang = torch.arange(T, device="cuda").double()[:, None] * half
        return torch.stack((ang.sin(), ang.cos()), dim=-1).reshape(T, W)
    xs = [table[i] + place(len(i)) for i in ids]
    for layer, spec in enumerate(cfg["layers"]):
        p, m, F = "l%d." % layer, spec["mixer"], spec["mlp"]["ff"]
        H, d, e = m["heads"], m["dim"], m["vdim"]
        if spec["type"] == "attention":
            G, size = m["kv_heads"], m["mask"]["size"]
            wq, wk, wg = w(p + "mix.q", H * d, W).t(), w(p + "mix.k", G * d, W).t(), w(p + "mix.g", H * d, W).t()
            qn, kn = w(p + "mix.q.norm", H * d), w(p + "mix.k.norm", G * d)
            talk, wo = w(p + "mix.talk", H, H, mean=0.0, std=0.35), w(p + "mix.o", W, H * d).t()
            slope = 2.0 ** (-8.0 * (torch.arange(H, device="cuda").double() + 1) / H)
        else:
            wq, wf, wv = w(p + "mix.q", H * d, W).t(), w(p + "mix.f", H * d, W).t(), w(p + "mix.v", H * e, W).t()
            bias, low = w(p + "mix.f.b", H * d, mean=0.0, std=0.5), w(p + "mix.lower", H * d, mean=0.5, std=0.1)
            norm, wo = w(p + "mix.norm", e), w(p + "mix.o", W, H * e).t()
        n1, n2 = w(p + "norm1"), w(p + "norm2")
        s1, s2, up, down = w(p + "ls1", W), w(p + "ls2", W), w(p + "mlp.up", F, W).t(), w(p + "mlp.down", W, F).t()
        for i, x in enumerate(xs):
            T = x.shape[0]
            if spec["type"] == "attention":
                q, k = (_rms(x @ wq, eps) * qn).view(T, H, d), x @ wk
                kn_ = (_rms(k, eps) * kn).view(T, G, d)
                k = k.view(T, G, d)
                y = []
                for a in range(0, T, size):                     # a chunk of positions at a time: nothing sees past its own
                    b = min(T, a + size)
                    at = torch.arange(a, b, device="cuda")
                    s = torch.einsum("thd,shd->hts", q[a:b], kn_[a:b].repeat_interleave(H // G, dim=1)) * m["scale"]
                    s = torch.einsum("ji,its->jts", talk, s - slope[:, None, None] * (at[:, None] - at[None, :]))
                    s = s.masked_fill(at[None, :] > at[:, None], -math.inf).softmax(-1)
                    y.append(torch.einsum("hts,shd->thd", s, k[a:b].repeat_interleave(H // G, dim=1)))
                y = (torch.cat(y).reshape(T, H * d) * torch.sigmoid(x @ wg)) @ wo
            else:
                q = torch.nn.functional.silu(x @ wq).view(T, H, 1, d)
                f = (low + (1 - low) * torch.sigmoid(x @ wf + bias)).view(T, H, d, 1)
                v = (x @ wv).view(T, H, 1, e)
                S, y = torch.zeros(H, d, e, dtype=torch.float64, device="cuda"), []
                for t in range(T):
                    S = torch.lerp(v[t].expand(H, d, e), S, f[t].expand(H, d, e))
                    y.append(q[t] @ S)
                y = (_rms(torch.stack(y).view(T, H, e), eps) * norm).reshape(T, H * e) @ wo
            x = x + s1 * _rms(y, eps) * n1
            xs[i] = x + s2 * _rms((x @ up).relu().pow(2) @ down, eps) * n2
    n = w("final.norm")
    return [_rms(x, eps) * n for x in xs], w("head", V, W)


def exact(case, seed):
    cfg, w = _config(case), _Weights(seed)
    vocab, lengths, kind = _vocab(cfg), _lengths(case), case["kind"]
    forward = _kafunex if "layers" in cfg else _qwen3
    prompts = [_tokens(vocab, seed, n, i) for i, n in enumerate(lengths)]
    if kind == "generate":
        todo = [list(p) for p in prompts]
        for _ in range(case["tokens"]):
            rows, head = forward(cfg, w, todo)
            for p, r in zip(todo, rows):
                p.append(int((r[-1] @ head.t()).argmax()))
        return [np.array(p[n:]) for p, n in zip(todo, lengths)]
    more = {"decode": 1, "mixed": 2}.get(kind, 0)
    following = np.random.RandomState(seed % (1 << 32)).randint(0, vocab, (2 * ROOM, max(1, len(prompts)))).tolist()
    seqs = [p + [following[s][i] for s in range(more)] for i, p in enumerate(prompts)]
    new = _tokens(vocab, seed, case["tokens"] + 2, 9999)
    if kind == "mixed":
        seqs.append(new[:-2])
    if kind == "replay":
        seqs = [new]
    rows, head = forward(cfg, w, seqs)
    if kind == "replay":
        logits = rows[0] @ head.t()
        return [logits[:-2], logits[-2:-1], logits[-1:]]
    if kind == "mixed":
        return [torch.stack([r[-2] for r in rows[:-1]]) @ head.t(), torch.stack([r[-1] for r in rows]) @ head.t()]
    return torch.stack([r[-1] for r in rows]) @ head.t()
