"""The measured work of the engine: what a serving process asks of ``ModelRunner.step``, the call through which every
token reaches a model, from one reply of one request to thousands of prompt rows in a step.

A case is a model (sizes of ``bench.py``, with fewer layers where the depth only repeats the work), a kind of step and
the lengths of its requests (``requests`` of them from ``shortest`` to ``longest`` tokens, evenly spread over the
logarithm, so that most are odd):

* ``decode``: every request has that many tokens in the cache; a pass decodes ``steps`` tokens of each, one step
  after the other, and takes the requests back to where they were (as a caller does that scores continuations);
* ``prompt``: a pass runs new requests of that many tokens, whole or in portions of ``portion`` tokens a step;
* ``mixed``: one step that decodes a row of every request beside ``portion`` tokens of a prompt whose first ``after``
  tokens are in the cache: what a scheduler under load asks for;
* ``serve``: the life of new requests: their prompts in one step, then ``steps`` tokens of each.

Outputs are the float32 logits of every row asked for.  The tokens are given (a decoded token does not depend on the
logits before it), so that a difference in the last bit of one step does not turn into other work in the next.
Weights are random as in ``bench.py`` (the engine's random-weights mode); ``exact`` draws the same ones by the
documented rule and runs the models in float64.
"""
import hashlib
import json
import math
import os
import tempfile

import torch

from nano_vllm_cpp_b200.engine.batch import StepEntry
from nano_vllm_cpp_b200.engine.runner import ModelRunner

STD = 0.014     # of the random weights: with bench.py's 0.02 the experts of the wider models, whose choice rounding may
#                 turn where two are nearly equal, weigh several percent of the stream
PAGE = 16
CONTEXT_STEP = 8192             # tokens a step when a decode case's contexts are put into the cache


# ------------------------------------------------------------------------------------------------ models
def _qwen(layers, hidden, heads, kv, experts, top, inter, shared, vocab, window=0):
    return dict(architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=layers,
                hidden_size=hidden, num_attention_heads=heads, num_key_value_heads=kv, head_dim=128, num_experts=experts,
                num_experts_per_tok=top, moe_intermediate_size=inter, shared_expert_intermediate_size=shared,
                intermediate_size=4 * inter, decoder_sparse_step=1, mlp_only_layers=[], norm_topk_prob=False,
                vocab_size=vocab, rope_theta=1e6, rms_norm_eps=1e-6, max_position_embeddings=32768,
                use_sliding_window=window > 0, sliding_window=window, max_window_layers=0, tie_word_embeddings=False,
                qkv_bias=True)


def _sanesun(layers, W, H, G, ff, vocab):
    latent = {"heads": H, "dim": 128, "vdim": 128, "q_rank": W // 2, "kv_rank": 256, "scale": 128 ** -0.5}
    delta = {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
    window = {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
              "mask": {"size": 1024, "keep_first": 4}, "rot": {"dims": 64, "base": 1e6}}
    kinds = [("latent_attention", latent), ("channel_delta", delta), ("attention", window), ("channel_delta", delta)]
    return {"architecture": "Sanesun", "vocab": vocab, "width": W, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
            "layers": [{"type": kinds[i % 4][0], "mixer": kinds[i % 4][1], "mlp": {"kind": "dense", "ff": ff}}
                       for i in range(layers)]}


def _bizodra(layers, W, H, G, ff, vocab):
    lstm = {"heads": H, "dim": 128, "vdim": 128, "gate_cap": 15.0}
    rot = {"dims": 128, "base": 1e6, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    par = {"left": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": rot},
           "right": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "conv": 4}}
    kinds = [("mlstm", lstm), ("parallel", par)]
    return {"architecture": "Bizodra", "vocab": vocab, "width": W, "norm": {"eps": 1e-6}, "token_side": {"dim": 64},
            "layers": [{"type": kinds[i % 2][0], "mixer": kinds[i % 2][1], "mlp": {"kind": "dense", "ff": ff}}
                       for i in range(layers)]}


MODELS = {  # name -> config.json of that many layers
    "qwen1.5-moe-a2.7b": lambda n: _qwen(n, 2048, 16, 16, 60, 4, 1408, 5632, 151936),
    "qwen2-57b-a14b": lambda n: _qwen(n, 3584, 28, 4, 64, 8, 2560, 20480, 151936),
    "qwen2-moe-s": lambda n: _qwen(n, 1024, 8, 2, 16, 4, 512, 1024, 32000, window=1024),
    "qwen2-moe-m": lambda n: _qwen(n, 2048, 16, 4, 32, 4, 768, 1536, 32000, window=1024),
    "sanesun-s": lambda n: _sanesun(n, 1024, 8, 2, 4096, 32000),
    "sanesun-m": lambda n: _sanesun(n, 2048, 16, 4, 8192, 32000),
    "bizodra-s": lambda n: _bizodra(n, 1024, 8, 2, 4096, 32000),
}


# ------------------------------------------------------------------------------------------------ the cases
def _case(name, model, layers, kind, requests, shortest, longest, steps=1, portion=0, after=0, dtype="bfloat16"):
    c = {"model": model, "layers": layers, "kind": kind, "requests": requests, "shortest": shortest,
         "longest": longest, "steps": steps, "portion": portion, "after": after, "dtype": dtype}
    return dict(c, name=name) if name else c


def listed():
    a27, big = "qwen1.5-moe-a2.7b", "qwen2-57b-a14b"
    return [
        # one user's chat: latency of a reply, nothing to share a launch with
        _case("reply_1", a27, 24, "decode", 1, 2048, 2048, steps=8),
        # the headline batch of bench.py
        _case("replies_8", a27, 24, "decode", 8, 2048, 2048, steps=8),
        # a busy server: many replies whose contexts differ widely
        _case("replies_64_ragged", a27, 8, "decode", 64, 67, 2048, steps=4),
        # grouped-query attention over long contexts, large experts
        _case("replies_16_gqa", big, 3, "decode", 16, 500, 4096, steps=4),
        # short questions that arrive together: small enough for a captured step
        _case("prompts_short", a27, 8, "prompt", 6, 17, 211),
        # the headline prompt of bench.py
        _case("prompt_2048", a27, 24, "prompt", 1, 2048, 2048),
        # a document near the longest sequence, in the portions a scheduler cuts
        _case("prompt_long", a27, 8, "prompt", 1, 7681, 7681, portion=2048),
        # several prompts in one step at the larger layer sizes
        _case("prompts_gqa", big, 3, "prompt", 3, 700, 2500),
        # replies beside a portion of a prompt
        _case("mixed", a27, 8, "mixed", 64, 200, 2048, portion=512, after=1024),
        # the float32 run (its sums have one order whatever the batch is), through a window
        _case("serve_float32", "qwen2-moe-s", 4, "serve", 2, 75, 333, steps=8, dtype="float32"),
        # matrix memories, mixed-head window attention and latent attention around dense layers
        _case("serve_memories", "sanesun-m", 8, "serve", 8, 200, 2048, steps=8),
        # one request of the decoder with gated memories of two kinds beside attention with a sink
        _case("serve_gated", "bizodra-s", 4, "serve", 1, 1500, 1500, steps=8),
    ]


def draw(rng):
    """A case of the listed ones' ranges that costs no more than the largest of them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(_cost(c) for c in listed())
    while True:
        model = rng.choice(["qwen1.5-moe-a2.7b"] * 4 + ["qwen2-57b-a14b"] * 2
                           + ["qwen2-moe-s", "qwen2-moe-m", "sanesun-s", "sanesun-m", "bizodra-s"])
        kind = rng.choice(["decode", "prompt", "mixed", "serve"])
        dtype = "bfloat16"
        if model.startswith("qwen2-moe") and rng.random() < 0.4:
            dtype = "float32"
        if model.startswith(("sanesun", "bizodra", "qwen2-moe")):
            kind = "serve" if kind != "prompt" else kind    # (windows and states: requests run from their start)
        layers = {"qwen1.5-moe-a2.7b": rng.randint(4, 12), "qwen2-57b-a14b": rng.randint(2, 3), "bizodra-s": 4}.get(model, 4 * rng.randint(1, 2))
        longest = size(24, 4096 if kind != "prompt" else 7681) if dtype == "bfloat16" else size(24, 512)
        shortest = max(1, int(longest * rng.choice([1.0, 0.5, 0.1])))
        requests = size(1, 64 if kind in ("decode", "mixed") else 8) if dtype == "bfloat16" else size(1, 4)
        c = _case(None, model, layers, kind, requests, shortest, longest, dtype=dtype,
                  steps=1 if kind in ("prompt", "mixed") else rng.randint(2, 8))
        if kind == "mixed":
            c.update(portion=size(16, 1024), after=16 * rng.randint(0, 128))
        elif kind == "prompt" and rng.random() < 0.3:
            c.update(portion=size(128, 4096))
        tokens = sum(_lengths(c))
        if _cost(c) <= most and (kind in ("decode", "mixed") or tokens <= 16384) and tokens <= 50000:
            return c


def _lengths(case):
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    return [int(round(lo * (hi / lo) ** (i / max(1, n - 1)))) if n > 1 else hi for i in range(n)]


def _plan(case):
    """(tokens in the cache per request before a pass, steps): a step is a list of (request, tokens, whether the
    last one's logits are wanted)."""
    lens = _lengths(case)
    if case["kind"] == "decode":
        return lens, [[(i, 1, True) for i in range(len(lens))] for _ in range(case["steps"])]
    if case["kind"] == "mixed":
        return lens + [case["after"]], [[(i, 1, True) for i in range(len(lens))] + [(len(lens), case["portion"], True)]]
    steps, step, room = [], [], case["portion"] or sum(lens)
    for i, n in enumerate(lens):
        while n:
            k = min(n, room)
            n, room = n - k, room - k
            step.append((i, k, n == 0))
            if room == 0:
                steps, step, room = steps + [step], [], case["portion"] or sum(lens)
    steps += [step] if step else []
    if case["kind"] == "serve":
        steps += [[(i, 1, True) for i in range(len(lens))] for _ in range(case["steps"])]
    return [0] * len(lens), steps


def _tokens(case, seed):
    """Every request's ids: what is in the cache before a pass, then what a pass runs."""
    cached, steps = _plan(case)
    total = list(cached)
    for step in steps:
        for i, n, _ in step:
            total[i] += n
    g = torch.Generator().manual_seed(seed)
    cfg = MODELS[case["model"]](case["layers"])
    return [torch.randint(0, cfg.get("vocab_size") or cfg["vocab"], (n,), generator=g).tolist() for n in total]


# ------------------------------------------------------------------------------------------------ a pass
class State:
    pass


def prepare(case, seed):
    """A runner with its weights, the requests' contexts in its cache, and its step shapes seen (a server warms up
    before it takes requests)."""
    cached, steps = _plan(case)
    ids = _tokens(case, seed)
    s = State()
    with tempfile.TemporaryDirectory() as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(MODELS[case["model"]](case["layers"]), f)
        s.runner = ModelRunner(folder, dtype=case["dtype"], num_pages=sum(len(t) // PAGE + 2 for t in ids), page_size=PAGE,
                               max_requests=len(ids), max_model_len=max(len(t) for t in ids) + PAGE,
                               random_seed=seed, std=STD, norm_std=STD)
    s.cached, s.steps, at = cached, [], list(cached)
    for step in steps:
        entries = []
        for i, n, want in step:
            entries.append(StepEntry(i, ids[i][at[i]:at[i] + n], [n - 1] if want else []))
            at[i] += n
        s.steps.append(entries)

    room, entries = CONTEXT_STEP, []
    for i, n in enumerate(cached):
        done = 0
        while done < n:
            k = min(n - done, room)
            entries.append(StepEntry(i, ids[i][done:done + k], []))
            done, room = done + k, room - k
            if room == 0 or (done == n and i == len(cached) - 1):
                s.runner.step(entries)
                room, entries = CONTEXT_STEP, []
    if entries:
        s.runner.step(entries)
    for _ in range(2):
        run(s)
    return s


def run(s):
    out = []
    for entries in s.steps:
        logits = s.runner.step(entries, check=False)
        if logits.shape[0]:
            out.append(logits.clone())          # (a captured step's logits are valid until the next one)
    for i, n in enumerate(s.cached):
        if n:
            s.runner.manager.commit(i, n)
        else:
            s.runner.close(i)
    return out


# ------------------------------------------------------------------------------------------------ bytes and operations
def _layers(case):
    """Per layer: weights every row uses, (experts, used per row, weights of one), elements cached per token, window,
    multiply-adds per (row, key), floats of state per request."""
    cfg = MODELS[case["model"]](case["layers"])
    rows = []
    if "layers" not in cfg:
        H, D, q, kv = cfg["hidden_size"], 128, cfg["num_attention_heads"] * 128, cfg["num_key_value_heads"] * 128
        shared, E = cfg["shared_expert_intermediate_size"], cfg["num_experts"]
        for _ in range(cfg["num_hidden_layers"]):
            rows.append(((2 * q + 2 * kv) * H + 3 * H * shared + (E + 1) * H,
                         (E, cfg["num_experts_per_tok"], 3 * H * cfg["moe_intermediate_size"]), 2 * kv,
                         cfg["sliding_window"], 2 * q, 0))
        return H, cfg["vocab_size"], rows
    W = cfg["width"]
    for L in cfg["layers"]:
        m, kind, ff = L["mixer"], L["type"], 2 * W * L["mlp"]["ff"] + (128 * W if "token_side" in cfg else 0)
        parts = {"mlstm": 0, "parallel": m.get("left"), "channel_delta": 0}.get(kind, m) or m
        H, G, D = parts["heads"], parts.get("kv_heads", 1), parts["dim"]
        attention, delta = (2 * H + 2 * G) * D * W, (2 * G + 3 * H) * D * W + 2 * H * W
        if kind == "channel_delta":
            row = (delta - H * D * W + 2 * 64 * (W + H * D), 0, 0, 0, H * D * D)
        elif kind == "mlstm":
            row = (5 * H * D * W + 2 * H * W, 0, 0, 0, H * D * D)
        elif kind == "parallel":
            row = (attention + delta, 2 * G * D, 0, 2 * H * D, H * D * D)
        elif kind == "attention":
            row = (attention, 2 * G * D, m["mask"]["size"], 2 * H * D, 0)
        else:
            rq, rk = m["q_rank"], m["kv_rank"]
            row = (rq * (W + H * D) + rk * W + 2 * H * D * rk + H * D * W + H * W, rk, 0, 2 * H * rk, 0)
        rows.append((row[0] + ff, (0, 0, 0)) + row[1:])
    return W, cfg["vocab"], rows


def work(case):
    width, vocab, layers = _layers(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    at, steps = _plan(case)
    at, nbytes, flops = list(at), 0.0, 0.0
    for step in steps:
        T, want = sum(n for _, n, _ in step), sum(w for _, _, w in step)
        nbytes += size * (T * width + vocab * width * (want > 0)) + 4 * want * vocab
        flops += 2.0 * want * vocab * width
        for dense, (E, K, one), kept, window, macs, state in layers:
            nbytes += size * (dense + (E * one * (1 - (1 - K / E) ** T) if E else 0)) + 8 * state * len(step)
            flops += 2.0 * T * (dense + K * one + 3 * state)
            for i, n, _ in step:
                seen = at[i] + n if not window else min(at[i] + n, window + n - 1)
                nbytes += size * kept * (seen + n)
                pairs = sum(min(at[i] + r + 1, window or at[i] + r + 1) for r in range(n))
                flops += 2.0 * macs * pairs
        for i, n, _ in step:
            at[i] += n
    return {"bytes": nbytes, "flops": flops}


def _cost(case):
    w = work(case)
    return w["bytes"] / 6.5e12 + w["flops"] / (1.6e15 if case["dtype"] == "bfloat16" else 6e13)


def tolerance(case):
    """Against float64 the engine is off by 1.2e-6 in float32, by 0.005 to 0.006 in bfloat16 (0.008 where the matrix
    memories of Bizodra divide by a small sum); two correct ones differ by about 1.4 times that."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 3e-2 if case["model"].startswith("bizodra") else 2e-2}


# ------------------------------------------------------------------------------------------------ float64
class Weights:
    """The engine's random weights by their documented rule: a function of seed, name and element index."""

    def __init__(self, seed):
        self.seed = seed

    def __call__(self, name, *shape, mean=0.0):
        n, dev = math.prod(shape), "cuda"
        signed = lambda v: v - (1 << 64) if v >> 63 else v                                   # noqa: E731
        shift = lambda x, k: (x >> k) & ((1 << (64 - k)) - 1)                                # noqa: E731
        key = int.from_bytes(hashlib.sha256(f"{self.seed}:{name}".encode()).digest()[:8], "little")
        out = torch.empty(n, dtype=torch.float64, device=dev)
        for lo in range(0, n, 1 << 26):
            hi = min(n, lo + (1 << 26))
            c = torch.arange(lo, hi, device=dev) * signed(0x9E3779B97F4A7C15) + signed(key)
            total = torch.zeros_like(c)
            for turn in (0, 0xD6E8FEB86659FD93, 0xA0761D6478BD642F):
                z = c ^ signed(turn)
                z = (z ^ shift(z, 30)) * signed(0xBF58476D1CE4E5B9)
                z = (z ^ shift(z, 27)) * signed(0x94D049BB133111EB)
                z = z ^ shift(z, 31)
                for k in (0, 16, 32, 48):
                    total += shift(z, k) & 0xFFFF if k else z & 0xFFFF
            z = (total - 393210).float() * (1.0 / 65536.0)
            out[lo:hi] = (mean + z * torch.tensor(STD, device=dev)).bfloat16().double()
        return out.view(*shape)


def _rms(x, eps=1e-6):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, rot, pos, neighbours=False, sign=1.0):
    """x [T, heads, D]: pairs of the first ``dims`` elements turned by their positions; ``scaling`` stretches the slow
    ones."""
    dims, base, sc, amp = rot["dims"], rot["base"], rot.get("scaling"), 1.0
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], device=x.device).double()
    if sc:
        lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * sc[c])) / (2 * math.log(base)) for c in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = ((torch.arange(dims // 2, device=x.device).double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, amp = f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1
    ang = sign * pos.double()[:, None, None] * f
    c, s = ang.cos() * amp, ang.sin() * amp
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :dims // 2], x[..., dims // 2:dims])
    both = (a * c - b * s, b * c + a * s)
    turned = torch.stack(both, -1).flatten(-2) if neighbours else torch.cat(both, -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _attend(q, k, v, scale, window=0, keep=0, sink=None):
    """Causal attention of one sequence: q [T, H, D], k and v [T, G, ...]; ``sink`` [H] adds a score without a value."""
    T, H = q.shape[:2]
    k, v = (t.repeat_interleave(H // t.shape[1], 1).transpose(0, 1) for t in (k, v))
    q, out, rows = q.transpose(0, 1), [], max(1, (1 << 27) // (H * T))
    for lo in range(0, T, rows):
        hi = min(T, lo + rows)
        s = q[:, lo:hi] @ k[:, :hi].transpose(1, 2) * scale
        i, j = torch.arange(lo, hi, device=q.device)[:, None], torch.arange(hi, device=q.device)[None]
        seen = (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, hi - lo, 1)], -1)
        p = s.softmax(-1)
        out.append((p[..., :hi] @ v[:, :hi]).transpose(0, 1))
    return torch.cat(out)


def _mixture(h, K, router, expert):
    """Sum over the K best experts of softmax(router h), weighted; ``expert(e, rows)``."""
    w, idx = (h @ router.T).softmax(-1).topk(K, -1)
    y = torch.zeros_like(h)
    for e in idx.unique().tolist():
        rows, place = (idx == e).nonzero(as_tuple=True)
        y[rows] += w[rows, place, None] * expert(e, h[rows])
    return y


def _side_by_side(spans, step, *rows):
    """Runs ``step(n, t, *rows of the tokens)`` for all sequences side by side, token by token."""
    longest, dev = max(b - a for a, b in spans), rows[0].device
    at = torch.stack([torch.arange(longest, device=dev).clamp(max=b - a - 1) + a for a, b in spans], 1)
    out = torch.empty_like(rows[0])
    for t in range(longest):
        o = step(*(x[at[t]] for x in rows))
        live = [n for n, (a, b) in enumerate(spans) if t < b - a]
        out[at[t][live]] = o[live]
    return out


def _delta(h, w, p, m, spans, by_channel):
    """The delta rule; ``by_channel``: a decay per head and key channel and a sigmoid gate, each through a low-rank
    pair, instead of a decay per head and a silu gate."""
    H, G, D, W = m["heads"], m["kv_heads"], m["dim"], h.shape[1]
    silu = torch.nn.functional.silu

    def conv(name, heads):
        x, taps = h @ w(p + name, heads * D, W).T, w(p + name + ".conv", heads * D, 4)
        parts = []
        for a, b in spans:
            y = torch.cat([x.new_zeros(3, x.shape[1]), x[a:b]])
            parts.append(sum(y[d:d + b - a] * taps[:, d] for d in range(4)))
        return silu(torch.cat(parts)).view(-1, heads, D).repeat_interleave(H // heads, 1)

    q, k, v = conv("q", G), conv("k", G), conv("v", H)
    q, k = (x / ((x * x).sum(-1, keepdim=True) + 1e-6).sqrt() for x in (q, k))
    beta = (h @ w(p + "b", H, W).T).sigmoid()[..., None]
    if by_channel:
        decay = (h @ w(p + "a1", 64, W).T) @ w(p + "a2", H * D, 64).T
        gate = ((h @ w(p + "g1", 64, W).T) @ w(p + "g2", H * D, 64).T).sigmoid().view(-1, H, D)
    else:
        decay, gate = h @ w(p + "a", H, W).T, silu(h @ w(p + "g", H * D, W).T).view(-1, H, D)
    decay = torch.exp(-torch.nn.functional.softplus(decay)).view(-1, H, D if by_channel else 1)
    S = h.new_zeros(len(spans), H, D, D)

    def step(v, q, k, beta, g):
        S.mul_(g[..., None])
        u = beta * (v - (S * k[..., None]).sum(-2))
        S.add_(k[..., None] * u[..., None, :])
        return (S * q[..., None]).sum(-2)
    out = _side_by_side(spans, step, v, q * D ** -0.5, k, beta, decay)
    return (_rms(out) * w(p + "norm", D, mean=1.0) * gate).flatten(1) @ w(p + "o", W, H * D).T


def _mlstm(h, w, p, m, spans):
    H, D, W, cap = m["heads"], m["dim"], h.shape[1], m["gate_cap"]
    q, k, v = ((h @ w(p + c, H * D, W).T).view(-1, H, D) for c in "qkv")
    gi, gf = (cap * torch.tanh((h @ w(p + c, H, W).T + w(p + c + ".b", H)) / cap) for c in "if")
    S, n, top = h.new_zeros(len(spans), H, D, D), h.new_zeros(len(spans), H, D), h.new_zeros(len(spans), H)

    def step(v, q, k, gi, gf):
        new = torch.maximum(gf + top, gi)
        keep, take = torch.exp(gf + top - new)[..., None], torch.exp(gi - new)[..., None]
        S.mul_(keep[..., None]).add_((take * k)[..., None] * v[..., None, :])
        n.mul_(keep).add_(take * k)
        top.copy_(new)
        den = torch.maximum((n * q).sum(-1).abs(), torch.exp(-new)) + 1e-6
        return (S * q[..., None]).sum(-2) / den[..., None]
    out = _side_by_side(spans, step, v, q * D ** -0.5, k, gi, torch.nn.functional.logsigmoid(gf))
    y = _rms(out).flatten(1) * w(p + "norm", H * D, mean=1.0) * (h @ w(p + "g", H * D, W).T).sigmoid()
    return y @ w(p + "o", W, H * D).T


def _forward(case, w, ids, wanted):
    """Logits of the rows ``wanted`` (numbers over all sequences one after the other), float64."""
    cfg = MODELS[case["model"]](case["layers"])
    ends = torch.tensor([len(t) for t in ids]).cumsum(0).tolist()
    spans = [(e - len(t), e) for e, t in zip(ends, ids)]
    pos = torch.cat([torch.arange(len(t)) for t in ids]).cuda()
    flat = torch.tensor([t for s in ids for t in s], device="cuda")

    def each(f, *xs):
        return torch.cat([f(*(x[a:b] for x in xs)) for a, b in spans])

    if "layers" not in cfg:
        W, H, G, V = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["vocab_size"]
        I, SI = cfg["moe_intermediate_size"], cfg["shared_expert_intermediate_size"]
        x = w("model.embed_tokens.weight", V, W)[flat]
        silu = torch.nn.functional.silu
        for n in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{n}."
            a, f = p + "self_attn.", p + "mlp."
            h = _rms(x) * w(p + "input_layernorm.weight", W, mean=1.0)
            q, k, v = ((h @ w(f"{a}{c}_proj.weight", r * 128, W).T + w(f"{a}{c}_proj.bias", r * 128)).view(-1, r, 128)
                       for c, r in (("q", H), ("k", G), ("v", G)))
            rot = {"dims": 128, "base": cfg["rope_theta"]}
            q, k = _turn(q, rot, pos), _turn(k, rot, pos)
            y = each(lambda q, k, v: _attend(q, k, v, 128 ** -0.5, cfg["sliding_window"]), q, k, v)
            x = x + y.flatten(1) @ w(a + "o_proj.weight", W, H * 128).T
            h = _rms(x) * w(p + "post_attention_layernorm.weight", W, mean=1.0)

            def glu(r, name, ff):
                up = silu(r @ w(name + "gate_proj.weight", ff, W).T) * (r @ w(name + "up_proj.weight", ff, W).T)
                return up @ w(name + "down_proj.weight", W, ff).T
            x = x + (h @ w(f + "shared_expert_gate.weight", 1, W).T).sigmoid() * glu(h, f + "shared_expert.", SI)
            x = x + _mixture(h, cfg["num_experts_per_tok"], w(f + "gate.weight", cfg["num_experts"], W),
                             lambda e, r: glu(r, f"{f}experts.{e}.", I))
        h = _rms(x[wanted]) * w("model.norm.weight", W, mean=1.0)
        return h @ w("lm_head.weight", V, W).T

    W, V = cfg["width"], cfg["vocab"]
    bizodra = cfg["architecture"] == "Bizodra"
    x = w("embed", V, W)[flat]
    for n, L in enumerate(cfg["layers"]):
        m, kind, p, f = L["mixer"], L["type"], f"l{n}.mix.", f"l{n}.mlp."
        h = x if bizodra else _rms(x) * w(f"l{n}.norm1", W, mean=1.0)
        if kind == "channel_delta":
            y = _delta(h, w, p, m, spans, True)
        elif kind == "mlstm":
            y = _mlstm(h, w, p, m, spans)
        elif kind == "latent_attention":
            H, D, rq, rk = m["heads"], m["dim"], m["q_rank"], m["kv_rank"]
            q = (_rms(h @ w(p + "dq", rq, W).T) * w(p + "dq.norm", rq, mean=1.0)) @ w(p + "uq", H * D, rq).T
            c = _rms(h @ w(p + "dkv", rk, W).T) * w(p + "dkv.norm", rk, mean=1.0)
            k, v = c @ w(p + "uk", H * D, rk).T, c @ w(p + "uv", H * D, rk).T
            y = each(lambda *t: _attend(*t, m["scale"]), *(t.view(-1, H, D) for t in (q, k, v)))
            y = (y * (h @ w(p + "g", H, W).T).sigmoid()[..., None]).flatten(1) @ w(p + "o", W, H * D).T
        else:
            a, pa = (m["left"], p + "left.") if bizodra else (m, p)
            H, G, D, rot = a["heads"], a["kv_heads"], a["dim"], a["rot"]
            q, k, v = ((h @ w(pa + c, r * D, W).T + w(pa + c + ".b", r * D)).view(-1, r, D)
                       for c, r in (("q", H), ("k", G), ("v", G)))
            sink = torch.zeros(H, device="cuda").double()
            if bizodra:         # normed heads, neighbouring pairs turned, a sink of score zero; a memory beside it
                q, k = (_turn(_rms(t) * w(f"{pa}{c}.norm", D, mean=1.0), rot, pos, True) for t, c in ((q, "q"), (k, "k")))
                y = each(lambda *t: _attend(*t, a["scale"], sink=sink), q, k, v).flatten(1)
                y = _rms(y @ w(pa + "o", W, H * D).T + w(pa + "o.b", W)) * w(p + "left.out", W, mean=1.0)
                r = _rms(_delta(h, w, p + "right.", m["right"], spans, False)) * w(p + "right.out", W, mean=1.0)
                y = 0.5 * (y + r)
            else:               # kept first tokens, values turned and turned back; heads mixed by the unit matrix
                whole = dict(rot, dims=D)
                q, k, v = _turn(q, rot, pos), _turn(k, rot, pos), _turn(v, whole, pos)
                mask = m["mask"]
                y = each(lambda *t: _attend(*t, m["scale"], mask["size"], mask["keep_first"], sink), q, k, v)
                y = _turn(y, whole, pos, sign=-1.0).flatten(1) @ w(p + "o", W, H * D).T
        if bizodra:
            x = x + _rms(y) * (1 + w(f"l{n}.norm1", W))
            h = x
        u = h @ w(f + "up", L["mlp"]["ff"], W).T
        if bizodra:
            u = torch.nn.functional.gelu(u)
        else:
            a, b = torch.nn.functional.softplus(w(f + "act", 2)).unbind()
            u = torch.where(u > 0, a * u * u, (0.5 + b) * (torch.expm1(u.clamp(max=0)) - u)) + 0.5 * u
        z = u @ w(f + "down", W, L["mlp"]["ff"]).T
        if not bizodra:
            x = x + y + z
            continue
        x, f, r = x + _rms(z) * (1 + w(f"l{n}.norm2", W)), f"l{n}.side.", cfg["token_side"]["dim"]
        row = w("side.embed", V, r * len(cfg["layers"]))[flat][:, n * r:(n + 1) * r]
        gate = torch.nn.functional.gelu(x @ w(f + "gate", r, W).T, approximate="tanh") * row
        x = x + _rms(gate @ w(f + "proj", W, r).T) * w(f + "norm", W, mean=1.0)
    return (_rms(x[wanted]) * w("final.norm", W, mean=1.0)) @ w("head", V, W).T


@torch.no_grad()
def exact(case, seed):
    ids = _tokens(case, seed)
    cached, steps = _plan(case)
    first = [sum(len(t) for t in ids[:i]) for i in range(len(ids))]
    at, rows = list(cached), []
    for step in steps:
        got = []
        for i, n, want in step:
            at[i] += n
            got += [first[i] + at[i] - 1] if want else []
        rows += [got] if got else []
    logits = _forward(case, Weights(seed), ids, torch.tensor([r for got in rows for r in got], device="cuda"))
    return list(logits.split([len(got) for got in rows]))
