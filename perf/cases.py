"""What the engine is measured on: steps of a served model at the sizes that ``bench.py`` names, through the public entry
points (``Engine``, ``StepEntry``, ``Sampler``).

A case is a dict of plain values.  ``kind`` says what one pass is:

  decode    one token for each of ``requests`` requests that hold up to ``context`` tokens (from ``shortest`` on, where given)
  prefill   ``requests`` whole prompts in one step, the logits of their last tokens
  mixed     a prompt portion of ``portion`` tokens beside one token for each of ``requests`` requests: a loaded server's step
  replay    ``context`` given tokens in one step in 32 bits, the logits of every one of them: how a model is verified
  serve     whole requests: their prompts in one step, then ``steps`` tokens each, then closed
  sample    the next token of ``requests`` rows of logits under the parameters that requests bring

Weights are random, drawn on the device as ``random_model_on_device`` does; token ids are uniform in the vocabulary.  The designs
with routed experts are left out: two correct evaluations in 16 bits choose other experts for some tokens.
"""
import hashlib
import math
import random

import torch

from lightllm_b200 import Engine, SamplingParams, StepEntry
from lightllm_b200.models import random_model_on_device
from lightllm_b200.sampling import Sampler

PAGE = 16
ROOM = 2048          # tokens that a decoding request may add before it ends and another takes its place
STEP_TOKENS = 8192   # the tokens that a step may bring

VOCAB = 151936
_QWEN2 = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": VOCAB, "rope_theta": 1000000.0,
          "rms_norm_eps": 1e-6, "tie_word_embeddings": True, "max_position_embeddings": 32768, "use_sliding_window": False,
          "hidden_act": "silu"}
CONFIGS = {
    "0.5b": dict(_QWEN2, num_hidden_layers=24, hidden_size=896, num_attention_heads=14, num_key_value_heads=2, head_dim=64,
                 intermediate_size=4864),
    "1.5b": dict(_QWEN2, num_hidden_layers=28, hidden_size=1536, num_attention_heads=12, num_key_value_heads=2, head_dim=128,
                 intermediate_size=8960),
    # (half of its layers: the differences of two evaluations in 16 bits grow from layer to layer at this width, to 4 % after all 28)
    "7b": dict(_QWEN2, num_hidden_layers=14, hidden_size=3584, num_attention_heads=28, num_key_value_heads=4, head_dim=128,
               intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False),
}


def _laralix():
    """The design at the 0.5B width with six layer runs, as ``bench.py --design laralix`` has it."""
    heads, hd, width, ff = 14, 64, 896, 4864
    left = {"heads": heads, "kv_heads": 2, "dim": hd, "vdim": hd, "scale": hd ** -0.5}
    layers = [
        ("parallel", {"left": {**left, "softcap": 50.0, "mask": {"size": 1024}},
                      "right": {"heads": heads, "kv_heads": heads, "dim": hd, "vdim": hd, "conv": 4}}),
        ("parallel_2", {"left": {**left, "mask": {"size": 1024, "keep_first": 4}}, "left_scale": 1.1, "right_scale": 0.8,
                        "right": {"heads": heads, "dim": hd, "vdim": hd, "tau": 12.0, "decay_rank": 64}}),
        ("latent_attention", {"heads": heads, "dim": hd, "rot_dim": 32, "vdim": hd, "q_rank": width // 2, "kv_rank": 256,
                              "scale": (hd + 32) ** -0.5, "rot": {"dims": 32, "base": 50000.0}}),
    ]
    return {"architecture": "Laralix", "vocab": VOCAB, "width": width, "embedding": {"scale": 6.0}, "norm": {"eps": 1e-5},
            "logit_scale": 0.5, "loop": {"start": 0, "stop": 3, "times": 2},
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": ff}} for t, m in layers]}


CONFIGS["laralix"] = _laralix()


def listed():
    return [
        # one user at a terminal: nothing hides a launch or a wait
        {"name": "decode-0.5b-1", "kind": "decode", "model": "0.5b", "requests": 1, "context": 2048},
        # the benchmark's batch, and its largest
        {"name": "decode-0.5b-8", "kind": "decode", "model": "0.5b", "requests": 8, "context": 2048},
        {"name": "decode-0.5b-64", "kind": "decode", "model": "0.5b", "requests": 64, "context": 2048},
        # a server's decoding step: an odd batch whose requests are at different places (heads of 128)
        {"name": "decode-1.5b-27-ragged", "kind": "decode", "model": "1.5b", "requests": 27, "context": 4001, "shortest": 65},
        # the widest model, bound by its weights
        {"name": "decode-7b-8", "kind": "decode", "model": "7b", "requests": 8, "context": 2048},
        # the benchmark's prompt
        {"name": "prefill-0.5b-2048", "kind": "prefill", "model": "0.5b", "requests": 1, "context": 2048},
        # several prompts of odd lengths in one step of the widest model: the most arithmetic
        {"name": "prefill-7b-ragged", "kind": "prefill", "model": "7b", "requests": 5, "context": 1103, "shortest": 77},
        # a long portion under the chunked budget of 2,048 tokens beside the decoding requests
        {"name": "mixed-1.5b-1999", "kind": "mixed", "model": "1.5b", "requests": 31, "context": 1537, "shortest": 65, "portion": 1999},
        # a short message coming in while others decode
        {"name": "mixed-0.5b-19", "kind": "mixed", "model": "0.5b", "requests": 13, "context": 1290, "shortest": 131, "portion": 19},
        # verification in true 32 bits, logits everywhere
        {"name": "replay-0.5b-fp32", "kind": "replay", "model": "0.5b", "dtype": "float32", "requests": 1, "context": 389},
        # requests from their prompts to their last token in a design of attention beside recurrences
        {"name": "serve-laralix-4", "kind": "serve", "model": "laralix", "requests": 4, "context": 811, "shortest": 90, "steps": 24},
        # the sampler's share of every served step: the default parameters beside the filters
        {"name": "sample-64", "kind": "sample", "requests": 64, "vocab": VOCAB},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mixed", "mixed", "replay", "serve", "sample"])
    if kind == "sample":
        return {"kind": kind, "requests": _log_int(rng, 1, 64), "vocab": rng.choice([VOCAB, VOCAB, 152064, 32000 + rng.randrange(1000)])}
    if kind == "replay":
        return {"kind": kind, "model": "0.5b", "dtype": "float32", "requests": 1, "context": _log_int(rng, 5, 400)}
    if kind == "serve":
        c = {"kind": kind, "model": "laralix", "requests": _log_int(rng, 1, 8), "context": _log_int(rng, 33, 820), "steps": rng.randint(4, 24)}
        return dict(c, shortest=rng.randint(17, c["context"])) if c["requests"] > 1 else c
    model = rng.choice(["0.5b", "0.5b", "1.5b", "1.5b", "7b"])
    held = {"0.5b": 1 << 17, "1.5b": 1 << 15, "7b": 1 << 14}[model]          # tokens that the requests hold together, at most
    if kind == "prefill":
        n = _log_int(rng, 1, 6)
        c = {"kind": kind, "model": model, "requests": n, "context": _log_int(rng, 40, 2048 // n if model == "7b" else 4096 // n)}
        return dict(c, shortest=rng.randint(17, c["context"])) if n > 1 and rng.random() < 0.7 else c
    c = {"kind": kind, "model": model, "requests": _log_int(rng, 1, 64 if kind == "decode" else 31)}
    c["context"] = _log_int(rng, 64, min(4096, held // c["requests"]))
    if c["requests"] > 1 and rng.random() < 0.7:
        c["shortest"] = rng.randint(33, c["context"])
    if kind == "mixed":
        c["portion"] = _log_int(rng, 3, 2000)
    return c


def _lengths(case):
    """How many tokens each request holds or brings: from ``shortest`` to ``context``, evenly over their logarithm and then
    moved a little, in no order."""
    n, high = case["requests"], case["context"]
    low = case.get("shortest", high)
    r = random.Random(n * 1000003 + high)
    out = [high] + [max(low, min(high, int(low * (high / low) ** (i / max(1, n - 1))) - (r.randrange(7) if low < high else 0)))
                    for i in range(n - 1)]
    r.shuffle(out)
    return out


def _dtype(case):
    return case.get("dtype", "bfloat16")


def _tokens(case, seed):
    """Every request's tokens: what it holds or brings, then those that it goes on with; and a mixed step's portion."""
    r = random.Random(seed * 7919 + 17)
    vocab = _vocab(case)
    more = {"decode": ROOM, "mixed": ROOM, "serve": case.get("steps", 0)}.get(case["kind"], 0)
    rows = [[r.randrange(vocab) for _ in range(n + more)] for n in _lengths(case)]
    return rows, [r.randrange(vocab) for _ in range(case.get("portion", 0))]


def _vocab(case):
    if "model" not in case:
        return case["vocab"]
    cfg = CONFIGS[case["model"]]
    return cfg.get("vocab_size") or cfg["vocab"]


def _fill(state):
    """Opens the requests and brings their held tokens, as many a step as a step may have."""
    engine, core = state["engine"], state["engine"].core
    for i in range(len(state["held"])):
        if core.is_open(i):
            core.close(i)
        core.open(i)
    batch, room = [], STEP_TOKENS
    for i, n in enumerate(state["held"]):
        if n > room:
            engine.step(batch)
            batch, room = [], STEP_TOKENS
        batch.append(StepEntry(i, state["tokens"][i][:n], []))
        room -= n
    engine.step(batch)
    state["at"] = 0


def prepare(case, seed):
    device = torch.device("cuda:0")
    if case["kind"] == "sample":
        g = torch.Generator(device=device)
        g.manual_seed(seed)
        logits = torch.randn((case["requests"], case["vocab"]), generator=g, device=device) * 3.0
        some = [SamplingParams(temperature=1.0), SamplingParams(temperature=0.7, top_p=0.9), SamplingParams(temperature=0.8, top_k=40),
                SamplingParams(temperature=1.0, min_p=0.05), SamplingParams(temperature=0.6, top_k=20, top_p=0.95),
                SamplingParams(temperature=0.0)]
        params = [SamplingParams(**{**vars(some[i % len(some)]), "seed": seed + i}) for i in range(case["requests"])]
        return {"kind": "sample", "sampler": Sampler(device), "logits": logits, "params": params, "ids": list(range(case["requests"]))}
    model = random_model_on_device(dict(CONFIGS[case["model"]]), seed, _dtype(case), device)
    lengths = _lengths(case)
    tokens, portion = _tokens(case, seed)
    longest = max(max(len(t) for t in tokens), len(portion)) + 1
    pages = sum(-(-(len(t) + 1) // PAGE) for t in tokens) + -(-len(portion) // PAGE) + 1
    engine = Engine(None, dtype=_dtype(case), max_seq_len=longest, max_batch_tokens=STEP_TOKENS, page_size=PAGE, num_pages=pages,
                    max_seqs=64, chunk_size=2048, model=model)
    state = {"kind": case["kind"], "engine": engine, "held": lengths, "tokens": tokens, "portion": portion}
    if case["kind"] in ("decode", "mixed"):
        _fill(state)
    return state


def run(state):
    kind = state["kind"]
    if kind == "sample":
        return state["sampler"].sample_device(state["logits"], state["ids"], state["params"])
    engine, held, tokens = state["engine"], state["held"], state["tokens"]
    core = engine.core
    if kind in ("decode", "mixed"):
        if state["at"] == ROOM:
            _fill(state)
        at = state["at"]
        state["at"] = at + 1
        entries = [StepEntry(i, [t[n + at]], [0]) for i, (t, n) in enumerate(zip(tokens, held))]
        if kind == "decode":
            return engine.step(entries)
        core.open("new")
        logits = engine.step(entries + [StepEntry("new", state["portion"], [len(state["portion"]) - 1])])
        core.close("new")
        return logits
    for i in range(len(held)):
        core.open(i)
    if kind == "replay":
        out = engine.step([StepEntry(i, t, list(range(len(t)))) for i, t in enumerate(tokens)])
    else:
        out = engine.step([StepEntry(i, t[:n], [n - 1]) for i, (t, n) in enumerate(zip(tokens, held))])
    if kind == "serve":
        out = [out]
        for at in range(len(tokens[0]) - held[0]):
            out.append(engine.step([StepEntry(i, [t[n + at]], [0]) for i, (t, n) in enumerate(zip(tokens, held))]))
    for i in range(len(held)):
        core.close(i)
    return out


# ---------------------------------------------------------------------------------------------------------------------

def _sizes(case):
    """(weights of the layers, weights of the head, bytes of cache a token, attention operations a (query, key) pair)."""
    c = CONFIGS[case["model"]]
    if case["model"] == "laralix":
        width, ff = c["width"], 4864
        mixers = (width * (896 * 2 + 256) + width * 896 * 5) + (width * (896 * 2 + 128) + width * 896 * 5 + 128 * 896) + (448 * (width + 1344) + 288 * width + 512 * 896 + 896 * 896)
        return mixers + 3 * 3 * width * ff, width * c["vocab"], 2 * 2 * (256 + 128 + 288), 4 * 896 * 6
    D, I, H, G, hd = c["hidden_size"], c["intermediate_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    layers, e = c["num_hidden_layers"], 4 if _dtype(case) == "float32" else 2
    return layers * (D * (H + 2 * G) * hd + H * hd * D + 3 * D * I), D * c["vocab_size"], layers * 2 * G * hd * e, layers * 4 * H * hd


def work(case):
    if case["kind"] == "sample":
        return {"bytes": case["requests"] * case["vocab"] * 4 + 4 * case["requests"], "flops": 4 * case["requests"] * case["vocab"]}
    layers, head, token, pair = _sizes(case)
    kind, n, lengths = case["kind"], case["requests"], _lengths(case)
    e = 4 if _dtype(case) == "float32" else 2
    whole = sum(x * (x + 1) // 2 for x in lengths)
    if kind in ("decode", "mixed"):
        p = case.get("portion", 0)
        rows, want, pairs, cached = n + p, n + (p > 0), sum(lengths) + n + p * (p + 1) // 2, sum(lengths) + n + p
        steps = 1
    elif kind == "serve":
        steps = 1 + case["steps"]
        rows, want = sum(lengths) + n * case["steps"], n * steps
        pairs, cached = whole + case["steps"] * sum(lengths), sum(lengths) * steps
    else:
        rows, pairs, cached, steps = sum(lengths), whole, sum(lengths), 1
        want = sum(lengths) if kind == "replay" else n
    runs = 2 if case["model"] == "laralix" else 1          # the loop runs every layer twice
    return {"bytes": steps * e * (layers + head) + cached * token + want * _vocab(case) * 4,
            "flops": 2 * runs * layers * rows + 2 * head * want + pair * pairs}


def tolerance(case):
    """Measured: the 32-bit replay is 3e-6 off 64 bits, the 16-bit cases 0.007 to 0.02; the same steps through other kernels of the
    engine (sums in another order) differ by up to 0.02."""
    if case["kind"] == "sample":
        return "exact"
    if _dtype(case) == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.03}


# ------------------------------------------------------------------------------------------- the same in 64 bits

def _weight(case, seed, name, shape, std, one=False):
    """The tensor of that name as the random-weights mode draws it on the device, in 64 bits."""
    device = torch.device("cuda:0")
    g = torch.Generator(device=device)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:8], "little") & 0x7FFF_FFFF_FFFF_FFFF)
    t = torch.randn(shape, generator=g, dtype=torch.float32, device=device) * std
    if one:
        t += 1.0
    return t.to(torch.float32 if _dtype(case) == "float32" else torch.bfloat16).double()


def _rms(x, eps, w=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, scale, size=None, keep=0, softcap=None, slope=None, plus_one=False):
    """q [T, H, d] at the positions of its rows, k and v [T, G, .]; ``size`` a window, ``keep`` first tokens seen beside it, ``slope`` [H]
    takes a head's slope times the distance off the score, ``plus_one`` adds one to the denominator."""
    T, H, _ = q.shape
    share = H // k.shape[1]
    out = torch.empty(T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for a in range(0, T, 512):          # (blocks of rows: the scores of all would not fit)
        b = min(T, a + 512)
        far = torch.arange(a, b, device=q.device)[:, None] - torch.arange(b, device=q.device)[None, :]
        seen = far >= 0
        if size is not None:
            seen &= (far < size) | (torch.arange(b, device=q.device) < keep)
        s = torch.einsum("ihd,jhd->hij", q[a:b], k[:b].repeat_interleave(share, 1)) * scale
        if softcap is not None:
            s = softcap * torch.tanh(s / softcap)
        if slope is not None:
            s = s - slope[:, None, None] * far
        s = s.masked_fill(~seen, -math.inf)
        m = s.max(-1, keepdim=True).values
        if plus_one:
            m = m.clamp(min=0.0)
        p = torch.exp(s - m)
        p = p / (p.sum(-1, keepdim=True) + (torch.exp(-m) if plus_one else 0.0))
        out[a:b] = torch.einsum("hij,jhe->ihe", p, v[:b].repeat_interleave(share, 1))
    return out


def _turn(x, angle, adjacent):
    """Rotates pairs (2i, 2i + 1), or (i, i + half), of x [T, heads, n] by angle [T, n / 2]."""
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    if adjacent:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _angles(T, n, base):
    i = torch.arange(n // 2, dtype=torch.float64, device="cuda:0")
    return torch.arange(T, dtype=torch.float64, device="cuda:0")[:, None] * base ** (-2.0 * i / n)


def _exact_qwen2(case, seed, rows, want):
    """Logits at ``want[i]`` of every sequence ``rows[i]``, all of them layer by layer."""
    c = CONFIGS[case["model"]]
    D, I, H, G, hd, eps = (c[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim", "rms_norm_eps"))
    w = lambda name, *shape: _weight(case, seed, name, shape, 0.02)  # noqa: E731
    norm = lambda name: _weight(case, seed, name, (D,), 0.01, one=True)  # noqa: E731
    table = w("model.embed_tokens.weight", c["vocab_size"], D)
    xs = [table[torch.tensor(r, device=table.device)] for r in rows]
    angle = _angles(max(len(r) for r in rows), hd, c["rope_theta"])
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a, m = p + "self_attn.", p + "mlp."
        n1, n2 = norm(p + "input_layernorm.weight"), norm(p + "post_attention_layernorm.weight")
        q, k, v = (torch.cat([w(f"{a}{x}_proj.weight", n, D), w(f"{a}{x}_proj.bias", n)[:, None]], 1) for x, n in (("q", H * hd), ("k", G * hd), ("v", G * hd)))
        o = w(a + "o_proj.weight", D, H * hd)
        gate, up, down = w(m + "gate_proj.weight", I, D), w(m + "up_proj.weight", I, D), w(m + "down_proj.weight", D, I)
        for j, x in enumerate(xs):
            T = x.shape[0]
            h = torch.cat([_rms(x, eps, n1), torch.ones(T, 1, dtype=x.dtype, device=x.device)], 1)
            turned = [_turn((h @ y.T).view(T, -1, hd), angle[:T], False) for y in (q, k)]
            x = x + _attend(*turned, (h @ v.T).view(T, G, hd), hd ** -0.5).reshape(T, H * hd) @ o.T
            h = _rms(x, eps, n2)
            xs[j] = x + (_silu(h @ gate.T) * (h @ up.T)) @ down.T
    n = norm("model.norm.weight")
    head = table if c["tie_word_embeddings"] else w("lm_head.weight", c["vocab_size"], D)
    return torch.cat([_rms(x[torch.tensor(at, device=x.device)], eps, n) @ head.T for x, at in zip(xs, want)])


def _conv(u, w):
    taps = w.shape[1]
    u = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return sum(w[:, j] * u[j: j + u.shape[0] - taps + 1] for j in range(taps))


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _laralix_parallel(h, w, p, m, eps):
    T = h.shape[0]
    a, b = m["left"], m["right"]
    H, G, d, wide = a["heads"], a["kv_heads"], a["dim"], h.shape[1]
    one = lambda name, n: w(name, (n,), 0.1, one=True)  # noqa: E731
    lin = lambda name, n: h @ w(name, (n, wide), 0.02).T  # noqa: E731
    slope = torch.tensor([2.0 ** (-8.0 * (i + 1) / H) for i in range(H)], dtype=h.dtype, device=h.device)
    q, k = (_rms(lin(f"{p}.left.{x}", n * d).view(T, n, d), eps, one(f"{p}.left.{x}.norm", d)) for x, n in (("q", H), ("k", G)))
    left = _attend(q, k, lin(f"{p}.left.v", G * d).view(T, G, d), a["scale"], a["mask"]["size"], 0, a["softcap"], slope, True)
    left = left.reshape(T, H * d) @ w(f"{p}.left.o", (wide, H * d), 0.02).T
    H, d = b["heads"], b["dim"]
    q, k, v = (_silu(_conv(lin(f"{p}.right.{x}", H * d), w(f"{p}.right.{x}.conv", (H * d, b["conv"]), 0.5))).view(T, H, d) for x in "qkv")
    q, k, beta = _unit(q) * d ** -0.5, _unit(k), torch.sigmoid(lin(f"{p}.right.b", H))
    z = lin(f"{p}.right.a", H) + w(f"{p}.right.dt_bias", (H,), 0.5)
    decay = torch.exp(-torch.exp(w(f"{p}.right.A_log", (H,), 0.5)) * torch.nn.functional.softplus(z))
    S, out = h.new_zeros(H, d, d), torch.empty_like(v)
    for t in range(T):
        S = decay[t][:, None, None] * S
        S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t])))[:, None]
        out[t] = torch.einsum("hde,hd->he", S, q[t])
    out = _rms(out, eps, one(f"{p}.right.norm", d)) * _silu(lin(f"{p}.right.g", H * d)).view(T, H, d)
    right = out.reshape(T, H * d) @ w(f"{p}.right.o", (wide, H * d), 0.02).T
    return 0.5 * (_rms(left, eps, one(f"{p}.left.out", wide)) + _rms(right, eps, one(f"{p}.right.out", wide)))


def _laralix_parallel_2(h, w, p, m, eps):
    T = h.shape[0]
    a, b = m["left"], m["right"]
    H, G, d, wide = a["heads"], a["kv_heads"], a["dim"], h.shape[1]
    one = lambda name, n: w(name, (n,), 0.1, one=True)  # noqa: E731
    lin = lambda name, n: h @ w(name, (n, wide), 0.02).T  # noqa: E731
    q = _rms(lin(f"{p}.left.q", H * d), eps, one(f"{p}.left.q.norm", H * d)).view(T, H, d)
    v = lin(f"{p}.left.k", G * d)
    k = _rms(v, eps, one(f"{p}.left.k.norm", G * d)).view(T, G, d)
    left = _attend(q, k, v.view(T, G, d), a["scale"], a["mask"]["size"], a["mask"]["keep_first"])
    left = left.reshape(T, H * d) @ w(f"{p}.left.o", (wide, H * d), 0.02).T
    H, d = b["heads"], b["dim"]
    q, k, v = (lin(f"{p}.right.{x}", H * d).view(T, H, d) for x in "qkv")
    z = lin(f"{p}.right.a1", b["decay_rank"]) @ w(f"{p}.right.a2", (H * d, b["decay_rank"]), 0.2).T + w(f"{p}.right.a2.b", (H * d,), 1.0)
    decay = (torch.sigmoid(z) ** (1.0 / b["tau"])).view(T, H, d)
    S, out = h.new_zeros(H, d, d), torch.empty_like(v)
    for t in range(T):
        S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
        out[t] = torch.einsum("hde,hd->he", S, q[t]) * d ** -0.5
    out = _rms(out, eps, one(f"{p}.right.norm", d)).reshape(T, H * d) * _silu(lin(f"{p}.right.g", H * d))
    return m["left_scale"] * left + m["right_scale"] * (out @ w(f"{p}.right.o", (wide, H * d), 0.02).T)


def _laralix_latent(h, w, p, m, eps):
    T, wide = h.shape
    H, d, rd, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"], m["q_rank"]
    one = lambda name, n: w(name, (n,), 0.1, one=True)  # noqa: E731
    q = _rms(h @ w(f"{p}.dq", (rank, wide), 0.02).T, eps, one(f"{p}.dq.norm", rank)) @ w(f"{p}.uq", (H * (d + rd), rank), 0.02).T
    q = q.view(T, H, d + rd)
    down = h @ w(f"{p}.dkv", (r + rd, wide), 0.02).T
    c = _rms(down[:, :r], eps, one(f"{p}.dkv.norm", r))
    angle = _angles(T, rd, m["rot"]["base"])
    q = torch.cat([q[..., :d], _turn(q[..., d:], angle, True)], -1)
    k = torch.cat([(c @ w(f"{p}.uk", (H * d, r), 0.02).T).view(T, H, d), _turn(down[:, None, r:], angle, True).expand(T, H, rd)], -1)
    o = _attend(q, k, (c @ w(f"{p}.uv", (H * d, r), 0.02).T).view(T, H, d), m["scale"])
    return o.reshape(T, H * d) @ w(f"{p}.o", (wide, H * d), 0.02).T


def _exact_laralix(case, seed, rows, want):
    c = CONFIGS["laralix"]
    wide, eps, loop = c["width"], c["norm"]["eps"], c["loop"]
    kept = {}

    def w(name, shape, std, one=False):
        if name not in kept:
            kept[name] = _weight(case, seed, name, shape, std, one)
        return kept[name]
    mixers = {"parallel": _laralix_parallel, "parallel_2": _laralix_parallel_2, "latent_attention": _laralix_latent}
    out = []
    for tokens, at in zip(rows, want):
        x = w("embed", (c["vocab"], wide), 0.02)[torch.tensor(tokens, device="cuda:0")] * c["embedding"]["scale"]
        first = x
        for t in range(loop["times"]):
            x = x + (first if t else 0.0) + w("loop.step", (loop["times"], wide), 0.1)[t]
            for i, layer in enumerate(c["layers"]):
                h = _rms(x, eps, 1.0 + w(f"l{i}.norm1", (wide,), 0.1))
                x = x + mixers[layer["type"]](h, w, f"l{i}.mix", layer["mixer"], eps)
                h = _rms(x, eps, 1.0 + w(f"l{i}.norm2", (wide,), 0.1))
                ff = layer["mlp"]["ff"]
                x = x + (_silu(h @ w(f"l{i}.mlp.gate", (ff, wide), 0.02).T) * (h @ w(f"l{i}.mlp.up", (ff, wide), 0.02).T)) @ w(f"l{i}.mlp.down", (wide, ff), 0.02).T
        x = _rms(x[torch.tensor(at, device="cuda:0")], eps, 1.0 + w("final.norm", (wide,), 0.1))
        out.append(x @ w("head", (c["vocab"], wide), 0.02).T * c["logit_scale"])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":          # whole numbers
        return None
    tokens, portion = _tokens(case, seed)
    held = _lengths(case)
    if kind == "serve":
        per = _exact_laralix(case, seed, tokens, [list(range(n - 1, len(t))) for n, t in zip(held, tokens)])
        return [torch.stack([x[s] for x in per]) for s in range(case["steps"] + 1)]
    if kind in ("decode", "mixed"):
        rows, want = [t[: n + 1] for t, n in zip(tokens, held)], [[n] for n in held]
        if kind == "mixed":
            rows, want = rows + [portion], want + [[len(portion) - 1]]
    else:
        rows, want = tokens, [list(range(n)) if kind == "replay" else [n - 1] for n in held]
    return _exact_qwen2(case, seed, rows, want)
