"""What the engine's speed is measured on: prompt steps, decode steps and mixtures of both, through `Engine`.

Three kinds of model: the dense Llama-style decoder (widths of the 1.3B, 7B and 67B sizes that the benchmark names),
the Tigitar hybrid (gated delta rule, latent attention, routed experts) and the Kerirax design (attention beside a
selective scan, latent attention with a sink, experts, layers that run twice).  Except for the 1.3B size, models have
fewer layers than the sizes they stand for, and a vocabulary that keeps the head's share of the work what it is there.

A case is one of three kinds of work:
  prompt   new requests (`lengths`: the tokens of each) come in with one step; the last token's logits of each
  decode   `batch` requests with about `context` tokens in the cache each bring one token; the logits of all of them
  mixed    a new prompt of `tokens` comes in portions of `portion` tokens beside `batch` decoding requests

Weights and tokens come from the seed; the weights have the spread that keeps every mechanism at work (softmaxes neither
flat nor one-hot, decays close to one, routers that are sure of their choice, as trained ones are).
"""
import hashlib
import math

import numpy as np
import torch

from fastllm_py_b200 import Engine, EngineConfig, StepEntry
from fastllm_py_b200.config.registry import architecture_of
from fastllm_py_b200.parts import BuildContext, Decoder
from fastllm_py_b200.weights import load_tensors

BUDGET = 2048               # tokens of one step
PAGE = 16
ROOM = 2048                 # tokens a decoding request can grow by before it starts over
VOCAB = 32256

DENSE = {                   # hidden, heads, key/value heads, feed-forward, rotary base
    2048: (16, 16, 5504, 100000.0),
    4096: (32, 32, 11008, 10000.0),
    8192: (64, 8, 22016, 10000.0),
}


def listed():
    return [
        # one user's chat with the whole 1.3B model: the smallest call, where launches and latency count
        dict(name="chat token 1.3B", model="dense", width=2048, layers=24, dtype="bfloat16", work="decode", batch=1,
             context=512, spread=0.0),
        # the benchmark's headline: eight requests over 2048-token contexts at the 7B widths
        dict(name="decode 8x2048 7B", model="dense", width=4096, layers=8, dtype="bfloat16", work="decode", batch=8,
             context=2048, spread=0.0),
        # a full server at the 67B widths: many requests of uneven lengths, grouped key/value heads
        dict(name="decode 64 uneven 67B", model="dense", width=8192, layers=2, dtype="bfloat16", work="decode", batch=64,
             context=700, spread=0.8),
        # the benchmark's prompt: 2048 tokens at the 7B widths
        dict(name="prompt 2048 7B", model="dense", width=4096, layers=8, dtype="bfloat16", work="prompt", lengths="2048"),
        # short prompts of several users in one step, odd lengths
        dict(name="prompts uneven 1.3B", model="dense", width=2048, layers=12, dtype="bfloat16", work="prompt",
             lengths="37,129,411,733"),
        # continuous batching: a long prompt in portions beside requests that decode
        dict(name="portions and decode 1.3B", model="dense", width=2048, layers=12, dtype="bfloat16", work="mixed", batch=24,
             context=900, spread=0.6, tokens=1950, portion=488),
        # the true 32-bit path (validation against a reference): a prompt, and decoding
        dict(name="prompt 300 float32", model="dense", width=2048, layers=4, dtype="float32", work="prompt", lengths="300"),
        dict(name="decode 4x700 float32", model="dense", width=2048, layers=4, dtype="float32", work="decode", batch=4,
             context=700, spread=0.3),
        # the two designs with recurrent layers, latent attention and experts: long prompts and decoding
        dict(name="prompt 2048 Tigitar", model="tigitar", width=2048, layers=4, dtype="bfloat16", work="prompt",
             lengths="2048"),
        dict(name="decode 8x2048 Tigitar", model="tigitar", width=2048, layers=8, dtype="bfloat16", work="decode", batch=8,
             context=2048, spread=0.0),
        dict(name="prompts uneven Kerirax", model="kerirax", width=2048, layers=3, dtype="bfloat16", work="prompt",
             lengths="1203,507"),
        dict(name="decode 4 uneven Kerirax", model="kerirax", width=2048, layers=3, dtype="bfloat16", work="decode", batch=4,
             context=1200, spread=0.7),
    ]


def _between(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    model, dtype = rng.choice([("dense", "bfloat16")] * 6 + [("dense", "float32")] * 2 + [("tigitar", "bfloat16")] * 2 +
                              [("kerirax", "bfloat16")] * 2)
    work = rng.choice(["prompt", "decode", "mixed"] if dtype == "bfloat16" and model == "dense" else ["prompt", "decode"])
    if model == "dense":
        width = 2048 if dtype == "float32" else rng.choice([2048, 4096, 4096, 8192])
        layers = {2048: rng.randint(3, 12), 4096: rng.randint(2, 6), 8192: rng.randint(1, 2)}[width]
        if dtype == "float32":
            layers = rng.randint(1, 4)
    else:
        width, layers = 2048, 4 if model == "tigitar" else 3
    case = dict(model=model, width=width, layers=layers, dtype=dtype, work=work)
    if work == "prompt":
        total = _between(rng, 24, 400 if dtype == "float32" else BUDGET)
        n = min(rng.choice([1, 1, 2, 3, 5, 8]), total // 8)
        cuts = sorted(rng.sample(range(4, total - 3), n - 1)) if n > 1 else []
        ends = cuts + [total]
        lengths = [b - a for a, b in zip([0] + cuts, ends)]
        case["lengths"] = ",".join(str(v) for v in lengths)
        return case
    most = 8 if dtype == "float32" else (16 if model != "dense" else (24 if work == "mixed" else 64))
    case["batch"] = _between(rng, 1, most)
    longest = 24000 // case["batch"] if model == "dense" else 8000 // case["batch"]
    case["context"] = _between(rng, 40, max(41, min(1000 if dtype == "float32" else 2200, longest)))
    case["spread"] = round(rng.uniform(0.0, 0.8), 2)
    if work == "mixed":
        case["tokens"] = _between(rng, 100, 1950)
        case["portion"] = _between(rng, 90, 1000)
    return case


# ---------------------------------------------------------------- the models

def _raw(case):
    """The model's config.json."""
    w, n = case["width"], case["layers"]
    if case["model"] == "dense":
        heads, kv, ff, theta = DENSE[w]
        return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": n, "hidden_size": w, "num_attention_heads": heads,
                "num_key_value_heads": kv, "head_dim": 128, "intermediate_size": ff, "vocab_size": VOCAB, "rope_theta": theta,
                "rms_norm_eps": 1e-6, "max_position_embeddings": 16384, "tie_word_embeddings": False}
    dense = {"kind": "dense", "ff": 5504}
    if case["model"] == "tigitar":
        delta = {"conv": 4, "dim": 128, "heads": 16, "kv_heads": 8, "vdim": 128}
        latent = {"dim": 128, "heads": 16, "kv_rank": 512, "rot": {"base": 10000.0, "dims": 64}, "rot_dim": 64,
                  "scale": 192 ** -0.5, "vdim": 128, "mask": {"size": 1024}}
        routed = {"kind": "moe", "expert": {"ff": 1408}, "router": {"experts": 32, "top": 4}}
        layers = []
        for i in range(n):
            kind = i % 4
            mixer = delta if kind in (0, 2) else (latent if kind == 1 else dict(latent, kv_from=i - 2))
            layers.append({"type": "delta" if kind in (0, 2) else "latent_attention", "mixer": mixer,
                           "mlp": routed if kind in (1, 2) else dense})
        return {"architecture": "Tigitar", "layers": layers, "norm": {"eps": 1e-6}, "vocab": VOCAB, "width": w,
                "logit_softcap": 30.0}
    left = {"dim": 128, "heads": 16, "kv_heads": 4, "scale": 128 ** -0.5, "vdim": 128,
            "rot": {"base": 500000.0, "dims": 128, "scaling": {"factor": 4.0}}}
    right = {"conv": 4, "dt_rank": 128, "inner": 4096, "state": 16}
    pair = {"left": left, "left_scale": 0.7, "right": right, "right_scale": 0.4}
    latent = {"dim": 128, "heads": 16, "kv_rank": 512, "q_rank": 1024, "rot": {"base": 10000.0, "dims": 64}, "rot_dim": 64,
              "scale": 192 ** -0.5, "vdim": 128}
    routed = {"kind": "moe", "expert": {"ff": 1408, "limit": 7.0}, "router": {"experts": 32, "top": 4}}
    layers = [{"type": "parallel", "mixer": pair, "mlp": dense}, {"type": "latent_attention", "mixer": latent, "mlp": routed},
              {"type": "parallel", "mixer": pair, "mlp": dense}]
    return {"architecture": "Kerirax", "embedding": {"scale": 8.0}, "layers": layers, "norm": {"eps": 1e-5}, "vocab": VOCAB,
            "width": w, "logit_softcap": 30.0, "loop": {"start": 1, "stop": 2, "times": 2}}


class _Weights:
    """The model's tensors by name, each from a generator of its own; a source that `load_tensors` reads."""

    def __init__(self, case, seed, shapes=None):
        self.case, self.seed, self.shapes = case, seed, shapes
        self.dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32

    def names(self):
        return self.shapes.keys()

    def describe(self, name):
        return tuple(self.shapes[name]), self.dtype

    def get(self, name, device):
        return self.make(name, tuple(self.shapes[name]))

    def make(self, name, shape):
        digest = hashlib.sha256(("%d:%s" % (self.seed, name)).encode()).digest()
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int.from_bytes(digest[:7], "little"))
        x = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(generator=gen)
        leaf = name.split(".")[-1]
        if "norm" in name:
            x = 1.0 + 0.1 * x
            if leaf in ("norm1b", "norm2b"):                       # what a sublayer adds is less than what is there
                x *= 0.3
        elif name == "embed":
            x = self._sure_tokens(x, gen) * (0.125 if self.case["model"] == "kerirax" else 1.0)
        elif leaf == "A_log" and len(shape) == 2:                  # selective scan: state n decays at rate n + 1
            x = torch.log(torch.arange(1, shape[1] + 1, device="cuda").float()).expand(shape) + 0.1 * x
        elif leaf == "A_log":
            x = 1.0 + 0.8 * x
        elif leaf == "dt_bias" or name.endswith("dt.b"):           # small steps: decays close to one
            x = -4.0 + 0.7 * x
        elif leaf == "conv":
            x = 0.5 * x
        elif leaf == "correction":
            x = 0.01 * x
        elif leaf == "D":
            x = 1.0 + 0.3 * x
        elif leaf in ("b", "sink") and len(shape) == 1:
            x = 0.3 * x
        elif name == "loop.step":
            x = 0.3 * x
        elif name == "loop.in":
            eye = torch.eye(shape[0], device="cuda")
            x = torch.cat([0.6 * eye, 0.4 * eye], 1) + 0.2 * shape[1] ** -0.5 * x
        elif "embed_tokens" not in name:
            x = x * shape[1] ** -0.5
            if leaf in ("o", "down") or "o_proj" in name or "down_proj" in name:
                x = 0.5 * x
            if "q_proj" in name or name.endswith(("mix.q", "uq")):
                x = 2.0 * x
        return x.to(self.dtype).contiguous()

    def _sure_tokens(self, x, gen):
        """Every token's vector leans towards `top` experts of each router, so that their choice is clear."""
        for i, layer in enumerate(_raw(self.case)["layers"]):
            if layer["mlp"]["kind"] == "moe":
                e, top = layer["mlp"]["router"]["experts"], layer["mlp"]["router"]["top"]
                r = self.make("l%d.mlp.router" % i, (e, x.shape[1])).float()
                pick = torch.rand((x.shape[0], e), device="cuda", generator=gen).topk(top).indices
                mark = torch.zeros((x.shape[0], e), device="cuda").scatter_(1, pick, 1.0)
                x = x + 6.0 * (mark @ (r / r.norm(dim=1, keepdim=True)))
        return x


# ------------------------------------------------------------------ requests

def _contexts(case):
    """Tokens in the cache of every decoding request: `context` on average, spread evenly to both sides."""
    n, c, s = case["batch"], case["context"], case["spread"]
    return [max(1, int(c * (1.0 + s * (2.0 * ((7 * i) % n + 0.5) / n - 1.0)))) for i in range(n)]


def _lengths(case):
    return [int(v) for v in case["lengths"].split(",")]


def _portions(case):
    t, p = case["tokens"], case["portion"]
    return [min(p, t - a) for a in range(0, t, p)]


def _tokens(case, seed):
    """The requests' token ids: (decoding requests' contexts and what follows, the new prompts)."""
    gen = torch.Generator().manual_seed(seed % (1 << 40) + 17)

    def some(n):
        return torch.randint(0, VOCAB, (n,), generator=gen).tolist()

    live = [] if case["work"] == "prompt" else [some(c + ROOM) for c in _contexts(case)]
    new = [some(n) for n in _lengths(case)] if case["work"] == "prompt" else \
        [some(case["tokens"])] if case["work"] == "mixed" else []
    return live, new


def _fill(state):
    """The decoding requests come in, each with its context."""
    engine = state["engine"]
    for r, n in enumerate(state["contexts"]):
        rid = "live%d" % r
        if engine.is_live(rid):
            engine.end(rid)
        engine.begin(rid)
        for at in range(0, n, BUDGET):
            engine.step([StepEntry(rid, state["live"][r][at:min(n, at + BUDGET)], [])])
    state["grown"] = 0


def prepare(case, seed):
    raw = _raw(case)
    arch = architecture_of(raw)
    plan = arch.make_plan(arch.config_class.from_hf(raw), None)
    live, new = _tokens(case, seed)
    longest = max(len(t) for t in live + new) + PAGE
    held = sum(-(-len(t) // PAGE) * PAGE for t in live + new) + PAGE
    device = torch.device("cuda:0")
    decoder = Decoder(plan, BuildContext(device, torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32, PAGE, longest))
    shapes = decoder.expected_tensors()
    decoder.load(load_tensors(shapes, _Weights(case, seed, shapes), device))
    config = EngineConfig(dtype=case["dtype"], page_size=PAGE, max_requests=len(live) + len(new), max_batched_tokens=BUDGET,
                          max_model_len=longest)
    engine = Engine(decoder, config, longest, held // PAGE)
    state = dict(engine=engine, live=live, new=new, work=case["work"],
                 contexts=[] if case["work"] == "prompt" else _contexts(case),
                 portions=_portions(case) if case["work"] == "mixed" else [])
    _fill(state)
    return state


def _next_tokens(state):
    """An entry for every decoding request: its next token, whose logits are wanted."""
    g = state["grown"]
    state["grown"] = g + 1
    return [StepEntry("live%d" % r, [state["live"][r][n + g]], [0]) for r, n in enumerate(state["contexts"])]


def run(state):
    engine = state["engine"]
    if state["work"] == "prompt":
        rids = ["new%d" % i for i in range(len(state["new"]))]
        for rid in rids:
            engine.begin(rid)
        logits = engine.step([StepEntry(rid, t, [len(t) - 1]) for rid, t in zip(rids, state["new"])])
        for rid in rids:
            engine.end(rid)
        return logits
    if state["grown"] + max(1, len(state["portions"])) > ROOM:
        _fill(state)
    if state["work"] == "decode":
        return engine.step(_next_tokens(state))
    out, at, prompt = [], 0, state["new"][0]
    engine.begin("new")
    for n in state["portions"]:
        last = at + n == len(prompt)
        out.append(engine.step(_next_tokens(state) + [StepEntry("new", prompt[at:at + n], [n - 1] if last else [])]).clone())
        at += n
    engine.end("new")
    return out


# ---------------------------------------------------------------- its work

def _dense_weights(raw):
    w, d, ff = raw["hidden_size"], raw["head_dim"], raw["intermediate_size"]
    h, g = raw["num_attention_heads"], raw["num_key_value_heads"]
    return w * d * (2 * h + 2 * g) + 3 * w * ff


def _mixer(kind, m, w):
    """(weights, floats of state, cache elements a token, FLOPs per query and key, FLOPs a token of a recurrence)."""
    if kind == "delta":
        qk, hv = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
        return (w * (2 * qk + 3 * hv + 2 * m["heads"]), hv * m["dim"] + (m["conv"] - 1) * (2 * qk + hv), 0, 0,
                6 * hv * m["dim"])
    if kind == "latent_attention":
        rows = 0 if "kv_from" in m else m["kv_rank"] + m["rot_dim"]
        q = m["heads"] * (m["dim"] + m["rot_dim"])
        weights = (w * m["q_rank"] + m["q_rank"] * q if "q_rank" in m else w * q) + w * rows + \
            m["kv_rank"] * m["heads"] * (m["dim"] + m["vdim"]) + m["heads"] * m["vdim"] * w
        return weights, 0, rows, 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), 0
    a, r = m["left"], m["right"]
    weights = w * (a["heads"] * (a["dim"] + a["vdim"] + 1) + a["kv_heads"] * (a["dim"] + a["vdim"]) + 3 * r["inner"]) + \
        r["inner"] * (2 * r["dt_rank"] + 2 * r["state"])
    return (weights, r["inner"] * (r["state"] + r["conv"] - 1), a["kv_heads"] * (a["dim"] + a["vdim"]),
            2 * a["heads"] * (a["dim"] + a["vdim"]), 6 * r["inner"] * r["state"])


def _step_work(case, raw, entries):
    """Bytes and FLOPs of one step: entries of (tokens in the cache, new tokens, logits wanted)."""
    size = 2 if case["dtype"] == "bfloat16" else 4
    w, n = case["width"], sum(q for _, q, _ in entries)
    wanted = sum(m for _, _, m in entries)
    nbytes = size * (VOCAB * w if wanted else 0) + size * n * w + 4 * wanted * VOCAB
    flops = 2.0 * wanted * VOCAB * w

    def attention(per_pair, per_token, window, reads=None):
        b = f = 0
        for ctx, q, _ in entries:
            seen = ctx + q if window is None else min(ctx + q, window + q - 1)
            pairs = sum(min(ctx + i + 1, window or ctx + i + 1) for i in range(q))
            f += per_pair * pairs
            b += size * (per_token * q + (reads or per_token) * (seen - q))
        return b, f

    if case["model"] == "dense":
        layer = _dense_weights(raw)
        g, h, d = raw["num_key_value_heads"], raw["num_attention_heads"], raw["head_dim"]
        b, f = attention(4 * h * d, 2 * g * d, None)
        return nbytes + case["layers"] * (size * layer + b), flops + case["layers"] * (2.0 * n * layer + f)
    order = list(enumerate(raw["layers"]))
    if case["model"] == "kerirax":
        order = [order[0], order[1], order[1], order[2]]
        nbytes, flops = nbytes + 2 * size * 2 * w * w, flops + 2 * 2.0 * n * 2 * w * w
    for _, layer in order:
        weights, state, cached, per_pair, per_token = _mixer(layer["type"], layer["mixer"], w)
        window = layer["mixer"].get("mask", {}).get("size")
        shared = 576 if "kv_from" in layer["mixer"] else None
        b, f = attention(per_pair, cached, window, shared) if per_pair else (0, 0)
        nbytes += size * weights + b + len(entries) * 8 * state
        flops += 2.0 * n * weights + f + n * per_token
        mlp = layer["mlp"]
        if mlp["kind"] == "dense":
            nbytes, flops = nbytes + size * 3 * w * mlp["ff"], flops + 2.0 * n * 3 * w * mlp["ff"]
        else:
            e, top, ff = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
            used = e * (1.0 - (1.0 - top / e) ** n)                    # experts that n tokens reach
            nbytes, flops = nbytes + size * (w * e + used * 3 * w * ff), flops + 2.0 * n * w * (e + top * 3 * ff)
    return nbytes, flops


def work(case):
    raw = _raw(case)
    if case["work"] == "prompt":
        steps = [[(0, n, 1) for n in _lengths(case)]]
    elif case["work"] == "decode":
        steps = [[(c, 1, 1) for c in _contexts(case)]]
    else:
        steps, at = [], 0
        for p in _portions(case):
            steps.append([(c, 1, 1) for c in _contexts(case)] + [(at, p, int(at + p == case["tokens"]))])
            at += p
    done = [_step_work(case, raw, s) for s in steps]
    return {"bytes": sum(b for b, _ in done), "flops": sum(f for _, f in done)}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5}                                       # 1.5e-6 off 64 bits was seen
    return {"rel": 0.02}                                           # 0.003 to 0.009 off 64 bits was seen


# --------------------------------------------------- the same in 64 bits

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _half(x, cos, sin):
    """Pairs (i, i + d / 2) turned; x [..., T, heads, d], cos and sin [T, d / 2]."""
    a, b = x.chunk(2, -1)
    c, s = cos[:, None], sin[:, None]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _neighbours(x, cos, sin):
    """Pairs (2 i, 2 i + 1) turned."""
    a, b = x[..., 0::2], x[..., 1::2]
    c, s = cos[:, None], sin[:, None]
    return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)


def _angles(t, dims, base, factor=1.0):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims) / factor
    ang = torch.arange(t, dtype=torch.float64, device="cuda")[:, None] * f
    return torch.cos(ang), torch.sin(ang)


def _attend(q, k, v, scale, window=None, sink=None):
    """Causal softmax attention of one sequence: q [T, H, d], k and v [T, G, ...], some heads at a time."""
    t, h = q.shape[:2]
    rep = h // k.shape[1]
    i = torch.arange(t, device="cuda")
    hidden = i[None, :] > i[:, None]
    if window is not None:
        hidden |= i[:, None] - i[None, :] >= window
    out = []
    for a in range(h):
        s = (q[:, a] @ k[:, a // rep].T * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[a].expand(t, 1)], 1)
        p = torch.softmax(s, -1)
        out.append(p[:, :t] @ v[:, a // rep])
    return torch.stack(out, 1).flatten(1)


def _conv(x, taps):
    """Causal, per channel: x [R, T, C], taps [C, K]."""
    k, t = taps.shape[1], x.shape[1]
    pad = torch.cat([x.new_zeros(x.shape[0], k - 1, x.shape[2]), x], 1)
    return sum(pad[:, j:j + t] * taps[:, j] for j in range(k))


class _Exact:
    def __init__(self, case, seed):
        self.raw, self.weights, self.w = _raw(case), _Weights(case, seed), case["width"]

    def get(self, name, *shape):
        return self.weights.make(name, shape).double()

    def dense(self, seqs, rows):
        raw, w = self.raw, self.w
        h, g, d, ff = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["intermediate_size"]
        eps, longest = raw["rms_norm_eps"], max(len(s) for s in seqs)
        # the tables of angles are 32-bit by definition
        freq = 1.0 / (raw["rope_theta"] ** (np.arange(0, d, 2, dtype=np.float32) / d))
        ang = np.arange(longest).astype(np.float32)[:, None] * freq[None, :]
        cos, sin = (torch.from_numpy(f(ang)).cuda().double() for f in (np.cos, np.sin))
        table = self.weights.make("model.embed_tokens.weight", (VOCAB, w))
        xs = [table[torch.tensor(s, device="cuda")].double() for s in seqs]
        for i in range(raw["num_hidden_layers"]):
            p = "model.layers.%d." % i
            n1, n2 = self.get(p + "input_layernorm.weight", w), self.get(p + "post_attention_layernorm.weight", w)
            q, k, v, o = (self.get(p + "self_attn.%s_proj.weight" % s, *z) for s, z in
                          (("q", (h * d, w)), ("k", (g * d, w)), ("v", (g * d, w)), ("o", (w, h * d))))
            gate, up, down = (self.get(p + "mlp.%s_proj.weight" % s, *z) for s, z in
                              (("gate", (ff, w)), ("up", (ff, w)), ("down", (w, ff))))
            for r, x in enumerate(xs):
                t = x.shape[0]
                y = _rms(x, eps) * n1
                a = _attend(_half((y @ q.T).view(t, h, d), cos[:t], sin[:t]), _half((y @ k.T).view(t, g, d), cos[:t], sin[:t]),
                            (y @ v.T).view(t, g, d), d ** -0.5)
                x = x + a @ o.T
                y = _rms(x, eps) * n2
                xs[r] = x + (_silu(y @ gate.T) * (y @ up.T)) @ down.T
        final, head = self.get("model.norm.weight", w), self.get("lm_head.weight", VOCAB, w)
        return [(_rms(x[at], eps) * final) @ head.T for x, at in zip(xs, rows)]

    def delta(self, h, p, m, eps):
        w, H, G, D, V = self.w, m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        r, t = h.shape[:2]

        def part(s, n):
            return _silu(_conv(h @ self.get(p + s, n, w).T, self.get(p + s + ".conv", n, m["conv"])))

        q, k, v = part("q", G * D).view(r, t, G, D), part("k", G * D).view(r, t, G, D), part("v", H * V).view(r, t, H, V)
        q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5).repeat_interleave(H // G, 2)
        k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)
        beta = torch.sigmoid(h @ self.get(p + "b", H, w).T)
        rate = torch.nn.functional.softplus(h @ self.get(p + "a", H, w).T + self.get(p + "dt_bias", H))
        decay = torch.exp(-torch.exp(self.get(p + "A_log", H)) * rate)
        S, out = h.new_zeros(r, H, D, V), h.new_zeros(r, t, H, V)
        for i in range(t):
            S = S * decay[:, i, :, None, None]
            u = beta[:, i, :, None] * (v[:, i] - (k[:, i, :, None] @ S)[:, :, 0])
            S = S + k[:, i, :, :, None] * u[:, :, None]
            out[:, i] = (q[:, i, :, None] @ S)[:, :, 0]
        out = _rms(out, eps) * self.get(p + "norm", V) * _silu(h @ self.get(p + "g", H * V, w).T).view(r, t, H, V)
        return out.flatten(2) @ self.get(p + "o", w, H * V).T

    def latent(self, h, p, m, eps, kept, turn):
        """`kept`: the layer's (latent, rotated key part), or None where this layer makes its own."""
        w, H, D, R, V, rank = self.w, m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        r, t = h.shape[:2]
        cos, sin = _angles(t, R, m["rot"]["base"])
        if kept is None:
            kv = h @ self.get(p + "dkv", rank + R, w).T
            kept = (_rms(kv[..., :rank], eps) * self.get(p + "dkv.norm", rank), turn(kv[..., None, rank:], cos, sin))
        c, kr = kept
        if "q_rank" in m:
            cq = _rms(h @ self.get(p + "dq", m["q_rank"], w).T, eps) * self.get(p + "dq.norm", m["q_rank"])
            q = cq @ self.get(p + "uq", H * (D + R), m["q_rank"]).T
        else:
            q = h @ self.get(p + "q", H * (D + R), w).T
        q = q.view(r, t, H, D + R)
        q = torch.cat([q[..., :D], turn(q[..., D:], cos, sin)], -1)
        k = torch.cat([(c @ self.get(p + "uk", H * D, rank).T).view(r, t, H, D), kr.expand(r, t, H, R)], -1)
        v = (c @ self.get(p + "uv", H * V, rank).T).view(r, t, H, V)
        sink = self.get(p + "sink", H) if "q_rank" in m else None
        window = m.get("mask", {}).get("size")
        o = torch.stack([_attend(q[i], k[i], v[i], m["scale"], window, sink) for i in range(r)])
        return o @ self.get(p + "o", w, H * V).T, kept

    def unit(self, h, p, ff, act):
        return (act(h @ self.get(p + "gate", ff, self.w).T) * (h @ self.get(p + "up", ff, self.w).T)) @ \
            self.get(p + "down", self.w, ff).T

    def experts(self, h, p, f, on_input):
        E, top, ff = f["router"]["experts"], f["router"]["top"], f["expert"]["ff"]
        x = h.flatten(0, 1)
        s = torch.sigmoid(x @ self.get(p + "router", E, self.w).T)
        chosen = torch.topk(s if on_input else s + self.get(p + "correction", E), top, -1).indices
        out = torch.zeros_like(x)
        for e in range(E):
            at = (chosen == e).any(-1).nonzero()[:, 0]
            if at.numel() and on_input:
                lim, y = f["expert"]["limit"], x[at] * s[at, e:e + 1]
                g = (y @ self.get(p + "e%d.gate" % e, ff, self.w).T).clamp(max=lim)
                u = (y @ self.get(p + "e%d.up" % e, ff, self.w).T).clamp(-lim, lim)
                out[at] += (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ self.get(p + "e%d.down" % e, self.w, ff).T
            elif at.numel():
                out[at] += s[at, e:e + 1] * self.unit(x[at], p + "e%d." % e, ff, _silu)
        return out.view_as(h)

    def scan(self, h, p, m):
        n, N, rank = m["inner"], m["state"], m["dt_rank"]
        u, z = (h @ self.get(p + "in", 2 * n, self.w).T).split(n, -1)
        x = _silu(_conv(u, self.get(p + "conv", n, m["conv"])) + self.get(p + "conv.b", n))
        low = x @ self.get(p + "x", rank + 2 * N, n).T
        dt = torch.nn.functional.softplus(low[..., :rank] @ self.get(p + "dt", n, rank).T + self.get(p + "dt.b", n))
        B, C = low[..., rank:rank + N], low[..., rank + N:]
        A, S, y = -torch.exp(self.get(p + "A_log", n, N)), h.new_zeros(h.shape[0], n, N), torch.zeros_like(x)
        for i in range(h.shape[1]):
            S = torch.exp(dt[:, i, :, None] * A) * S + (dt[:, i] * x[:, i])[..., None] * B[:, i, None]
            y[:, i] = (S @ C[:, i, :, None])[..., 0]
        return ((y + self.get(p + "D", n) * x) * _silu(z)) @ self.get(p + "o", self.w, n).T

    def left(self, h, p, m, eps):
        w, H, G, d, r, t = self.w, m["heads"], m["kv_heads"], m["dim"], h.shape[0], h.shape[1]
        cos, sin = _angles(t, m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]["factor"])
        q, k = (_neighbours((_rms(h @ self.get(p + s, c * d, w).T, eps) * self.get(p + s + ".norm", c * d)).view(r, t, c, d),
                            cos, sin) for s, c in (("q", H), ("k", G)))
        v = (h @ self.get(p + "v", G * m["vdim"], w).T).view(r, t, G, m["vdim"])
        o = torch.stack([_attend(q[i], k[i], v[i], m["scale"]) for i in range(r)]).view(r, t, H, m["vdim"])
        return (o * torch.sigmoid(h @ self.get(p + "g", H, w).T)[..., None]).flatten(2) @ self.get(p + "o", w, H * m["vdim"]).T

    def design(self, seqs, rows):
        """Tigitar or Kerirax; sequences are filled up on the right, where nothing before can see it."""
        raw, w, eps, t = self.raw, self.w, self.raw["norm"]["eps"], max(len(s) for s in seqs)
        rejoined = raw["architecture"] == "Kerirax"
        ids = torch.tensor([s + [0] * (t - len(s)) for s in seqs], device="cuda")
        x = x0 = self.weights.make("embed", (VOCAB, w))[ids].double() * raw.get("embedding", {}).get("scale", 1.0)
        order = [(0, None), (1, 0), (1, 1), (2, None)] if rejoined else [(i, None) for i in range(len(raw["layers"]))]
        kept = {}
        for i, turn in order:
            layer, p = raw["layers"][i], "l%d." % i
            m, f = layer["mixer"], layer["mlp"]
            if turn is not None:
                x = torch.cat([x, x0], -1) @ self.get("loop.in", w, 2 * w).T + self.get("loop.step", 2, w)[turn]
            h = _rms(x, eps) * self.get(p + "norm1", w)
            if layer["type"] == "delta":
                y = self.delta(h, p + "mix.", m, eps)
            elif layer["type"] == "latent_attention":
                y, kept[i] = self.latent(h, p + "mix.", m, eps, kept.get(m.get("kv_from")), _neighbours if rejoined else _half)
            else:
                y = m["left_scale"] * self.left(h, p + "mix.left.", m["left"], eps) + \
                    m["right_scale"] * self.scan(h, p + "mix.right.", m["right"])
            if not rejoined:
                x = x + _rms(y, eps) * self.get(p + "norm1b", w)
                h = _rms(x, eps) * self.get(p + "norm2", w)
            if f["kind"] == "moe":
                z = self.experts(h, p + "mlp.", f, rejoined)
            else:
                z = self.unit(h, p + "mlp.", f["ff"], _silu if rejoined else torch.relu)
            x = x + y + z if rejoined else x + _rms(z, eps) * self.get(p + "norm2b", w)
        picked = torch.stack([x[i, at] for i, at in enumerate(rows)])
        logits = (_rms(picked, eps) * self.get("final.norm", w)) @ self.get("head", VOCAB, w).T
        cap = raw["logit_softcap"]
        return cap * torch.tanh(logits / cap)


def exact(case, seed):
    live, new = _tokens(case, seed)
    model = _Exact(case, seed)
    with torch.no_grad():
        if case["work"] == "prompt":
            seqs, rows = new, [len(t) - 1 for t in new]
        elif case["work"] == "decode":
            seqs = [t[:n + 1] for t, n in zip(live, _contexts(case))]
            rows = [len(t) - 1 for t in seqs]
        else:
            steps = len(_portions(case))
            seqs = [t[:n + steps] for t, n in zip(live, _contexts(case))] + new
            rows = [list(range(n, n + steps)) for n in _contexts(case)] + [[len(new[0]) - 1]]
        if case["model"] != "dense":
            return model.design(seqs, rows)
        out = model.dense(seqs, rows)
    if case["work"] != "mixed":
        return torch.stack(out)
    return [torch.stack([o[i] for o in out[:-1]] + ([out[-1][0]] if i == steps - 1 else [])) for i in range(steps)]
