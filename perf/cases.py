"""The work by which this engine's speed is judged: steps of the models that it runs, at the sizes of its presets.

A case is one call of the step function (``ModelRunner.step``) as the engine, the replay and the benchmark make it, or
one call of the sampler.  Keys of a step: ``model`` (a preset), ``dtype``, ``rows`` requests that decode one token each
after ``context`` tokens (``ragged``: 35 to 100 % of them), ``prompts`` requests that bring a whole prompt of up to ``prompt``
tokens, ``wanted`` places of each prompt whose logits come back (1: the last).  Keys of a sampling: ``vocab`` and
``rows``.  Weights are random with a checkpoint's names, shapes and magnitudes, token ids uniform.

``exact`` restates the models as plain torch in 64 bits.
"""

from __future__ import annotations

import math
import zlib

import torch

from acorninfer_b200 import ModelRunner, SamplingParams
from acorninfer_b200.config.presets import preset
from acorninfer_b200.engine.batch import StepEntry
from acorninfer_b200.models.decoder import expected_tensors
from acorninfer_b200.registry import config_from_dict, spec_for
from acorninfer_b200.sampling.sampler import Sampler

PAGE = 16
SPAN = 128          # decode passes after which the requests end and others of the starting length take their place
DEVICE = "cuda:0"
KINDS = 64          # kinds of tokens that a routed model's routers tell apart
F64 = torch.float64
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# ------------------------------------------------------------------ the cases


def _step(name, model, *, rows=0, context=0, ragged=False, prompts=0, prompt=0, wanted=1, dtype="bfloat16"):
    return {"name": name, "kind": "step", "model": model, "dtype": dtype, "rows": rows, "context": context, "ragged": ragged,
            "prompts": prompts, "prompt": prompt, "wanted": wanted}


def listed():
    return [
        # one user of a small model early in an answer: launches and latencies, hardly any bytes
        _step("qwen3-0.6b-decode-1", "qwen3-0.6b", rows=1, context=300),
        # the benchmark's headline: eight users late in their answers
        _step("qwen3-8b-decode-8", "qwen3-8b", rows=8, context=4000),
        # a server's steady state: answers of many lengths, a number of rows that fills no tile
        _step("qwen3-4b-decode-41-ragged", "qwen3-4b", rows=41, context=1700, ragged=True),
        # continuous batching: new prompts beside running answers in one step
        _step("qwen3-0.6b-mixed", "qwen3-0.6b", rows=27, context=900, ragged=True, prompts=3, prompt=511),
        # a long prompt to its first token
        _step("qwen3-8b-prefill-2048", "qwen3-8b", prompts=1, prompt=2048),
        # the true 32-bit path, which replays and comparisons use: a prompt of odd length, a decode step
        _step("qwen3-0.6b-f32-prefill-777", "qwen3-0.6b", prompts=1, prompt=777, dtype="float32"),
        _step("qwen3-1.7b-f32-decode-6", "qwen3-1.7b", rows=6, context=1500, dtype="float32"),
        # a token for each of a full batch with temperature, top-k and top-p over a large vocabulary
        {"name": "sample-64", "kind": "sample", "vocab": 151936, "rows": 64},
        # the other mixers' prompts: cached latents, a delta rule and routed experts (scored at many places)
        _step("kogonex-w2048-prefill-2000", "kogonex-w2048", prompts=1, prompt=2000, wanted=250),
        # ... and their decode steps with recurrent state
        _step("kogonex-w1024-decode-16", "kogonex-w1024", rows=16, context=700),
        # state space and linear attention over a prompt
        _step("vagulorn-w2048-prefill-2048", "vagulorn-w2048", prompts=1, prompt=2048),
        # time mixing, convolved attention and latent attention over several prompts at once
        _step("tedenex-w2048-prefill-3x601", "tedenex-w2048", prompts=3, prompt=601),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "mixed", "float32", "sample", "design", "design", "design"])
    if kind == "sample":
        c = {"kind": "sample", "vocab": rng.choice([32768, 65536, 151936]), "rows": _log(rng, 1, 64)}
    elif kind == "design":
        model = rng.choice(["kogonex", "vagulorn", "tedenex"]) + rng.choice(["-w1024", "-w2048"])
        if rng.random() < 0.5:
            c = _step("", model, rows=_log(rng, 1, 48), context=_log(rng, 30, 1200))
        else:
            n = rng.choice([1, 1, 2, 3])
            c = _step("", model, prompts=n, prompt=_log(rng, 16, 2048 // n))
            if model.startswith("kogonex"):
                c["wanted"] = max(1, c["prompt"] // 8)
    elif kind == "float32":
        if rng.random() < 0.5:
            c = _step("", "qwen3-0.6b", prompts=1, prompt=_log(rng, 16, 800), dtype="float32")
        else:
            c = _step("", rng.choice(["qwen3-0.6b", "qwen3-1.7b"]), rows=_log(rng, 1, 12), context=_log(rng, 30, 1600),
                      ragged=rng.random() < 0.5, dtype="float32")
    else:
        model = rng.choice(["qwen3-0.6b", "qwen3-1.7b", "qwen3-4b", "qwen3-8b"])
        if kind == "decode":
            rows = _log(rng, 1, 64)
            c = _step("", model, rows=rows, context=_log(rng, 30, min(4000, 60000 // rows)), ragged=rng.random() < 0.5)
        elif kind == "prefill":
            c = _step("", model, prompts=1, prompt=_log(rng, 8, 2048))
        else:
            n = rng.choice([1, 2, 3])
            c = _step("", model, rows=_log(rng, 1, 48), context=_log(rng, 30, 1000), ragged=True, prompts=n,
                      prompt=_log(rng, 8, 1400 // n))
    c.pop("name", None)
    return c


def _contexts(case):
    """Tokens that each decoding request holds before the step."""
    n = case["context"]
    if not case["ragged"]:
        return [n] * case["rows"]
    return [max(1, int(n * (0.35 + 0.65 * ((i + 1) * 0.6180339887 % 1.0)))) for i in range(case["rows"])]


def _prompts(case):
    """Tokens of each prompt: the first is the longest."""
    return [max(1, int(case["prompt"] * (1.0 - 0.37 * i))) for i in range(case["prompts"])]


def _wanted(case, n):
    w = min(case["wanted"], n)
    return [n - 1 - (n * i) // w for i in range(w)][::-1]


# ------------------------------------------------------------------ inputs


def _generator(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & (2 ** 62 - 1))


#: (spread, mean) of a checkpoint's tensors by what they are.  The products that write into the residual stream start
#: smaller by the root of their number, and Qwen3's token rows larger, as trained ones are: the stream then carries more
#: than any one layer adds to it.
MAGNITUDES = {"matrix": (0.02, 0.0), "norm": (0.1, 1.0), "norm_offset": (0.1, 0.0), "bias": (0.5, 0.0), "sink": (1.0, 0.0),
              "conv": (0.5, 0.25), "decay_log": (0.5, -1.0), "blend": (0.2, 0.5)}


class Checkpoint:
    """The tensors of a random model, each made from the seed and its name alone."""

    def __init__(self, case, seed):
        self.raw = preset(case["model"])
        self.config = config_from_dict(self.raw)
        self.specs = expected_tensors(spec_for(self.config))
        self.dtype, self.seed = DTYPES[case["dtype"]], seed
        self.routed = any(name.endswith("router") for name in self.specs)

    def tensor(self, name):
        spec = self.specs[name]
        spread, mean = MAGNITUDES[spec.init]
        if name.endswith(("o_proj.weight", "down_proj.weight")):
            spread /= math.sqrt(2 * self.config.num_hidden_layers)
        elif name == "model.embed_tokens.weight":
            spread = 0.5
        elif name.endswith("correction"):
            spread = 0.01
        t = torch.empty(spec.shape, dtype=self.dtype, device=DEVICE).normal_(mean, spread, generator=_generator(self.seed, name))
        return self._with_kinds(name, t) if self.routed else t

    def _with_kinds(self, name, t):
        """A routed model's token rows and routers.  Trained routers mostly go by the token: every token is of one of
        ``KINDS`` kinds, its row holds the kind's direction, and a router scores its kind's experts well above the others."""
        if name != "embed" and not name.endswith("router"):
            return t
        kinds = torch.empty((KINDS, t.shape[1]), device=DEVICE).normal_(generator=_generator(self.seed, "kinds"))
        if name == "embed":
            return (t + 2.0 * kinds[torch.arange(t.shape[0], device=DEVICE) % KINDS]).to(t.dtype)
        r, n, g = self.raw["layers"][0]["mlp"]["router"], t.shape[0], _generator(self.seed, name + ".likes")
        likes = torch.rand((KINDS, n), device=DEVICE, generator=g)
        groups = torch.rand((KINDS, r["groups"]["count"]), device=DEVICE, generator=g).argsort(-1) < r["groups"]["keep"]
        likes += 2.0 * groups.repeat_interleave(n // r["groups"]["count"], 1)
        best = likes.argsort(-1, descending=True).argsort(-1) < r["top"]
        score = torch.where(best, 1.5, -1.5) + torch.rand((KINDS, n), device=DEVICE, generator=g) - 0.5
        return (score.T @ kinds / (2.0 * t.shape[1]) + 0.05 * t).to(t.dtype)

    def exact(self, name):
        return self.tensor(name).to(F64)

    def all(self):
        return {name: self.tensor(name) for name, spec in self.specs.items() if not spec.optional}

    def tokens(self, name, *shape):
        return torch.randint(0, self.config.vocab_size, shape, device=DEVICE, generator=_generator(self.seed, name))

    def past(self, layer, row, length):
        """Keys and values [2, kv_heads, length rounded up to pages, head_dim] that a request holds before the step."""
        c = self.config
        n = -(-length // PAGE) * PAGE
        return torch.empty((2, c.num_key_value_heads, n, c.head_dim), dtype=self.dtype, device=DEVICE).normal_(
            0.0, 1.0, generator=_generator(self.seed, f"past.{layer}.{row}"))


class Serving:
    """A runner with its live requests: what a serving program holds between two steps."""

    def __init__(self, case, seed):
        ck = Checkpoint(case, seed)
        self.contexts, prompts = _contexts(case), _prompts(case)
        pages = sum(-(-(n + SPAN + 8) // PAGE) for n in self.contexts) + sum(-(-n // PAGE) + 1 for n in prompts) + 8
        self.runner = ModelRunner(ck.config, ck.all(), dtype=case["dtype"], device=DEVICE, num_blocks=pages, page_size=PAGE,
                                  max_requests=len(self.contexts) + len(prompts) + 1, max_step_tokens=4096)
        self.feed = ck.tokens("decoded", SPAN, len(self.contexts)).tolist() if self.contexts else []
        self.prompts = [(ck.tokens(f"prompt.{i}", n).tolist(), _wanted(case, n)) for i, n in enumerate(prompts)]
        self.live, self.passes = [], 0
        # what a server does when it starts: the libraries' kernels loaded, the graphs of these steps captured
        for held in ({0, SPAN - 8} if self.contexts else {0}):
            self._open(held)
            for _ in range(4):
                self.step()
            self._close()
        self._open(0, fill=False)
        if case["model"].startswith("qwen3"):
            self._fill_pages(ck)
        else:
            self._read_contexts(ck)
        self.passes = 0

    def _open(self, more, fill=True):
        for i, n in enumerate(self.contexts):
            rc = self.runner.open(("row", i))
            self.live.append(rc)
            if fill:                                     # the pages of a request of that length, with what lies in them
                self.runner.manager.extend(rc, n + more)
                self.runner.manager.commit(rc, n + more)
        self.passes = 0

    def _close(self):
        for rc in self.live:
            self.runner.close(rc)
        self.live = []

    def _fill_pages(self, ck):
        manager = self.runner.manager
        for r, (rc, n) in enumerate(zip(self.live, self.contexts)):
            manager.extend(rc, n)
            manager.commit(rc, n)
            table = torch.tensor(rc.tables[0], device=DEVICE)
            for layer in range(ck.config.num_hidden_layers):
                past = ck.past(layer, r, n)
                for pages, x in zip(manager.kv_pages(layer), past):
                    pages[table] = x.view(x.shape[0], -1, PAGE, x.shape[-1]).transpose(0, 1)

    def _read_contexts(self, ck):
        history = ck.tokens("history", len(self.contexts), max(self.contexts, default=0)).tolist()
        per_step = max(1, 4096 // max(self.contexts, default=1))
        for at in range(0, len(self.live), per_step):
            self.runner.step([StepEntry(rc, h[:n], []) for rc, h, n in
                              zip(self.live[at:at + per_step], history[at:at + per_step], self.contexts[at:at + per_step])])

    def step(self):
        if self.live and self.passes == SPAN:
            self._close()
            self._open(0)
        entries = [StepEntry(rc, [tok], [0]) for rc, tok in zip(self.live, self.feed[self.passes] if self.live else ())]
        opened = []
        for i, (tokens, want) in enumerate(self.prompts):
            opened.append(self.runner.open(("prompt", i)))
            entries.append(StepEntry(opened[-1], tokens, want))
        logits = self.runner.step(entries)
        for rc in opened:
            self.runner.close(rc)
        self.passes += 1
        return logits


class Sampling:
    """A step's logits and its requests' parameters."""

    def __init__(self, case, seed):
        rows, vocab = case["rows"], case["vocab"]
        g = _generator(seed, "logits")
        self.logits = torch.empty((rows, vocab), dtype=torch.float32, device=DEVICE).normal_(0.0, 2.5, generator=g)
        self.params = [SamplingParams(temperature=(0.7, 1.0, 0.6)[i % 3], top_p=(0.95, 0.8, 1.0, 0.9)[i % 4],
                                      top_k=(0, 20, 50)[i % 3], seed=seed + i) for i in range(rows)]
        self.counters = [(17 * i) % 400 for i in range(rows)]
        self.sampler = Sampler(DEVICE)

    def step(self):
        return self.sampler.launch(self.logits, self.params, self.counters, True)


def prepare(case, seed):
    return Sampling(case, seed) if case["kind"] == "sample" else Serving(case, seed)


def run(state):
    return state.step()


# ------------------------------------------------------------------ what a pass cannot do without


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    ck = Checkpoint(case, 0)
    size = 4 if case["dtype"] == "float32" else 2
    contexts, prompts = _contexts(case), _prompts(case)
    tokens, logits = len(contexts) + sum(prompts), len(contexts) + sum(len(_wanted(case, n)) for n in prompts)
    pairs = sum(n + 1 for n in contexts) + sum(n * (n + 1) // 2 for n in prompts)        # (query, key) pairs of a causal head
    raw, c = ck.raw, ck.config
    width, vocab = c.hidden_size, c.vocab_size
    nbytes, flops = float(size) * vocab * width, 2.0 * vocab * width * logits              # the output matrix
    for name, spec in ck.specs.items():
        if len(spec.shape) != 2 or spec.shape[0] == vocab or "embed" in name or name == "bigram" or name.endswith("conv"):
            continue
        n, reads, runs = float(spec.shape[0] * spec.shape[1]), 1.0, 1
        if ".mlp.e" in name:                              # a routed expert: the share of tokens and steps that choose it
            r = raw["layers"][0]["mlp"]["router"]
            share = r["top"] / (r["experts"] + r["identity"])
            flops += 2.0 * n * tokens * share
            reads = 1.0 - (1.0 - share) ** tokens
        else:
            if raw.get("loop") and name.startswith("l") and int(name[1:name.index(".")]) < raw["loop"]["stop"]:
                runs = raw["loop"]["times"]
            flops += 2.0 * n * tokens * runs
        nbytes += size * n * reads * (1 if size * n > 0 else 0)
    nbytes += 4.0 * logits * vocab + size * width * tokens
    for m in _mixers(case, raw):
        kind = m["type"]
        if kind == "attention":
            span = m.get("span")
            seen = pairs if span is None else (sum(min(n % span + 1, n + 1) for n in contexts)
                                               + sum(sum(min(i, i % span) + 1 for i in range(n)) for n in prompts))
            flops += 2.0 * m["heads"] * (m["dim"] + m["vdim"]) * seen
            kept = size * m["kv_heads"] * (m["dim"] + m["vdim"])
            nbytes += kept * (sum(min(n, span or n) for n in contexts) + tokens)
        else:                                             # recurrent: about four operations an entry of the state and token
            state = float(m["heads"] * m["dim"] * m["vdim"])
            flops += 4.0 * state * tokens
            nbytes += 4.0 * state * (2 * len(contexts) + len(prompts))
    return {"bytes": nbytes, "flops": flops}


def _mixers(case, raw):
    """The mixers of every layer run: attention heads with what is cached of a token, or recurrent states."""
    if case["model"].startswith("qwen3"):
        d = raw["head_dim"]
        return [{"type": "attention", "heads": raw["num_attention_heads"], "kv_heads": raw["num_key_value_heads"], "dim": d,
                 "vdim": d}] * raw["num_hidden_layers"]
    order = list(range(len(raw["layers"])))
    if raw.get("loop"):
        a, b = raw["loop"]["start"], raw["loop"]["stop"]
        order = order[:a] + order[a:b] * raw["loop"]["times"] + order[b:]
    out = []
    for i in order:
        layer, m = raw["layers"][i], raw["layers"][i]["mixer"]
        if layer["type"] == "latent_attention":           # keys and values of a head are made from the cached latent
            out.append({"type": "attention", "heads": m["heads"], "kv_heads": 1, "dim": m["dim"] + m["rot_dim"], "vdim": m["vdim"],
                        "span": (m.get("mask") or {}).get("size")})
        elif layer["type"] == "attention":
            out.append(dict(m, type="attention", span=(m.get("mask") or {}).get("size")))
        elif layer["type"] == "parallel":
            out += [dict(m["left"], type="attention", span=m["left"]["mask"]["size"]), dict(m["right"], type="recurrent")]
        elif layer["type"] == "mamba2":
            out.append({"type": "recurrent", "heads": m["heads"], "dim": m["state"], "vdim": m["vdim"]})
        else:
            out.append(dict(m, type="recurrent", vdim=m.get("vdim", m["dim"])))
    return out


def tolerance(case):
    # About four times the distance from ``exact`` that was measured: 3.3e-8 for log-probabilities (a few units of the last
    # place of the largest allowed here), 0.8e-6 to 2.2e-6 in float32; in bfloat16 0.2 % at the two smallest Qwen3 sizes and
    # 0.6 to 1.4 % elsewhere, with single logits off by 1 % and 3 to 10 % of their root mean square.
    if case["kind"] == "sample":
        return {"rel": 4e-7, "max": 1e-5, "differ": 0.01}
    if case["dtype"] == "float32":
        return {"rel": 9e-6, "max": 1e-4}
    if case["model"] in ("qwen3-0.6b", "qwen3-1.7b"):
        return {"rel": 0.01, "max": 0.05}
    return {"rel": 0.03, "max": 0.4}


# ------------------------------------------------------------------ the same in 64 bits


def exact(case, seed):
    if case["kind"] == "sample":
        return _sample(Sampling(case, seed))
    ck = Checkpoint(case, seed)
    family = case["model"].split("-")[0]
    if family == "qwen3":
        return _qwen3(case, ck)
    forward = {"kogonex": _kogonex, "vagulorn": _vagulorn, "tedenex": _tedenex}[family]
    out = []
    if case["rows"]:
        history = ck.tokens("history", case["rows"], case["context"])
        tokens = torch.cat([history, ck.tokens("decoded", SPAN, case["rows"])[0][:, None]], 1)
        per = max(1, 4800 // tokens.shape[1])
        for at in range(0, case["rows"], per):
            out.append(forward(ck, tokens[at:at + per], [case["context"]])[:, 0])
    for i, n in enumerate(_prompts(case)):
        out.append(forward(ck, ck.tokens(f"prompt.{i}", n)[None], _wanted(case, n))[0])
    return torch.cat(out)


def _rms(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _softmax_attention(q, k, v, scale, seen, sink=None, slopes=None):
    """q [B, T, H, d], k and v [B, S, G, .]; ``seen`` [T, S]: which keys a query reads; a sink is one more term per head of
    the denominator, a slope a penalty per head on the distance.  One query head at a time."""
    group = q.shape[2] // k.shape[2]
    out = []
    for h in range(q.shape[2]):
        s = q[:, :, h] @ k[:, :, h // group].transpose(1, 2) * scale
        if slopes is not None:
            at = torch.arange(s.shape[-1], device=s.device)
            s = s - slopes[h] * (at[:, None] - at[None]).abs()
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(*s.shape[:2], 1)], -1)
        p = torch.softmax(s, -1)[..., :k.shape[1]]
        out.append(p @ v[:, :, h // group])
    return torch.stack(out, 2)


def _seen(T, *, window=None, blocks=None, keep=0):
    i, j = torch.arange(T, device=DEVICE)[:, None], torch.arange(T, device=DEVICE)[None]
    ok = j <= i
    if window is not None:
        ok = ok & ((i - j < window) | (j < keep))
    if blocks is not None:
        ok = ok & (i // blocks == j // blocks)
    return ok


def _angles(T, rot):
    """Angle [T, dims / 2] and the factor on cos and sin; with ``scaling`` the slow pairs' frequencies are divided."""
    dims, base = rot["dims"], rot["base"]
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEVICE) / dims)
    sc, factor = rot.get("scaling"), 1.0
    if sc:
        lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base)) for turns in (sc["fast"], sc["slow"]))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=F64, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, factor = f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    return torch.arange(T, dtype=F64, device=DEVICE)[:, None] * f, factor


def _rotate(x, rot, interleaved):
    """x [B, T, heads, n]: the first ``dims`` entries turned in pairs (2i, 2i+1) or (i, i + dims/2)."""
    if not rot or not rot["dims"]:
        return x
    ang, factor = _angles(x.shape[1], rot)
    cos, sin, dims = (ang.cos() * factor)[:, None], (ang.sin() * factor)[:, None], rot["dims"]
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out = x.clone()
    out[..., a] = x[..., a] * cos - x[..., b] * sin
    out[..., b] = x[..., b] * cos + x[..., a] * sin
    return out


def _conv(x, taps, bias=None):
    """x [B, T, C]; taps [C, K], the last for the current token; nothing before the first token."""
    K = taps.shape[1]
    padded = torch.cat([x.new_zeros(x.shape[0], K - 1, x.shape[2]), x], 1)
    y = sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(K))
    return y if bias is None else y + bias


def _recurrence(update, shape, T):
    """Walks a state over T tokens: ``update(t, S) -> (S, o)``; the outputs [B, T, ...]."""
    S, out = torch.zeros(shape, dtype=F64, device=DEVICE), []
    for t in range(T):
        S, o = update(t, S)
        out.append(o)
    return torch.stack(out, 1)


def _qwen3(case, ck):
    c, w = ck.raw, ck.exact
    nq, nkv, d, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    decoded = ck.tokens("decoded", SPAN, case["rows"])[0] if case["rows"] else None
    rows = [(n, decoded[r:r + 1], [0]) for r, n in enumerate(_contexts(case))]
    rows += [(0, ck.tokens(f"prompt.{i}", n), _wanted(case, n)) for i, n in enumerate(_prompts(case))]
    starts = [0]
    for _, tokens, _ in rows:
        starts.append(starts[-1] + tokens.numel())
    at = torch.cat([torch.arange(n, n + t.numel(), device=DEVICE) for n, t, _ in rows])
    # the model's definition: frequencies and angles are 32-bit numbers
    freq = 1.0 / (c["rope_theta"] ** (torch.arange(0, d, 2, dtype=torch.float32, device="cpu") / d))
    ang = torch.outer(at.float(), freq.to(DEVICE)).to(F64)
    cos, sin = (torch.cat([f, f], -1)[:, None] for f in (ang.cos(), ang.sin()))

    def turn(x):
        return x * cos + torch.cat([-x[..., d // 2:], x[..., :d // 2]], -1) * sin

    table = ck.tensor("model.embed_tokens.weight")
    x = table[torch.cat([t for _, t, _ in rows])].to(F64)
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).view(-1, heads, d) for n, heads in (("q", nq), ("k", nkv), ("v", nkv)))
        q = turn(_rms(q, eps) * w(p + "self_attn.q_norm.weight"))
        k = turn(_rms(k, eps) * w(p + "self_attn.k_norm.weight"))
        parts = []
        for r, (n, tokens, _) in enumerate(rows):
            a, b = starts[r], starts[r + 1]
            kr, vr, T = k[a:b], v[a:b], b - a
            if n:
                past = ck.past(i, r, n)[:, :, :n].transpose(1, 2).to(F64)
                kr, vr = torch.cat([past[0], kr]), torch.cat([past[1], vr])
            seen = torch.arange(n + T, device=DEVICE)[None] <= torch.arange(n, n + T, device=DEVICE)[:, None]
            # the heads of a group of queries read one key head
            s = torch.einsum("tgjd,sgd->gjts", q[a:b].view(T, nkv, nq // nkv, d), kr) * d ** -0.5
            prob = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
            parts.append(torch.einsum("gjts,sgd->tgjd", prob, vr).reshape(T, nq * d))
        x = x + torch.cat(parts) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        x = x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    x = x[[starts[r] + j for r, (_, _, want) in enumerate(rows) for j in want]]
    head = table if c["tie_word_embeddings"] else ck.tensor("lm_head.weight")
    return _rms(x, eps) * w("model.norm.weight") @ head.to(F64).T


def _kogonex(ck, tokens, want):
    c, w, eps = ck.raw, ck.exact, ck.raw["norm"]["eps"]
    B, T = tokens.shape
    big = c["embedding"]["bigram"]
    rows = torch.full_like(tokens, big["buckets"])
    rows[:, 1:] = (tokens[:, :-1] * big["mul_prev"] + tokens[:, 1:] * big["mul_cur"]) % big["buckets"]
    x = ck.tensor("embed")[tokens].to(F64) + ck.tensor("bigram")[rows].to(F64)
    kept = {}

    def latent(i, m, p):
        H, rank = m["heads"], m["kv_rank"]
        q = (x @ w(p + "q").T).view(B, T, H, -1)
        if m.get("kv_from") is None:
            z = x @ w(p + "dkv").T
            kept[i] = _rms(z[..., :rank], eps) * w(p + "dkv.norm"), _rotate(z[:, :, None, rank:], m["rot"], True)
        lat, kr = kept[m["kv_from"] if m.get("kv_from") is not None else i]
        k = torch.cat([(lat @ w(p + "uk").T).view(B, T, H, -1), kr.expand(-1, -1, H, -1)], -1)
        q = torch.cat([q[..., :m["dim"]], _rotate(q[..., m["dim"]:], m["rot"], True)], -1)
        o = _softmax_attention(q, k, (lat @ w(p + "uv").T).view(B, T, H, -1), m["scale"], _seen(T, window=m["mask"]["size"]),
                               sink=w(p + "sink"))
        return o.reshape(B, T, -1) @ w(p + "o").T

    def delta(m, p):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(_conv(x @ w(p + n).T, w(p + n + ".conv"))) for n in "qkv")
        q, k = (y.view(B, T, G, d) / torch.sqrt(y.view(B, T, G, d).square().sum(-1, keepdim=True) + 1e-6) for y in (q, k))
        q, k = (y.repeat_interleave(H // G, 2) for y in (q * d ** -0.5, k))
        v, beta = v.view(B, T, H, dv), torch.sigmoid(x @ w(p + "b").T)
        step = torch.nn.functional.softplus((x @ w(p + "a1").T) @ w(p + "a2").T + w(p + "dt_bias")).view(B, T, H, d)
        g = torch.exp(-torch.exp(w(p + "A_log"))[:, None] * step)

        def update(t, S):
            S = g[:, t, :, :, None] * S
            u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", S, k[:, t]))
            S = S + k[:, t, :, :, None] * u[:, :, None]
            return S, torch.einsum("bhdv,bhd->bhv", S, q[:, t])

        gate = torch.sigmoid((x @ w(p + "g1").T) @ w(p + "g2").T).view(B, T, H, dv)
        o = _rms(_recurrence(update, (B, H, d, dv), T), eps) * w(p + "norm") * gate
        return o.reshape(B, T, -1) @ w(p + "o").T

    def experts(f, p):
        r, h = f["router"], x.view(B * T, -1)
        s = torch.softmax(h @ w(p + "router").T, -1)
        choice = s + w(p + "correction")
        n, groups = choice.shape[1], r["groups"]["count"]
        best = choice.view(-1, groups, n // groups).max(-1).values.topk(r["groups"]["keep"], -1).indices
        allowed = torch.zeros(B * T, groups, dtype=torch.bool, device=DEVICE).scatter(1, best, True)
        choice = choice.masked_fill(~allowed.repeat_interleave(n // groups, 1), -math.inf)
        weight = torch.zeros_like(s).scatter(1, choice.topk(r["top"], -1).indices, 1.0) * s
        y = weight[:, r["experts"]:].sum(-1, keepdim=True) * h                  # the identity experts
        for e in range(r["experts"]):
            t = weight[:, e].nonzero()[:, 0]
            he = h[t]
            y[t] += weight[t, e, None] * ((_silu(he @ w(f"{p}e{e}.gate").T) * (he @ w(f"{p}e{e}.up").T)) @ w(f"{p}e{e}.down").T)
        return y.view(B, T, -1)

    for i, layer in enumerate(c["layers"]):
        m, p = layer["mixer"], f"l{i}."
        y = latent(i, m, p + "mix.") if layer["type"] == "latent_attention" else delta(m, p + "mix.")
        x = x + _rms(y, eps) * w(p + "norm1")
        x = x + _rms(experts(layer["mlp"], p + "mlp."), eps) * w(p + "norm2")
    return _rms(x[:, want], eps) * w("final.norm") @ w("head").T


def _vagulorn(ck, tokens, want):
    c, w, eps = ck.raw, ck.exact, ck.raw["norm"]["eps"]
    B, T = tokens.shape

    def layer_norm(x, p):
        x = x - x.mean(-1, keepdim=True)
        return _rms(x, eps) * w(p) + w(p + ".b")

    def attention(m, p, h, beside):
        heads = lambda y, n: y.view(B, T, n, -1)  # noqa: E731
        q, k = heads(h @ w(p + "q").T, m["heads"]), heads(h @ w(p + "k").T, m["kv_heads"])
        v = k if beside else heads(h @ w(p + "v").T, m["kv_heads"])
        q, k = (_rotate(_rms(y, eps) * w(p + n), m["rot"], beside) for y, n in ((q, "q.norm"), (k, "k.norm")))
        size = m["mask"]["size"]
        seen = _seen(T, window=size, keep=m["mask"].get("keep_first", 0)) if beside else _seen(T, blocks=size)
        o = _softmax_attention(q, k, v, m["scale"], seen)
        if beside:
            o = o * torch.sigmoid(h @ w(p + "g").T)[..., None]
        return o.reshape(B, T, -1) @ w(p + "o").T

    def linear(m, p, h):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(h @ w(p + n).T).view(B, T, H, -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=F64, device=DEVICE)[:, None, None]

        def update(t, S):
            S = decay * S + k[:, t, :, :, None] * v[:, t, :, None]
            return S, torch.einsum("bhdv,bhd->bhv", S, q[:, t])

        o = _recurrence(update, (B, H, d, dv), T).reshape(B, T, -1)
        return (_rms(o, eps) * w(p + "norm") * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T

    def space(m, p, h):
        H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        z, xbc, dt = (h @ w(p + "in").T).split([H * V, H * V + 2 * G * N, H], -1)
        u, b, g = _silu(_conv(xbc, w(p + "conv"), w(p + "conv.b"))).split([H * V, G * N, G * N], -1)
        u = u.view(B, T, H, V)
        b, g = (y.reshape(B, T, G, N).repeat_interleave(H // G, 2) for y in (b, g))
        dt = torch.nn.functional.softplus(dt + w(p + "dt_bias"))
        a, D = torch.exp(-torch.exp(w(p + "A_log")) * dt), w(p + "D")[:, None]

        def update(t, S):
            S = a[:, t, :, None, None] * S + (dt[:, t, :, None] * b[:, t])[..., None] * u[:, t, :, None]
            return S, torch.einsum("bhnv,bhn->bhv", S, g[:, t]) + D * u[:, t]

        y = _recurrence(update, (B, H, N, V), T).reshape(B, T, -1) * _silu(z)
        y = _rms(y.view(B, T, m["norm_groups"], -1), eps).reshape(B, T, -1) * w(p + "norm")
        return y @ w(p + "o").T

    x = ck.tensor("embed")[tokens].to(F64) * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        m, p = layer["mixer"], f"l{i}."
        h, q = layer_norm(x, p + "norm1"), p + "mix."
        if layer["type"] == "attention":
            y = attention(m, q, h, False)
        elif layer["type"] == "parallel":
            y = m["left_scale"] * attention(m["left"], q + "left.", h, True) + m["right_scale"] * linear(m["right"], q + "right.", h)
        else:
            y = space(m, q, h)
        x = x + y + (_gelu(h @ w(p + "mlp.gate").T) * (h @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
    return layer_norm(x[:, want], "final.norm") @ w("embed").T


def _tedenex(ck, tokens, want):
    c, w, eps = ck.raw, ck.exact, ck.raw["norm"]["eps"]
    B, T = tokens.shape

    def norm(x, p):
        return _rms(x, eps) * (1.0 + w(p))

    def attention(m, p, h):
        def project(n, heads):
            return _conv(h @ w(p + n).T + w(p + n + ".b"), w(p + n + ".conv")).view(B, T, heads, -1)

        H = m["heads"]
        q, k, v = project("q", H), project("k", m["kv_heads"]), project("v", m["kv_heads"])
        o = _softmax_attention(_rms(q, eps) * w(p + "q.norm"), _rms(k, eps) * w(p + "k.norm"), v, m["scale"],
                               _seen(T, blocks=m["mask"]["size"]), slopes=[2.0 ** (-8.0 * (a + 1) / H) for a in range(H)])
        return o.reshape(B, T, -1) @ w(p + "o").T

    def mixing(m, p, h):
        H, d = m["heads"], m["dim"]
        before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
        blend = {s: h + (before - h) * w(p + "mu." + s) for s in "rkvgw"}
        r, k, v = ((blend[s] @ w(p + s).T).view(B, T, H, d) for s in "rkv")
        decay = torch.exp(-torch.exp(torch.tanh(blend["w"] @ w(p + "w1").T) @ w(p + "w2").T + w(p + "w0"))).view(B, T, H, d)
        first = w(p + "u")[..., None]

        def update(t, S):
            kv = k[:, t, :, :, None] * v[:, t, :, None]
            return decay[:, t, :, :, None] * S + kv, torch.einsum("bhdv,bhd->bhv", S + first * kv, r[:, t])

        o = _rms(_recurrence(update, (B, H, d, d), T), eps).reshape(B, T, -1)
        return (o * w(p + "norm") * _silu(blend["g"] @ w(p + "g").T)) @ w(p + "o").T

    def latent(m, p, h):
        H, d, rank = m["heads"], m["dim"], m["kv_rank"]
        q = ((_rms(h @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T).view(B, T, H, -1)
        z = h @ w(p + "dkv").T
        lat = _rms(z[..., :rank], eps) * w(p + "dkv.norm")
        kr = _rotate(z[:, :, None, rank:], m["rot"], True).expand(-1, -1, H, -1)
        k = torch.cat([(lat @ w(p + "uk").T).view(B, T, H, d), kr], -1)
        q = torch.cat([q[..., :d], _rotate(q[..., d:], m["rot"], True)], -1)
        o = _softmax_attention(q, k, (lat @ w(p + "uv").T).view(B, T, H, -1), m["scale"], _seen(T))
        return o.reshape(B, T, -1) @ w(p + "o").T

    mixers = {"attention": attention, "wkv": mixing, "latent_attention": latent}
    loop, order = c["loop"], list(range(len(c["layers"])))
    span = order[loop["start"]:loop["stop"]]
    order = [(i, False) for i in order[:loop["start"]]] + [(i, n > 0 and i == span[0]) for n in range(loop["times"]) for i in span] + [
        (i, False) for i in order[loop["stop"]:]]
    side, dim = ck.tensor("side.embed")[tokens], c["token_side"]["dim"]
    entered = ck.tensor("embed")[tokens].to(F64)
    x = entered
    for i, again in order:
        layer, p = c["layers"][i], f"l{i}."
        x = x + entered if again else x
        x = x + norm(mixers[layer["type"]](layer["mixer"], p + "mix.", norm(x, p + "norm1")), p + "norm1b")
        y = (norm(x, p + "norm2") @ w(p + "mlp.up").T).clamp(min=0).square() @ w(p + "mlp.down").T
        x = x + norm(y, p + "norm2b")
        y = (_gelu(x @ w(p + "side.gate").T) * side[..., i * dim:(i + 1) * dim].to(F64)) @ w(p + "side.proj").T
        x = x + _rms(y, eps) * w(p + "side.norm")
    return norm(x[:, want], "final.norm") @ w("embed").T


def _splitmix64(z):
    mask = 2 ** 64 - 1
    z = (z + 0x9E3779B97F4A7C15) & mask
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
    return z ^ (z >> 31)


def _sample(state):
    tokens, logprobs = [], []
    for x, p, counter in zip(state.logits.to(F64), state.params, state.counters):
        x = x / p.temperature
        if p.top_k:
            x = x.masked_fill(x < x.topk(p.top_k).values[-1], -math.inf)
        if p.top_p < 1.0:
            ascending, order = x.sort()
            drop = ascending.softmax(-1).cumsum(-1) <= 1.0 - p.top_p
            drop[-1] = False
            x = x.masked_fill(torch.zeros_like(drop).scatter(0, order, drop), -math.inf)
        u = (_splitmix64(_splitmix64(p.seed) ^ (counter * 0xD1342543DE82EF95 & (2 ** 64 - 1))) >> 40) / 2.0 ** 24
        prob = x.softmax(-1)
        t = int((prob.cumsum(-1) <= u).sum().clamp(max=x.numel() - 1))
        tokens.append(t)
        logprobs.append(float(prob[t].log()))
    return torch.tensor(tokens, dtype=torch.int32), torch.tensor(logprobs, dtype=F64)
