"""What is timed when this engine's speed is measured: steps of the step function as a serving program makes them.

Every case is one stretch of serving on a loaded model (random weights of a real architecture's sizes).  A number of
requests are being decoded already (``running``, their contexts in the paged cache); ``prompts`` new requests arrive
with ``tokens`` prompt tokens between them and are run in portions of at most ``portion`` tokens a step beside the
decoded ones; then ``steps`` more tokens are decoded for all of them, and the new requests end.  Token ids are given,
as in a replay, so that two implementations run the same work; what comes back is the float32 logits of every wanted
place, step by step.  One pass is one such stretch, through ``ModelRunner.step`` and the cache manager's
``open``/``close`` (the calls that ``LLM.generate`` and the trace replay make).

The running requests go on from pass to pass for ``TURN`` new tokens; then they start again from their prompts, whose
pages other requests hold (a shared prefix).  Contexts in the cache are whole pages, prompts of any length.
"""
from __future__ import annotations

import hashlib
import math
import random

import torch

from qwen_engine_b200.cache.manager import CacheManager
from qwen_engine_b200.config import preset_config_dict
from qwen_engine_b200.engine.runner import ModelRunner, StepEntry
from qwen_engine_b200.registry import build_model, config_from_dict

PAGE = 16
TURN = 256             # tokens that a running request gains before it starts again from its prompt
FILL = 4096            # tokens a step while the contexts are filled
DEVICE = "cuda:0"


# ---- the cases -------------------------------------------------------------------------------------------------------

def _case(name, model, dtype="bfloat16", running=0, context=0, ragged=False, shared=0, prompts=0, tokens=0, portion=2048,
          steps=0):
    c = dict(model=model, dtype=dtype, running=running, context=context, ragged=ragged, shared=shared, prompts=prompts,
             tokens=tokens, portion=portion, steps=steps)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short question on an idle engine: the time to its first token, all latency
        _case("0.6b-prompt-23", "qwen3-0.6b", prompts=1, tokens=23),
        # one prompt that fills the default token budget
        _case("0.6b-prompt-2048", "qwen3-0.6b", prompts=1, tokens=2048),
        # one user's answer streaming
        _case("0.6b-decode-1", "qwen3-0.6b", running=1, context=1024, steps=16),
        # a few users, contexts of every length
        _case("0.6b-decode-8", "qwen3-0.6b", running=8, context=1024, ragged=True, steps=16),
        # a loaded server with a small model
        _case("0.6b-decode-64", "qwen3-0.6b", running=64, context=1024, steps=16),
        # the 32-bit path, as one checks a model: ragged prompts in one step, a few decoded tokens
        _case("0.6b-float32", "qwen3-0.6b", dtype="float32", prompts=3, tokens=141, steps=4),
        # chunked prefill: a prompt of odd length goes through in portions of 512 beside fifteen decoded requests
        _case("1.7b-mixed", "qwen3-1.7b", running=15, context=1088, ragged=True, prompts=1, tokens=1403, portion=512),
        # the same server between arrivals, contexts as prompts of 128 to 2 048 tokens leave them
        _case("1.7b-decode-28", "qwen3-1.7b", running=28, context=1088, ragged=True, steps=16),
        # eight requests bring their own 256 tokens behind a system prompt of 1 024 that is in the cache
        _case("4b-suffixes", "qwen3-4b", shared=1024, prompts=8, tokens=2051),
        # sixteen such requests being decoded
        _case("4b-decode-16", "qwen3-4b", running=16, context=1280, shared=1024, steps=16),
        # the designs with recurrent state: a prompt and the first tokens of its answer, and a batch of ragged ones
        _case("ganidra-request", "ganidra-w1024", prompts=1, tokens=2048, steps=16),
        _case("funudra-requests", "funudra-w1024", prompts=4, tokens=1531, steps=16),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["prompt", "prompt", "decode", "decode", "decode", "mixed", "float32", "state"])
    model = rng.choice(["qwen3-0.6b", "qwen3-1.7b", "qwen3-4b"])
    most_running = {"qwen3-0.6b": 64, "qwen3-1.7b": 32, "qwen3-4b": 16}[model]
    if kind == "prompt":
        prompts = rng.choice([1, 1, 2, 3, 8])
        tokens = max(prompts, _log_uniform(rng, 5, 2560))
        return _case(None, model, prompts=prompts, tokens=tokens, shared=PAGE * rng.choice([0, 0, rng.randint(1, 96)]),
                     portion=rng.choice([512, 2048]))
    if kind == "decode":
        return _case(None, model, running=_log_uniform(rng, 1, most_running), context=PAGE * _log_uniform(rng, 4, 96),
                     ragged=rng.random() < 0.6, steps=rng.randint(8, 16))
    if kind == "mixed":
        return _case(None, model, running=_log_uniform(rng, 1, most_running // 2), context=PAGE * _log_uniform(rng, 4, 96),
                     ragged=True, prompts=rng.choice([1, 2]), tokens=_log_uniform(rng, 64, 1600), portion=rng.choice([256, 512]),
                     steps=rng.randint(0, 4))
    if kind == "float32":
        prompts = rng.choice([1, 2, 3, 4])
        return _case(None, "qwen3-0.6b", dtype="float32", prompts=prompts, tokens=_log_uniform(rng, 8, 256), steps=rng.randint(0, 6))
    prompts = rng.choice([1, 2, 4, 8])
    return _case(None, rng.choice(["ganidra-w1024", "funudra-w1024"]), prompts=prompts, tokens=_log_uniform(rng, 32, 2048),
                 steps=rng.randint(4, 16))


# ---- lengths and the order of work: the same for every seed ------------------------------------------------------------

def _split(total, parts, rng):
    """``total`` tokens in ``parts`` prompts of ragged lengths, at least one each."""
    if parts == 0:
        return []
    shares = [rng.uniform(0.5, 1.5) for _ in range(parts)]
    lens = [max(1, int(total * s / sum(shares))) for s in shares]
    lens[0] += total - sum(lens)
    return lens


def _lengths(case):
    """Contexts of the running requests (whole pages, the shared prefix included) and lengths of the new prompts."""
    rng = random.Random("%s %s %s" % (case["running"], case["context"], case["tokens"]))
    least = case["shared"] // PAGE + 1
    pages = case["context"] // PAGE
    contexts = [PAGE * max(least, round(pages * rng.uniform(0.12, 1.88)) if case["ragged"] else pages) for _ in range(case["running"])]
    return contexts, _split(case["tokens"], case["prompts"], rng)


def _order(case):
    """The steps of a pass: for each, how many tokens every new request runs (running requests run one in each)."""
    _, lens = _lengths(case)
    fed, out, left = [0] * len(lens), [], case["steps"]
    while True:
        room, row = case["portion"], []
        feeding = any(f < n for f, n in zip(fed, lens))
        if not feeding:
            if left == 0:
                return out
            left -= 1
        for i, n in enumerate(lens):
            k = 1 if fed[i] >= n else min(room, n - fed[i])
            if fed[i] < n:
                room -= k
            row.append(k)
            fed[i] += k
        out.append(row)


# ---- models --------------------------------------------------------------------------------------------------------------

def _config(model):
    if model in ("qwen3-0.6b", "qwen3-1.7b", "qwen3-4b"):
        return preset_config_dict(model)
    width, ff, heads, kv_heads, dim, window, vocab, pairs = 1024, 3072, 16, 8, 128, 1024, 32768, 4
    if model == "ganidra-w1024":
        gla = dict(heads=8, dim=64, vdim=128, tau=16.0, rank=16)
        left = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, mask=dict(size=window), scale=dim ** -0.5)
        mlp = dict(kind="dense", ff=ff)
        layers = [dict(type="gla", mixer=gla, mlp=mlp),
                  dict(type="parallel", mixer=dict(left=left, right=dict(gla, heads=4), left_scale=0.7, right_scale=0.7), mlp=mlp)]
        return dict(architecture="Ganidra", vocab=vocab, width=width, embedding=dict(scale=1.0), norm=dict(eps=1e-6),
                    layers=layers * pairs, loop=dict(start=0, stop=0, times=1))
    ssm = dict(heads=2 * width // 64, vdim=64, state=128, groups=8, conv=4, norm_groups=8)
    left = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=2 * dim, conv=4, scale=dim ** -0.5, softcap=50.0,
                rot=dict(base=500000.0, dims=dim // 2, scaling=dict(factor=4.0)))
    right = dict(heads=4, dim=64, vdim=128, gate_cap=15.0)
    mlp = dict(kind="dense", ff=ff)
    layers = [dict(type="mamba2", mixer=ssm, mlp=mlp),
              dict(type="parallel", mixer=dict(left=left, right=right, left_scale=0.7, right_scale=0.7), mlp=mlp)]
    return dict(architecture="Funudra", vocab=vocab, width=width, norm=dict(eps=1e-6), layers=layers * pairs)


def _drawn(seed, name, shape, kind):
    """One weight tensor, rounded to bfloat16 as a checkpoint stores it: matrices N(0, 0.41 / inputs) (0.02 at a width of
    1 024) whatever the width, the table N(0, 0.02^2), norm scales around one (or zero), biases N(0, 1), taps N(0, 1 / n).
    The matrices that write back into the stream are 16 times smaller, so that a layer changes the stream by a part of it,
    as in a trained model."""
    digest = hashlib.blake2b(("%d:%s" % (seed, name)).encode(), digest_size=7).digest()
    gen = torch.Generator(device=DEVICE).manual_seed(int.from_bytes(digest, "little"))
    t = torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32)
    if kind == "norm":
        t = 1.0 + 0.1 * t
    elif kind == "norm_zero":
        t = 0.1 * t
    elif kind == "taps":
        t = t * shape[-1] ** -0.5
    elif kind == "matrix":
        table, back = "embed" in name, name.removesuffix("_proj.weight").rsplit(".", 1)[-1] in ("o", "down")
        t = t * (0.02 if table else 0.64 * shape[-1] ** -0.5 / (16 if back else 1))
    return t.to(torch.bfloat16)


class _Weights:
    """A source of tensors by checkpoint name, drawn on the device when asked."""

    def __init__(self, manifest, seed):
        self._specs = {s.name: s for s in manifest if not s.optional}
        self._seed = seed

    def names(self):
        return self._specs.keys()

    def shape(self, name):
        return self._specs[name].drawn_shape

    def get(self, name):
        return _drawn(self._seed, name, self._specs[name].drawn_shape, self._specs[name].kind)


def _tokens(case, seed):
    """Token ids: the shared prefix; per running request its context and what is decoded; per new request its prompt and
    what is decoded after it."""
    rng = random.Random("tokens %d" % seed)
    cfg = _config(case["model"])
    vocab = cfg.get("vocab_size", cfg.get("vocab"))
    ids = lambda n: [rng.randrange(vocab) for _ in range(n)]
    contexts, lens = _lengths(case)
    shared = ids(case["shared"])
    running = [(shared + ids(n - len(shared)), ids(TURN)) for n in contexts]
    fresh = [(ids(n), ids(len(_order(case)))) for n in lens]
    return shared, running, fresh


# ---- one stretch of serving ------------------------------------------------------------------------------------------------

class _Serving:
    """A loaded model with its cache, the running requests' contexts in it, and the token ids of a pass."""

    def __init__(self, case, seed):
        dtype = getattr(torch, case["dtype"])
        self.case, self.order = case, _order(case)
        self.shared, self.running_tokens, self.fresh_tokens = _tokens(case, seed)
        model = build_model(config_from_dict(_config(case["model"])))
        model.load_weights(_Weights(model.weight_manifest(), seed), dtype, DEVICE, "drawn weights")
        contexts, lens = _lengths(case)
        pages = len(self.shared) // PAGE + sum(n // PAGE for n in contexts) + len(contexts) * (TURN // PAGE + 2)
        pages += sum((n + len(self.order)) // PAGE + 2 for n in lens) + 8
        self.cache = CacheManager(model.cache_specs(), PAGE, pages, 2 * len(contexts) + len(lens) + 1, dtype, DEVICE)
        self.runner = ModelRunner(model, self.cache, DEVICE, dtype)
        # requests that hold the contexts' pages for as long as the state lives
        held = []
        if self.shared:
            held.append((self.cache.open("shared"), self.shared))
        self._fill(held)
        n = len(self.shared)
        held = [(self.cache.open("held %d" % i, self.shared + t[n:n + 1] if n else None, n), t)
                for i, (t, _) in enumerate(self.running_tokens)]
        self._fill(held)
        self.running, self.turn = [], TURN
        self._again()

    def _fill(self, held):
        batch, room = [], FILL
        for rc, tokens in held:
            at = rc.num_tokens
            while at < len(tokens):
                k = min(room, len(tokens) - at)
                batch.append(StepEntry(rc, tokens[at:at + k]))
                at, room = at + k, room - k
                if room == 0:
                    self.runner.step(batch)
                    batch, room = [], FILL
        if batch:
            self.runner.step(batch)

    def _again(self):
        """The running requests start (again) behind their contexts."""
        for rc in self.running:
            self.cache.close(rc)
        self.running = [self.cache.open("running %d" % i, t + more[:1], len(t)) for i, (t, more) in enumerate(self.running_tokens)]
        self.turn = 0

    def serve(self):
        if self.running and self.turn + len(self.order) > TURN:
            self._again()
        n = len(self.shared)
        fresh = [self.cache.open("new %d" % i, self.shared + t[:1] if n else None, n) for i, (t, _) in enumerate(self.fresh_tokens)]
        fed = [0] * len(fresh)
        logits = []
        for row in self.order:
            entries = [StepEntry(rc, [more[self.turn]], [0]) for rc, (_, more) in zip(self.running, self.running_tokens)]
            for i, k in enumerate(row):
                if k:
                    prompt, more = self.fresh_tokens[i]
                    tokens = prompt[fed[i]:fed[i] + k] if fed[i] < len(prompt) else [more[fed[i] - len(prompt)]]
                    fed[i] += k
                    entries.append(StepEntry(fresh[i], tokens, [k - 1] if fed[i] >= len(prompt) else []))
            self.turn += 1
            out = self.runner.step(entries)
            if out is not None:
                logits.append(out.clone())       # the step's own buffer is written again by the next step
        for rc in fresh:
            self.cache.close(rc)
        return logits


def prepare(case, seed):
    return _Serving(case, seed)


def run(state):
    return state.serve()


# ---- what a pass cannot do without, and how close its results are ------------------------------------------------------------

def _matrix_sizes(case):
    """Elements of the matrices that every token passes, and of the head."""
    cfg = _config(case["model"])
    if "hidden_size" in cfg:
        H, D = cfg["hidden_size"], cfg["head_dim"]
        heads, kv, I = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"]
        layer = H * D * (2 * heads + 2 * kv) + 3 * H * I
        return cfg["num_hidden_layers"] * layer, cfg["vocab_size"] * H
    total = 0
    W = cfg["width"]
    for spec in cfg["layers"]:
        m = spec["mixer"]
        if spec["type"] == "mamba2":
            inner = m["heads"] * m["vdim"]
            total += W * (2 * inner + 2 * m["groups"] * m["state"] + m["heads"]) + inner * W
        for part in ([m] if spec["type"] == "gla" else [m["right"]] if spec["type"] == "parallel" else []):
            total += W * part["heads"] * (2 * part["dim"] + 3 * part["vdim"])
        if spec["type"] == "parallel":
            a = m["left"]
            total += W * (a["heads"] * (a["dim"] + 2 * a["vdim"]) + a["kv_heads"] * (a["dim"] + a["vdim"]))
        total += W * spec["mlp"]["ff"] * (3 if cfg["architecture"] == "Ganidra" else 2)
    return total, cfg["vocab"] * W


def _memories(case):
    """Softmax layers (cache elements a token, query elements a token, window) and elements of recurrent state."""
    cfg = _config(case["model"])
    if "hidden_size" in cfg:
        D = cfg["head_dim"]
        n = cfg["num_hidden_layers"]
        return n * 2 * cfg["num_key_value_heads"] * D, n * 2 * cfg["num_attention_heads"] * D, None, 0
    kv = q = state = 0
    window = None
    for spec in cfg["layers"]:
        m = spec["mixer"]
        if spec["type"] == "mamba2":
            state += m["heads"] * m["vdim"] * m["state"]
        else:
            r = m if spec["type"] == "gla" else m["right"]
            state += r["heads"] * r["dim"] * r["vdim"]
        if spec["type"] == "parallel":
            a = m["left"]
            kv += a["kv_heads"] * (a["dim"] + a["vdim"])
            q += a["heads"] * (a["dim"] + a["vdim"])
            window = a.get("mask", {}).get("size")
    return kv, q, window, state


def work(case):
    """Per step: every matrix read once, the caches of its requests read and their new entries written, the logits
    written; two operations a weight and token, and the scores and weighted sums of the causal attention."""
    size = 2 if case["dtype"] == "bfloat16" else 4
    matrices, head = _matrix_sizes(case)
    kv, q, window, state = _memories(case)
    vocab = head // (_config(case["model"]).get("hidden_size") or _config(case["model"])["width"])
    contexts, lens = _lengths(case)
    at = list(contexts) + [case["shared"]] * len(lens)
    prompt_end = [0] * len(contexts) + [case["shared"] + n for n in lens]
    nbytes = flops = 0.0
    for row in _order(case):
        tokens = [1] * len(contexts) + row
        wanted = sum(1 for a, k, e in zip(at, tokens, prompt_end) if k and a + k >= e)
        T = sum(tokens)
        nbytes += size * (matrices + (head if wanted else 0)) + 4.0 * wanted * vocab
        flops += 2.0 * matrices * T + 2.0 * head * wanted
        for i, k in enumerate(tokens):
            if k:
                reach = lambda n: min(n, window) if window else n
                nbytes += size * kv * (min(at[i], reach(at[i] + k)) + k) + 2 * 4.0 * state
                flops += 2.0 * q * sum(reach(a + 1) for a in range(at[i], at[i] + k)) + 4.0 * state * k
            at[i] += k
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # measured against 64 bits: Qwen3 and Funudra logits in bfloat16 are 0.2 to 0.6 % off, Ganidra's 1.5 % (its per-head
    # norms follow sums that nearly cancel), 32-bit ones 2e-6; two implementations differ by up to twice that and more
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03 if case["model"].startswith("ganidra") else 0.02, "max": 0.5}


# ---- the same logits in 64 bits, plain torch -----------------------------------------------------------------------------------

def exact(case, seed):
    shared, running, fresh = _tokens(case, seed)
    order = _order(case)
    cfg = _config(case["model"])
    forward = {"Ganidra": _Ganidra, "Funudra": _Funudra}.get(cfg.get("architecture"), _Qwen3)(cfg, seed)
    contexts, lens = _lengths(case)
    # the places of every request whose logits some step wants, in order
    rows = []
    for tokens, more in running:
        ids = tokens + more[:len(order)]
        rows.append(forward(ids, len(tokens)))
    counts = [0] * len(fresh)
    for row in order:
        for i, k in enumerate(row):
            counts[i] += k
    for (prompt, more), n in zip(fresh, counts):
        ids = shared + prompt + more[:n - len(prompt)]
        rows.append(forward(ids, len(shared) + len(prompt) - 1))
    out, at, fed = [], [0] * len(rows), [0] * len(fresh)
    for row in order:
        step = []
        for r in range(len(running)):
            step.append(rows[r][at[r]])
            at[r] += 1
        for i, k in enumerate(row):
            fed[i] += k
            r = len(running) + i
            if k and fed[i] >= lens[i]:
                step.append(rows[r][at[r]])
                at[r] += 1
        if step:
            out.append(torch.stack(step))
    return out


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _rotate(x, dims, freqs):
    """x [T, heads, D]: the pairs (i, i + dims / 2) of the first ``dims`` channels turn by position * freqs[i]."""
    half = dims // 2
    a = (torch.arange(x.shape[0], dtype=x.dtype, device=x.device)[:, None] * freqs[None, :])[:, None, :]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * torch.cos(a) - v * torch.sin(a), v * torch.cos(a) + u * torch.sin(a), x[..., dims:]], dim=-1)


def _attention(q, k, v, bend, window=None):
    """q [T, H, D], k [T, G, D], v [T, G, Dv]: causal softmax attention of one request; ``bend(scores, distance)``."""
    T, H, _ = q.shape
    group = H // k.shape[1]
    kt = k.repeat_interleave(group, 1).permute(1, 2, 0)
    vh = v.repeat_interleave(group, 1).transpose(0, 1)
    place = torch.arange(T, device=q.device)
    out = []
    for lo in range(0, T, 512):
        hi = min(T, lo + 512)
        apart = (place[lo:hi, None] - place[None, :hi])
        s = bend(q[lo:hi].transpose(0, 1) @ kt[:, :, :hi], apart.to(q.dtype))
        hidden = apart < 0 if window is None else (apart < 0) | (apart >= window)
        out.append((torch.softmax(s.masked_fill(hidden, -math.inf), dim=-1) @ vh[:, :hi]).transpose(0, 1))
    return torch.cat(out)


class _Plain:
    """A decoder in 64 bits: calling it gives the logits of one request's tokens from place ``first`` on."""

    def __init__(self, cfg, seed):
        self.cfg, self.seed, self._kept = cfg, seed, {}

    def w(self, name, *shape, kind="matrix"):
        if name not in self._kept:
            self._kept[name] = _drawn(self.seed, name, shape, kind).double()
        return self._kept[name]

    def lin(self, x, name, rows):
        return x @ self.w(name, rows, x.shape[-1]).T


class _Qwen3(_Plain):
    def __call__(self, ids, first):
        c = self.cfg
        H, D, I, eps = c["hidden_size"], c["head_dim"], c["intermediate_size"], c["rms_norm_eps"]
        heads, kv = c["num_attention_heads"], c["num_key_value_heads"]
        T = len(ids)
        freqs = c["rope_theta"] ** (-torch.arange(0, D, 2, dtype=torch.float64, device=DEVICE) / D)
        table = self.w("model.embed_tokens.weight", c["vocab_size"], H)
        x = table[torch.tensor(ids, device=DEVICE)]
        norm = lambda t, name, n: _rms(t, eps) * self.w(name, n, kind="norm")
        for i in range(c["num_hidden_layers"]):
            p = "model.layers.%d." % i
            a = p + "self_attn."
            h = norm(x, p + "input_layernorm.weight", H)
            q = norm(self.lin(h, a + "q_proj.weight", heads * D).view(T, heads, D), a + "q_norm.weight", D)
            k = norm(self.lin(h, a + "k_proj.weight", kv * D).view(T, kv, D), a + "k_norm.weight", D)
            v = self.lin(h, a + "v_proj.weight", kv * D).view(T, kv, D)
            o = _attention(_rotate(q, D, freqs), _rotate(k, D, freqs), v, lambda s, _: s * D ** -0.5)
            x = x + self.lin(o.reshape(T, heads * D), a + "o_proj.weight", H)
            h = norm(x, p + "post_attention_layernorm.weight", H)
            u = _silu(self.lin(h, p + "mlp.gate_proj.weight", I)) * self.lin(h, p + "mlp.up_proj.weight", I)
            x = x + self.lin(u, p + "mlp.down_proj.weight", H)
        return norm(x[first:], "model.norm.weight", H) @ table.T


class _Ganidra(_Plain):
    def _gla(self, h, p, m, eps):
        T, H, dk, dv = h.shape[0], m["heads"], m["dim"], m["vdim"]
        q = self.lin(h, p + "q", H * dk).view(T, H, dk) * dk ** -0.5
        k = self.lin(h, p + "k", H * dk).view(T, H, dk)
        v = self.lin(h, p + "v", H * dv).view(T, H, dv)
        z = self.lin(self.lin(h, p + "a1", m["rank"]), p + "a2", H * dk) + self.w(p + "a2.b", H * dk, kind="vector")
        keep = (torch.sigmoid(z) ** (1.0 / m["tau"])).view(T, H, dk)
        S = torch.zeros(H, dk, dv, dtype=h.dtype, device=h.device)
        o = torch.empty(T, H, dv, dtype=h.dtype, device=h.device)
        for t in range(T):
            S = torch.baddbmm(keep[t, :, :, None] * S, k[t, :, :, None], v[t, :, None, :])
            o[t] = (q[t, :, None, :] @ S)[:, 0]
        o = (_rms(o, eps) * self.w(p + "norm", dv, kind="norm")).reshape(T, H * dv)
        return self.lin(o * _silu(self.lin(h, p + "g", H * dv)), p + "o", self.cfg["width"])

    def _softmax(self, h, p, m, eps):
        T, H, G, dk, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q = _rms(self.lin(h, p + "q", H * dk).view(T, H, dk), eps) * self.w(p + "q.norm", dk, kind="norm")
        k = _rms(self.lin(h, p + "k", G * dk).view(T, G, dk), eps) * self.w(p + "k.norm", dk, kind="norm")
        v = self.lin(h, p + "v", G * dv).view(T, G, dv)
        slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=h.dtype, device=h.device) / H)
        o = _attention(q, k, v, lambda s, apart: s * m["scale"] - slopes[:, None, None] * apart, m["mask"]["size"])
        return self.lin(o.reshape(T, H * dv) * torch.sigmoid(self.lin(h, p + "g", H * dv)), p + "o", self.cfg["width"])

    def __call__(self, ids, first):
        c = self.cfg
        W, eps = c["width"], c["norm"]["eps"]
        table = self.w("embed", c["vocab"], W)
        norm = lambda t, name: _rms(t, eps) * (1.0 + self.w(name, W, kind="norm_zero"))
        x = table[torch.tensor(ids, device=DEVICE)] * c["embedding"]["scale"]
        for i, spec in enumerate(c["layers"]):
            p, m = "l%d." % i, spec["mixer"]
            h = norm(x, p + "norm1")
            if spec["type"] == "gla":
                x = x + self._gla(h, p + "mix.", m, eps)
            else:
                x = x + m["left_scale"] * self._softmax(h, p + "mix.left.", m["left"], eps) \
                    + m["right_scale"] * self._gla(h, p + "mix.right.", m["right"], eps)
            h, ff = norm(x, p + "norm2"), spec["mlp"]["ff"]
            u = torch.nn.functional.gelu(self.lin(h, p + "mlp.gate", ff), approximate="tanh") * self.lin(h, p + "mlp.up", ff)
            x = x + self.lin(u, p + "mlp.down", W)
        return norm(x[first:], "final.norm") @ table.T


class _Funudra(_Plain):
    def _conv(self, u, name, bias=None):
        n = 4
        taps = self.w(name, u.shape[1], n, kind="taps")
        y = sum(taps[:, j] * torch.nn.functional.pad(u, (0, 0, n - 1 - j, 0))[:u.shape[0]] for j in range(n))
        return y if bias is None else y + bias

    def _softmax(self, h, p, m):
        T, H, G, dk, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        vec = lambda name, n: self.w(name, n, kind="vector")
        q, k, v = (self._conv(self.lin(h, p + n, size) + vec(p + n + ".b", size), p + n + ".conv").view(T, -1, d)
                   for n, size, d in (("q", H * dk, dk), ("k", G * dk, dk), ("v", G * dv, dv)))
        rot = m["rot"]
        freqs = rot["base"] ** (-torch.arange(0, rot["dims"], 2, dtype=h.dtype, device=h.device) / rot["dims"]) / rot["scaling"]["factor"]
        cap = m["softcap"]
        o = _attention(_rotate(q, rot["dims"], freqs), _rotate(k, rot["dims"], freqs), v,
                       lambda s, _: cap * torch.tanh(s * m["scale"] / cap))
        o = o.reshape(T, H * dv) * torch.sigmoid(self.lin(h, p + "g", H * dv))
        return self.lin(o, p + "o", self.cfg["width"]) + vec(p + "o.b", self.cfg["width"])

    def _memory(self, h, p, m, eps):
        T, H, dk, dv, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q = self.lin(h, p + "q", H * dk).view(T, H, dk) * dk ** -0.5
        k = self.lin(h, p + "k", H * dk).view(T, H, dk)
        v = self.lin(h, p + "v", H * dv).view(T, H, dv)
        gate = lambda n: cap * torch.tanh((self.lin(h, p + n, H) + self.w(p + n + ".b", H, kind="vector")) / cap)
        come, keep = gate("i"), torch.nn.functional.logsigmoid(gate("f"))
        S = torch.zeros(H, dk, dv + 1, dtype=h.dtype, device=h.device)       # the normaliser as one more column
        v1 = torch.cat([v, torch.ones_like(v[..., :1])], dim=-1)
        top = torch.zeros(H, dtype=h.dtype, device=h.device)
        sums, tops = torch.empty(T, H, dv + 1, dtype=h.dtype, device=h.device), torch.empty(T, H, dtype=h.dtype, device=h.device)
        for t in range(T):
            kept = keep[t] + top
            top = torch.maximum(kept, come[t])
            S = torch.exp(kept - top)[:, None, None] * S + (torch.exp(come[t] - top)[:, None] * k[t])[:, :, None] * v1[t, :, None, :]
            sums[t] = (q[t, :, None, :] @ S)[:, 0]
            tops[t] = top
        o = sums[..., :dv] / (torch.maximum(sums[..., dv].abs(), torch.exp(-tops)) + 1e-6)[..., None]
        o = _rms(o, eps).reshape(T, H * dv) * self.w(p + "norm", H * dv, kind="norm")
        return self.lin(o * torch.sigmoid(self.lin(h, p + "g", H * dv)), p + "o", self.cfg["width"])

    def _state_space(self, h, p, m, eps):
        T, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * P
        vec = lambda n, size: self.w(p + n, size, kind="vector")
        z, xbc, dt = torch.split(self.lin(h, p + "in", 2 * inner + 2 * G * N + H), [inner, inner + 2 * G * N, H], dim=1)
        xbc = _silu(self._conv(xbc, p + "conv", vec("conv.b", inner + 2 * G * N)))
        x, B, C = torch.split(xbc, [inner, G * N, G * N], dim=1)
        x = x.reshape(T, H, P)
        B, C = (t.reshape(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        dt = torch.nn.functional.softplus(dt + vec("dt_bias", H))
        keep = torch.exp(-torch.exp(vec("A_log", H)) * dt)
        S = torch.zeros(H, N, P, dtype=h.dtype, device=h.device)
        y = torch.empty(T, H, P, dtype=h.dtype, device=h.device)
        for t in range(T):
            S = torch.baddbmm(keep[t, :, None, None] * S, (dt[t, :, None] * B[t])[:, :, None], x[t, :, None, :])
            y[t] = (C[t, :, None, :] @ S)[:, 0]
        y = (y + vec("D", H)[:, None] * x).reshape(T, inner) * _silu(z)
        parts = m["norm_groups"]
        y = _rms(y.reshape(T, parts, inner // parts), eps).reshape(T, inner) * self.w(p + "norm", inner, kind="norm")
        return self.lin(y, p + "o", self.cfg["width"])

    def __call__(self, ids, first):
        c = self.cfg
        W, eps = c["width"], c["norm"]["eps"]
        table = self.w("embed", c["vocab"], W)
        norm = lambda t, name: _rms(t, eps) * self.w(name, W, kind="norm")
        x = norm(table[torch.tensor(ids, device=DEVICE)], "embed.norm")
        for i, spec in enumerate(c["layers"]):
            p, m = "l%d." % i, spec["mixer"]
            h = norm(x, p + "norm1")
            if spec["type"] == "mamba2":
                y = self._state_space(h, p + "mix.", m, eps)
            else:
                y = m["left_scale"] * self._softmax(h, p + "mix.left.", m["left"]) \
                    + m["right_scale"] * self._memory(h, p + "mix.right.", m["right"], eps)
            ff = spec["mlp"]["ff"]
            x = x + y + self.lin(torch.relu(self.lin(norm(x, p + "norm2"), p + "mlp.up", ff)) ** 2, p + "mlp.down", W)
        return norm(x[first:], "final.norm") @ table.T
