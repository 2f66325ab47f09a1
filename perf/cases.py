"""The work this engine is timed on: what a program that holds a model does through ``Engine`` and its step function.

Two kinds of pass.  ``answer``: requests are opened, their prompts are read in steps of at most 2,048 tokens (the engine's
default budget), a number of decode steps follow, and the requests are closed; the logits of every prompt's last token and of
every decode step come back.  ``decode``: one decode step of requests whose prompts are cached already, each pass one token
further on (a request that reaches the context limit is replaced by a new one with the same prompt), the way a server runs
between arrivals.  Token ids are given (the replay program's way), so that all that comes back is computed numbers.

Models are the ones the benchmark names (the Llama-3.2-1B shape with all layers, fewer layers of the Llama-3.1-8B shape, and of
each other decoder the layers of ``bench.py --design`` at the 1B sizes), with random weights at the scale of trained ones:
gates and decays are drawn from the ranges such models start from.
"""
import json
import math
import os
import shutil
import tempfile
import zlib

import numpy as np
import torch

from hfee_b200 import Engine, StepEntry
from hfee_b200.config.registry import resolve
from hfee_b200.parts.model import model_tensor_needs
from hfee_b200.weights import write_file

BUDGET, CONTEXT, PAGE = 2048, 4096, 64          # the engine's defaults: tokens of a step, of a request, of a page
LIVE = {"llama-1b": 192}                        # request slots of the engine (64 requests of three programs' worth); others:
LIVE_OTHERS = 24
ROUTED = ("muvetar", "pupinex", "bumisun")
H, G, D, WIDTH, FF = 32, 8, 64, 2048, 8192      # the 1B layer sizes


# ------------------------------------------------------------------------------------------------ the models
def _llama(layers, shape):
    big = shape == "8b"
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": layers,
            "hidden_size": 4096 if big else WIDTH, "num_attention_heads": 32, "num_key_value_heads": 8,
            "head_dim": 128 if big else D, "intermediate_size": 14336 if big else FF, "vocab_size": 128256,
            "rope_theta": 500000.0, "rms_norm_eps": 1e-5, "max_position_embeddings": 131072, "tie_word_embeddings": not big,
            "rope_scaling": {"rope_type": "llama3", "factor": 8.0 if big else 32.0, "low_freq_factor": 1.0,
                             "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}}


def _layers(model, n):
    """The layers of a decoder other than Llama, its types in turn."""
    dense = {"kind": "dense", "ff": FF}
    attn = {"heads": H, "kv_heads": G, "dim": D, "vdim": D}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 2}, "expert": {"ff": FF // 4}, "shared": {"ff": FF // 2}}
    clamped = dict(moe, expert={"ff": FF // 4, "limit": 7.0}, shared={"ff": FF // 2, "limit": 7.0})
    rot = {"dims": D // 2, "base": 500000.0}
    window = dict(attn, scale=D ** -0.5, mask={"size": 1024})
    if model == "dobelix":
        decay = [1.0 - 2.0 ** (-1 - 7 * i / (H - 1)) for i in range(H)]
        scan = {"type": "lightning", "mlp": dense, "mixer": {"heads": H, "dim": D, "vdim": D, "decay": decay}}
        kinds = [scan, {"type": "attention", "mlp": dense, "mixer": dict(
            attn, mask={"size": 128}, rot={"dims": D, "base": 10000.0}, scale=D ** -0.5)}, scan]
    elif model == "bamipel":
        kinds = [{"type": "delta", "mlp": dense, "mixer": dict(attn, conv=4)},
                 {"type": "latent_attention", "mlp": dense, "mixer": {
                     "heads": H, "dim": D, "rot_dim": D // 2, "vdim": D, "q_rank": 768, "kv_rank": 4 * D, "mask": {"size": 512},
                     "rot": {"dims": D // 2, "base": 10000.0}, "scale": (D + D // 2) ** -0.5}},
                 {"type": "attention", "mlp": dense, "mixer": dict(attn, scale=1.0 / D, rot={
                     "dims": D, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})}]
    elif model == "muvetar":
        clamped = dict(clamped, router={"experts": 16, "top": 2, "scale": 1.0})
        kinds = [{"type": "parallel", "mlp": clamped, "mixer": {
                     "left": dict(attn, scale=D ** -0.5), "right": {"inner": WIDTH, "state": 16, "dt_rank": WIDTH // 16, "conv": 4},
                     "left_scale": 1.0, "right_scale": 1.0}},
                 {"type": "mingru", "mlp": clamped, "mixer": {"width": WIDTH}}]
    elif model == "pupinex":
        moe = dict(moe, router={"experts": 16, "top": 2, "scale": 2.5, "groups": {"count": 2, "keep": 1}})
        kinds = [{"type": "parallel", "mlp": dict(dense, limit=7.0), "mixer": {
                     "left": dict(window, rot=dict(rot, scaling={"factor": 4.0})),
                     "right": {"heads": G, "dim": D, "vdim": WIDTH // G, "gate_cap": 15.0}, "left_scale": 1.0, "right_scale": 1.0}},
                 {"type": "attention", "mlp": moe, "mixer": dict(window, rot=rot)},
                 {"type": "gla", "mlp": dict(dense, limit=7.0),
                  "mixer": {"heads": G, "dim": 2 * D, "vdim": WIDTH // G, "tau": 16.0, "rank": 16}},
                 {"type": "attention", "mlp": moe, "mixer": dict(window, rot=rot)}]
    elif model == "fokalorn":
        kinds = [{"type": "channel_delta", "mlp": dense, "mixer": dict(attn, conv=4, rank=D, gate_rank=D)},
                 {"type": "latent_attention", "mlp": dense, "mixer": {
                     "heads": H, "dim": D, "rot_dim": D // 2, "vdim": D, "kv_rank": 4 * D,
                     "rot": {"dims": D // 2, "base": 10000.0}, "scale": (D + D // 2) ** -0.5}}]
    else:
        kinds = [{"type": "attention", "mlp": dense, "mixer": dict(
                     window, softcap=30.0, v_mix=True, mask={"size": 1024, "keep_first": 4}, rot=rot)},
                 {"type": "mamba2", "mlp": clamped, "mixer": {
                     "heads": 64, "vdim": 64, "state": 128, "groups": G, "conv": 4, "norm_groups": G}}]
    return [kinds[i % len(kinds)] for i in range(n)]


def _config(case):
    model, n = case["model"], case["layers"]
    if model.startswith("llama"):
        return _llama(n, model[-2:])
    cfg = {"architecture": model.capitalize(), "vocab": 32768, "width": WIDTH, "layers": _layers(model, n), "norm": {"eps": 1e-5}}
    cfg.update({"dobelix": {"canon": {"taps": 4}, "embedding": {"scale": 1.0}, "logit_scale": 1.0}, "bamipel": {},
                "muvetar": {"residual_mult": 1.0, "logit_softcap": 30.0},
                "pupinex": {"embedding": {"bigram": {"buckets": 65521, "mul_prev": 1000003, "mul_cur": 31}}},
                "fokalorn": {"streams": 4, "norm": {"eps": 1e-5, "groups": 2}, "embedding": {"scale": 1.0}},
                "bumisun": {"residual_mult": 0.5, "logit_scale": 1.0}}[model])
    return cfg


def _kinds(width):
    u = torch.randn(16, width, generator=torch.Generator(device="cuda").manual_seed(16), device="cuda", dtype=torch.float32)
    return u / u.norm(dim=1, keepdim=True)


def _tensor(name, shape, role, kinds=False):
    """A model tensor, from its name alone: matrices N(0, 0.02) in bfloat16, vectors in float32.  What decides how long a state
    remembers is drawn from the ranges such models start from (step sizes of 0.001 to 0.1, rates of 1 to 16, forget gates near
    one); residual streams start as copies that each sublayer reads evenly and adds to.  Where there are routers (``kinds``), tokens
    come in 16 kinds that an embedding shows and a router knows, two experts of one group for each, so that a choice is rarely a
    near tie, as after training."""
    g = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()))
    draw = lambda: torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * 0.02
    rand = lambda: torch.rand(shape, generator=g, device="cuda", dtype=torch.float32)
    last = name.rsplit(".", 1)[-1]
    if kinds and name == "embed":
        return (draw() + 16.0 * _kinds(shape[1])[torch.arange(shape[0], device="cuda") % 16]).to(torch.bfloat16)
    if last == "router":
        u = _kinds(shape[1])
        e = torch.arange(16, device="cuda")
        return (0.25 * (draw() + u + 0.8 * u[e // 8 * 8 + (e + 3) % 8])).to(torch.bfloat16)
    if role in ("matrix", "table"):
        return draw().to(torch.bfloat16)
    if last == "dt_bias" or name.endswith("dt.b"):
        dt = torch.exp(rand() * math.log(100.0) + math.log(0.001))
        return dt + torch.log(-torch.expm1(-dt))                       # softplus of this is dt
    if last == "A_log":
        rate = 1.0 + 15.0 * rand() if len(shape) == 1 else torch.arange(1.0, shape[1] + 1, device="cuda").expand(shape) * (1 + draw())
        return torch.log(rate).contiguous()
    if name.endswith(".f.b"):
        return 3.0 + 3.0 * rand()
    if last == "shift":
        return rand()
    if name.endswith("hc1.in") or name.endswith("hc2.in"):
        return 1.0 / shape[0] + draw()
    if name.endswith("hc1.mix") or name.endswith("hc2.mix"):
        return torch.eye(shape[0], device="cuda") + draw()
    if last == "vmix":
        return 0.5 + draw()
    if last == "dwa":
        return draw() + torch.nn.functional.one_hot(torch.tensor(shape[0] - 1), shape[0]).to("cuda")
    if role == "scale" or last == "D" or name.endswith("hc1.out") or name.endswith("hc2.out"):
        return 1.0 + draw()
    return draw().abs() if role == "positive" else draw()


_HELD = {}          # the engine of the model in use: a program loads its model once


def _needs(cfg):
    arch, c = resolve(cfg)
    return {n: need for n, need in model_tensor_needs(arch.build_spec(c)).items() if not need.optional}


def _engine(case):
    key = (case["model"], case["layers"], case["dtype"])
    if key not in _HELD:
        _HELD.clear()
        torch.cuda.empty_cache()
        cfg = _config(case)
        folder = tempfile.mkdtemp(prefix="perf_model_")
        try:
            with open(os.path.join(folder, "config.json"), "w") as f:
                json.dump(dict(cfg, torch_dtype="bfloat16"), f)
            write_file(os.path.join(folder, "model.safetensors"),
                       {n: _tensor(n, need.shape, need.role, case["model"] in ROUTED).cpu() for n, need in _needs(cfg).items()})
            live = LIVE.get(case["model"], LIVE_OTHERS)
            _HELD[key] = Engine(folder, dtype=case["dtype"], page_size=PAGE, max_requests=live, max_context=CONTEXT,
                                max_batch_tokens=BUDGET, max_cache_tokens=live * CONTEXT)
        finally:
            shutil.rmtree(folder, ignore_errors=True)
    return _HELD[key]


# ------------------------------------------------------------------------------------------------ the cases
def _case(name, model, layers, kind, requests, prompt, steps, dtype="bfloat16"):
    c = {"model": model, "layers": layers, "kind": kind, "requests": requests, "prompt": prompt, "steps": steps, "dtype": dtype}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one conversation that runs on: the smallest call, a step of one token (the headline model with all its layers)
        _case("decode_1", "llama-1b", 16, "decode", 1, 1024, 1),
        # the headline benchmark: a decode step of eight requests behind prompts of about 2,048 tokens
        _case("decode_8", "llama-1b", 16, "decode", 8, 2048, 1),
        # a full server: 64 requests of mixed lengths
        _case("decode_64", "llama-1b", 16, "decode", 64, 1500, 1),
        # a prompt of 2,048 tokens, the other half of the headline benchmark
        _case("prompt_2048", "llama-1b", 16, "answer", 1, 2048, 0),
        # a short question and the first words of its answer
        _case("question", "llama-1b", 16, "answer", 1, 77, 12),
        # three long documents on the larger shape, read in full steps: the largest work
        _case("documents_8b", "llama-8b", 8, "answer", 3, 2900, 0),
        # the 32-bit path, which a user takes to check a model's numbers
        _case("check_float32", "llama-1b", 4, "answer", 2, 150, 6, "float32"),
        # the other decoders: prompts, then some decode steps of the answers
        _case("dobelix", "dobelix", 3, "answer", 4, 600, 8),
        _case("bamipel", "bamipel", 3, "answer", 1, 1999, 8),
        _case("pupinex", "pupinex", 4, "answer", 2, 1100, 8),
        _case("fokalorn", "fokalorn", 4, "answer", 1, 2048, 8),
        _case("bumisun", "bumisun", 4, "answer", 3, 683, 8),
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["llama-1b", "llama-1b", "llama-8b", "dobelix", "bamipel", "muvetar", "pupinex", "fokalorn", "bumisun"])
    layers = {"llama-1b": rng.choice([4, 16]), "llama-8b": 4, "bamipel": 3, "dobelix": 3, "muvetar": 2}.get(model, rng.choice([2, 4]))
    dtype = "float32" if rng.random() < 0.08 else "bfloat16"
    if dtype == "float32":
        return _case(None, model, min(layers, 4), "answer", spread(1, 4), spread(8, 250), rng.randrange(5), dtype)
    if rng.random() < 0.4:
        return _case(None, model, layers, "decode", spread(1, 64 if model == "llama-1b" else 8), spread(16, 2500), 1)
    requests = spread(1, 16)
    return _case(None, model, layers, "answer", requests, spread(8, max(16, 5000 // requests) if requests > 1 else 4000), rng.randrange(13))


def _lengths(case):
    """The prompts' lengths: the longest is ``prompt``, the others down to half of it (whole numbers of no pattern)."""
    p = case["prompt"]
    return [max(1, p - (i * 7919) % (p // 2 + 1)) for i in range(case["requests"])]


class _State:
    """What the program has in hand: the engine, the prompts and the tokens that follow them; for ``decode`` the open requests."""

    def __init__(self, case, seed):
        self.engine = _engine(case)
        self.runner, self.case = self.engine.runner, case
        rng = np.random.default_rng(seed)
        vocab = self.runner.vocab
        self.prompts = [rng.integers(0, vocab, size=n).tolist() for n in _lengths(case)]
        self.room = CONTEXT - case["prompt"] if case["kind"] == "decode" else case["steps"]
        self.feed = rng.integers(0, vocab, size=(self.room, case["requests"])).tolist()
        self.slots, self.at = [], 0
        if case["kind"] == "decode":
            self.begin()

    def begin(self):
        """Open the requests and read their prompts in full steps; the logits of the prompts' last tokens."""
        self.close()
        runner = self.runner
        self.slots = [runner.open() for _ in self.prompts]
        self.at = 0
        rows, entries, free = [], [], BUDGET
        for slot, prompt in zip(self.slots, self.prompts):
            done = 0
            while done < len(prompt):
                k = min(free, len(prompt) - done)
                entries.append(StepEntry(slot, prompt[done:done + k], (k - 1,) if done + k == len(prompt) else ()))
                done, free = done + k, free - k
                if free == 0:
                    rows.append(self.keep(runner.step(entries)))
                    entries, free = [], BUDGET
        if entries:
            rows.append(self.keep(runner.step(entries)))
        return torch.cat([r for r in rows if r is not None])

    def keep(self, logits):
        return None if logits is None else logits.clone()             # the runner's buffer is the next step's

    def decode(self):
        feed = self.feed[self.at]
        self.at += 1
        return self.runner.step([StepEntry(s, (feed[j],), (0,)) for j, s in enumerate(self.slots)])

    def close(self):
        for s in self.slots:
            self.runner.close(s)
        self.slots = []

    def __del__(self):
        self.close()


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    if state.case["kind"] == "decode":
        if state.at == state.room:
            state.begin()
        return state.decode()
    out = [state.begin()]
    for _ in range(state.case["steps"]):
        out.append(state.keep(state.decode()))
    state.close()
    return out


def tolerance(case):
    # Measured against 64 bits: 0.006 to 0.022 in bfloat16 (the most for the Llama shapes' sixteen layers and wide matrices), 5e-6 in
    # float32.  Two correct bfloat16 implementations differ by about as much as either is off, so no more than this is stated.
    return {"rel": 2e-5, "max": 2e-3} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.5}


def work(case):
    """Per step: the matrices its tokens pass (of the experts those that are chosen), the embedding rows, the keys and values or
    states it reads and writes, the logits; products, and attention over the positions that are seen."""
    cfg, elem = _config(case), 4 if case["dtype"] == "float32" else 2
    llama = case["model"].startswith("llama")
    vocab, width = (cfg["vocab_size"], cfg["hidden_size"]) if llama else (cfg["vocab"], WIDTH)
    dense = experts = layers_with = 0
    for name, need in _needs(cfg).items():
        size = math.prod(need.shape)
        if ".mlp.e" in name:
            experts += size
            layers_with += name.endswith(".e0.down")
        elif need.role == "matrix" and name not in ("head", "lm_head.weight"):
            dense += size
    if llama:
        hd = cfg["head_dim"]
        mixers = [("attention", {"heads": 32, "kv_heads": 8, "dim": hd, "vdim": hd})] * case["layers"]
    else:
        mixers = []
        for layer in cfg["layers"]:
            m = layer["mixer"]
            mixers += [("attention", m["left"]), ("scan", m["right"])] if layer["type"] == "parallel" else [(layer["type"], m)]
    steps = []                                   # (tokens, [(context before, new tokens)], wanted rows)
    lengths = _lengths(case)
    if case["kind"] == "answer":
        now, free = [], BUDGET
        for n in lengths:
            done = 0
            while done < n:
                k = min(free, n - done)
                now.append((done, k, done + k == n))
                done, free = done + k, free - k
                if free == 0:
                    steps.append(now)
                    now, free = [], BUDGET
        if now:
            steps.append(now)
    for t in range(case["steps"]):
        steps.append([(n + t, 1, True) for n in lengths])
    total_bytes = flops = 0.0
    for now in steps:
        n, rows = sum(k for _, k, _ in now), sum(w for _, _, w in now)
        touched = experts * (1 - (1 - 2 / 16) ** n)
        total_bytes += elem * (dense + touched + n * width + (vocab * width if rows else 0)) + 4 * rows * vocab
        flops += 2.0 * n * (dense + experts * 2 / 16) + 2.0 * rows * vocab * width
        for kind, m in mixers:
            for before, k, _ in now:
                if "attention" in kind:
                    lat = kind == "latent_attention"
                    per = m["kv_rank"] + m["rot_dim"] if lat else m["kv_heads"] * (m["dim"] + m["vdim"])
                    mask = m.get("mask") or {}
                    window = mask.get("size", 1 << 30)
                    seen = sum(min(i + 1, window) for i in range(before, before + k))
                    total_bytes += elem * per * (min(before, window) + k)
                    flops += 2.0 * seen * m["heads"] * (m["dim"] + m["vdim"] + (m["rot_dim"] if lat else 0))
                else:
                    size = (m["inner"] * m["state"] if "inner" in m else m["width"] if "width" in m else
                            m["heads"] * m.get("dim", m.get("state", 0)) * m["vdim"])
                    total_bytes += 8.0 * size
                    flops += 4.0 * k * size
    return {"bytes": total_bytes, "flops": flops}


# ------------------------------------------------------------------------------------------------ in 64 bits
class _Plain:
    """The decoders in float64: whole sequences, all requests' tokens in one matrix, what runs along a sequence per request."""

    def __init__(self, cfg, spans):
        self.cfg, self.spans = cfg, spans

    def w(self, name, *shape, role="vector"):
        return _tensor(name, shape, role).double()

    def lin(self, x, name, rows, bias=False):
        y = x @ self.w(name, rows, x.shape[1], role="matrix").T
        return y + self.w(name + ".b", rows) if bias else y

    def each(self, fn, *xs):
        return torch.cat([fn(*(x[a:b] for x in xs)) for a, b in self.spans])

    def rms(self, x, name, eps, groups=1):
        y = x.reshape(x.shape[0], groups, -1)
        y = (y * torch.rsqrt((y * y).mean(-1, keepdim=True) + eps)).reshape(x.shape)
        return y if name is None else y * self.w(name, x.shape[1], role="scale")

    def conv(self, x, name, bias=False):
        w = self.w(name, x.shape[1], 4)
        y = self.each(lambda s: sum(torch.nn.functional.pad(s, (0, 0, 3 - j, 0))[:len(s)] * w[:, j] for j in range(4)), x)
        return y + self.w(name + ".b", x.shape[1]) if bias else y

    @staticmethod
    def freqs(dims, base, scaling):
        f = base ** (-torch.arange(0, dims, 2, device="cuda", dtype=torch.float64) / dims)
        if not scaling:
            return f
        if "low" not in scaling and "low_freq_factor" not in scaling:
            return f / scaling["factor"]
        low, high = scaling.get("low", scaling.get("low_freq_factor")), scaling.get("high", scaling.get("high_freq_factor"))
        orig = scaling.get("original", scaling.get("original_max_position_embeddings"))
        turns = orig * f / (2 * math.pi)                                # wavelengths in the original context
        s = ((turns - low) / (high - low)).clamp(0, 1)
        return (1 - s) * f / scaling["factor"] + s * f

    def rotate(self, x, dims, base, scaling=None, pairs=False):
        """x [T, heads, d]; dimension i turns with i + dims/2, or 2i with 2i + 1 (pairs)."""
        a = torch.cat([torch.arange(b - a, device="cuda", dtype=torch.float64) for a, b in self.spans])
        a = a[:, None] * self.freqs(dims, base, scaling)[None]
        c, s = a.cos()[:, None], a.sin()[:, None]
        at = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
        u, v = x[..., at[0]], x[..., at[1]]
        out = x.clone()
        out[..., at[0]], out[..., at[1]] = u * c - v * s, v * c + u * s
        return out

    def softmax_attention(self, q, k, v, scale, window=None, first=0, sink=None, cap=None, far=None):
        heads, groups = q.shape[1], k.shape[1]

        def one(q, k, v):
            n = len(q)
            back = torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None]
            hidden = back < 0
            if window is not None:
                hidden |= (back >= window) & (torch.arange(n, device="cuda")[None] >= first)
            out = torch.empty(n, heads, v.shape[2], device="cuda", dtype=torch.float64)
            for g in range(groups):
                for h in range(g * heads // groups, (g + 1) * heads // groups):
                    s = (q[:, h] @ k[:, g].T) * scale
                    s = cap * torch.tanh(s / cap) if cap else s
                    if far is not None:
                        s = s - far[0][h] * torch.log1p(far[1][h] * back.clamp(min=0))
                    s = s.masked_fill(hidden, -math.inf)
                    top = s.amax(1, keepdim=True) if sink is None else s.amax(1, keepdim=True).clamp(min=float(sink[h]))
                    e = torch.exp(s - top)
                    out[:, h] = (e @ v[:, g]) / (e.sum(1, keepdim=True) + (0 if sink is None else torch.exp(sink[h] - top)))
            return out
        return self.each(one, q, k, v)

    def heads(self, x, name, heads, dim, bias=False):
        return self.lin(x, name, heads * dim, bias).reshape(len(x), heads, dim)

    def qkv(self, x, p, m, bias=False):
        return (self.heads(x, p + "q", m["heads"], m["dim"], bias), self.heads(x, p + "k", m["kv_heads"], m["dim"], bias),
                self.heads(x, p + "v", m["kv_heads"], m["vdim"], bias))

    # -------------------------------------------------------------------------------------- mixers
    def lightning(self, x, p, m, eps):
        q, k, v = (torch.nn.functional.silu(self.heads(x, p + n, m["heads"], m["dim"])) for n in "qkv")
        decay = torch.tensor(m["decay"], device="cuda", dtype=torch.float64)[:, None, None]

        def one(q, k, v):
            s, out = 0, torch.empty_like(v)
            for t in range(len(q)):
                s = decay * s + k[t][:, :, None] * v[t][:, None, :]
                out[t] = (q[t][:, None, :] @ s)[:, 0]
            return out
        o = self.rms(self.each(one, q, k, v).flatten(1), p + "norm", eps)
        return self.lin(o * torch.sigmoid(self.lin(x, p + "g", WIDTH)), p + "o", WIDTH)

    def sigmoid_attention(self, x, p, m, eps):
        k = self.lin(x, p + "k", G * D)
        v = k.reshape(-1, G, D)
        q = self.rotate(self.rms(self.lin(x, p + "q", H * D), p + "q.norm", eps).reshape(-1, H, D), D, m["rot"]["base"])
        k = self.rotate(self.rms(k, p + "k.norm", eps).reshape(-1, G, D), D, m["rot"]["base"])
        temp, pb, size = self.w(p + "temp", H, role="scale"), self.w(p + "pb", H), m["mask"]["size"]

        def one(q, k, v):
            at = torch.arange(len(q), device="cuda")
            seen = (at[None] <= at[:, None]) & (at[None] // size == at[:, None] // size)
            s = torch.einsum("ihd,jhd->hij", q, k.repeat_interleave(H // G, 1)) * m["scale"] * temp[:, None, None] + pb[:, None, None]
            return torch.einsum("hij,jhd->ihd", torch.sigmoid(s) * seen, v.repeat_interleave(H // G, 1))
        o = self.each(one, q, k, v).flatten(1)
        return self.lin(o * torch.sigmoid(self.lin(x, p + "g", WIDTH)), p + "o", WIDTH)

    def delta(self, q, k, v, beta, g):
        """S <- g S + k (beta (v - (g S)^T k))^T;  o = S^T q.  g: a factor per head [T, H, 1] or per key channel [T, H, d]."""
        def one(q, k, v, beta, g):
            s = torch.zeros(H, q.shape[2], v.shape[2], device="cuda", dtype=torch.float64)
            out = torch.empty_like(v)
            for t in range(len(q)):
                s = s * g[t][:, :, None]
                s = torch.baddbmm(s, k[t][:, :, None], (beta[t][:, None] * (v[t] - (k[t][:, None] @ s)[:, 0]))[:, None])
                out[t] = (q[t][:, None] @ s)[:, 0]
            return out
        unit = lambda x: (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
        return self.each(one, unit(q) * D ** -0.5, unit(k), v, beta, g)

    def delta_inputs(self, x, p):
        act = lambda n, r: torch.nn.functional.silu(self.conv(self.lin(x, p + n, r), p + n + ".conv"))
        return (act("q", G * D).reshape(-1, G, D), act("k", G * D).reshape(-1, G, D), act("v", H * D).reshape(-1, H, D),
                torch.sigmoid(self.lin(x, p + "b", H)))

    def delta_mixer(self, x, p, m, eps):
        q, k, v, beta = self.delta_inputs(x, p)
        soft = torch.nn.functional.softplus(self.lin(x, p + "a", H) + self.w(p + "dt_bias", H))
        o = self.delta(q, k, v, beta, torch.exp(-torch.exp(self.w(p + "A_log", H)) * soft)[:, :, None])
        o = self.rms(o.reshape(-1, D), p + "norm", eps).reshape(len(x), -1) * torch.nn.functional.silu(self.lin(x, p + "g", H * D))
        return self.lin(o, p + "o", WIDTH)

    def channel_delta(self, x, p, m, eps):
        q, k, v, beta = self.delta_inputs(x, p)
        z = self.lin(self.lin(x, p + "a1", D), p + "a2", H * D) + self.w(p + "dt_bias", H * D)
        z = torch.nn.functional.softplus(z).reshape(-1, H, D)
        o = self.delta(q, k, v, beta, torch.exp(-torch.exp(self.w(p + "A_log", H))[:, None] * z))
        gate = torch.sigmoid(self.lin(self.lin(x, p + "g1", D), p + "g2", H * D))
        return self.lin(self.rms(o.reshape(-1, D), p + "norm", eps).reshape(len(x), -1) * gate, p + "o", WIDTH)

    def latent_attention(self, x, p, m, eps, pairs):
        r, rank, rot = m["rot_dim"], m["kv_rank"], m["rot"]
        low = x
        name = p + "q"
        if "q_rank" in m:
            low, name = self.rms(self.lin(x, p + "dq", m["q_rank"]), p + "dq.norm", eps), p + "uq"
        q = self.heads(low, name, H, D + r)
        down = self.lin(x, p + "dkv", rank + r)
        c = self.rms(down[:, :rank], p + "dkv.norm", eps)
        shared = self.rotate(down[:, None, rank:], rot["dims"], rot["base"], pairs=pairs).expand(-1, H, -1)
        q = torch.cat([q[..., :D], self.rotate(q[..., D:], rot["dims"], rot["base"], pairs=pairs)], -1)
        k = torch.cat([self.heads(c, p + "uk", H, D), shared], -1)
        o = self.softmax_attention(q, k, self.heads(c, p + "uv", H, D), m["scale"], (m.get("mask") or {}).get("size"),
                                   sink=self.w(p + "sink", H) if pairs else None)
        return self.lin((o * torch.sigmoid(self.lin(x, p + "g", H))[:, :, None]).flatten(1), p + "o", WIDTH)

    def unit_attention(self, x, p, m, eps):
        q, k, v = self.qkv(x, p, m)
        rot = m["rot"]
        q, k = (self.rms(self.rotate(y, rot["dims"], rot["base"], rot["scaling"]).reshape(-1, D), None, eps).reshape(y.shape)
                for y in (q, k))
        o = self.softmax_attention(q, k, v, m["scale"]) * torch.sigmoid(self.lin(x, p + "g", H))[:, :, None]
        return self.lin(o.flatten(1), p + "o", WIDTH)

    def mingru(self, x, p, m, eps):
        z, u = torch.sigmoid(self.lin(x, p + "z", WIDTH, True)), self.lin(x, p + "x", WIDTH, True)
        u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))

        def one(z, u):
            s, out = 0, torch.empty_like(z)
            for t in range(len(z)):
                s = (1 - z[t]) * s + z[t] * u[t]
                out[t] = s
            return out
        return self.lin(self.each(one, z, u) * torch.nn.functional.silu(self.lin(x, p + "g", WIDTH)), p + "o", WIDTH)

    def far_attention(self, x, p, m):
        q, k, v = self.qkv(x, p, m)
        far = [self.w(p + r, H, role="positive") for r in ("r1", "r2")]
        return self.lin(self.softmax_attention(q, k, v, m["scale"], far=far).flatten(1), p + "o", WIDTH)

    def selective_scan(self, x, p, m):
        inner, n, rank = m["inner"], m["state"], m["dt_rank"]
        u, z = self.lin(x, p + "in", 2 * inner).split(inner, 1)
        u = torch.nn.functional.silu(self.conv(u, p + "conv", True))
        dt, B, C = self.lin(u, p + "x", rank + 2 * n).split([rank, n, n], 1)
        dt = torch.nn.functional.softplus(self.lin(dt, p + "dt", inner, True))
        rate = -torch.exp(self.w(p + "A_log", inner, n))

        def one(u, dt, B, C):
            s, out = 0, torch.empty_like(u)
            for t in range(len(u)):
                s = torch.exp(dt[t][:, None] * rate) * s + (dt[t] * u[t])[:, None] * B[t]
                out[t] = s @ C[t]
            return out
        y = self.each(one, u, dt, B, C) + self.w(p + "D", inner) * u
        return self.lin(y * torch.nn.functional.silu(z), p + "o", WIDTH)

    def sink_attention(self, x, p, m, eps):
        q, k, v = self.qkv(x, p, m, True)
        q, k = (self.rotate(y, m["rot"]["dims"], m["rot"]["base"], pairs=True) for y in (q, k))
        o = self.softmax_attention(q, k, v, m["scale"], m["mask"]["size"], sink=self.w(p + "sink", H))
        return self.lin(o.flatten(1), p + "o", WIDTH, True)

    def normed_attention(self, x, p, m, eps):
        q, k, v = self.qkv(x, p, m, True)
        rot = m["rot"]
        q, k = (self.rotate(self.rms(y.flatten(1), p + n + ".norm", eps).reshape(y.shape), rot["dims"], rot["base"], rot["scaling"])
                for y, n in ((q, "q"), (k, "k")))
        return self.lin(self.softmax_attention(q, k, v, m["scale"], m["mask"]["size"]).flatten(1), p + "o", WIDTH)

    def gla(self, x, p, m, eps):
        h, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = self.heads(x, p + "q", h, d) * d ** -0.5, self.heads(x, p + "k", h, d), self.heads(x, p + "v", h, dv)
        z = self.lin(self.lin(x, p + "a1", m["rank"]), p + "a2", h * d, True)
        alpha = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(-1, h, d)

        def one(q, k, v, alpha):
            s, out = 0, torch.empty_like(v)
            for t in range(len(q)):
                s = alpha[t][:, :, None] * s + k[t][:, :, None] * v[t][:, None]
                out[t] = (q[t][:, None] @ s)[:, 0]
            return out
        o = self.rms(self.each(one, q, k, v, alpha).reshape(-1, dv), p + "norm", eps).reshape(len(x), -1)
        return self.lin(o * torch.nn.functional.silu(self.lin(x, p + "g", h * dv)), p + "o", WIDTH)

    def matrix_memory(self, x, p, m, eps):
        h, d, dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = self.heads(x, p + "q", h, d) * d ** -0.5, self.heads(x, p + "k", h, d), self.heads(x, p + "v", h, dv)
        i, f = (cap * torch.tanh(self.lin(x, p + n, h, True) / cap) for n in "if")

        def one(q, k, v, i, f):
            s = n = 0
            top = torch.zeros(h, device="cuda", dtype=torch.float64)
            out = torch.empty_like(v)
            for t in range(len(q)):
                new = torch.maximum(f[t] + top, i[t])
                a, b = torch.exp(f[t] + top - new), torch.exp(i[t] - new)
                s = a[:, None, None] * s + (b[:, None] * k[t])[:, :, None] * v[t][:, None]
                n, top = a[:, None] * n + b[:, None] * k[t], new
                den = torch.maximum((n * q[t]).sum(1).abs(), torch.exp(-top)) + 1e-6
                out[t] = (q[t][:, None] @ s)[:, 0] / den[:, None]
            return out
        o = self.each(one, q, k, v, i, torch.nn.functional.logsigmoid(f))
        o = self.rms(o.reshape(-1, dv), None, eps).reshape(len(x), -1) * self.w(p + "norm", h * dv, role="scale")
        return self.lin(o * torch.sigmoid(self.lin(x, p + "g", h * dv)), p + "o", WIDTH)

    def kept_attention(self, x, p, m, memo):
        q, k, v = self.qkv(x, p, m)
        q, k = (self.rotate(y, m["rot"]["dims"], m["rot"]["base"]) for y in (q, k))
        if "first" in memo:
            share = self.w(p + "vmix")
            v = (1 - share) * v + share * memo["first"]
        else:
            memo["first"] = v
        o = self.softmax_attention(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], self.w(p + "sink", H), m["softcap"])
        return self.lin(o.flatten(1), p + "o", WIDTH)

    def mamba2(self, x, p, m, eps):
        h, dv, n, g = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = h * dv
        z, u, dt = self.lin(x, p + "in", 2 * inner + 2 * g * n + h).split([inner, inner + 2 * g * n, h], 1)
        u, B, C = torch.nn.functional.silu(self.conv(u, p + "conv", True)).split([inner, g * n, g * n], 1)
        u = u.reshape(-1, h, dv)
        B, C = (y.reshape(-1, g, n).repeat_interleave(h // g, 1) for y in (B, C))
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias", h))
        decay = torch.exp(-torch.exp(self.w(p + "A_log", h)) * dt)

        def one(u, B, C, dt, decay):
            s, out = 0, torch.empty_like(u)
            for t in range(len(u)):
                s = decay[t][:, None, None] * s + (dt[t][:, None] * B[t])[:, :, None] * u[t][:, None]
                out[t] = (C[t][:, None] @ s)[:, 0]
            return out
        y = self.each(one, u, B, C, dt, decay) + self.w(p + "D", h)[:, None] * u
        y = self.rms(y.flatten(1) * torch.nn.functional.silu(z), None, eps, m["norm_groups"]) * self.w(p + "norm", inner, role="scale")
        return self.lin(y, p + "o", WIDTH)

    # -------------------------------------------------------------------------------------- feed-forwards
    def gated(self, x, p, ff, act):
        return self.lin(act(self.lin(x, p + "gate", ff), self.lin(x, p + "up", ff)), p + "down", x.shape[1])

    @staticmethod
    def clamped(g, u):
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        return g * torch.sigmoid(1.702 * g) * (u + 1)

    def experts(self, x, p, model):
        silu = lambda g, u: torch.nn.functional.silu(g) * u
        act = silu if model == "pupinex" else self.clamped
        z = self.lin(x, p + "router", 16) + (self.w(p + "router.b", 16) if model == "bumisun" else 0)
        if model == "pupinex":
            s = torch.sigmoid(z)
            best = s.reshape(-1, 2, 8).topk(2, -1).values.sum(-1).argmax(1)
            s = s.masked_fill(torch.arange(16, device="cuda")[None] // 8 != best[:, None], -1.0)
            weight, chosen = s.topk(2, 1)
            weight = weight / (weight.sum(1, keepdim=True) + 1e-20) * 2.5
        else:
            weight, chosen = (torch.softmax(z, 1) if model == "muvetar" else z).topk(2, 1)
            weight = weight if model == "muvetar" else torch.softmax(weight, 1)
        out = self.gated(x, p + "shared.", FF // 2, act)
        if model != "muvetar":
            out = out * torch.sigmoid(self.lin(x, p + "shared.sg", 1))
        for e in range(16):
            t, slot = torch.nonzero(chosen == e, as_tuple=True)
            if len(t):
                out.index_add_(0, t, weight[t, slot][:, None] * self.gated(x[t], f"{p}e{e}.", FF // 4, act))
        return out

    def squared(self, x, p):
        return self.lin(torch.relu(self.lin(x, p + "up", FF)) ** 2, p + "down", WIDTH)

    # -------------------------------------------------------------------------------------- whole models
    def layer_norm(self, x, name, eps):
        x = x - x.mean(1, keepdim=True)
        return self.rms(x, name, eps)

    def llama(self, tokens, rows):
        c = self.cfg
        width, eps = c["hidden_size"], c["rms_norm_eps"]
        table = self.w("model.embed_tokens.weight", c["vocab_size"], width, role="table")
        x = table[tokens]
        m = {"heads": 32, "kv_heads": 8, "dim": c["head_dim"], "vdim": c["head_dim"]}
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            y = self.rms(x, p + "input_layernorm.weight", eps)
            q, k, v = (self.heads(y, f"{p}self_attn.{n}_proj.weight", h, c["head_dim"]) for n, h in (("q", 32), ("k", 8), ("v", 8)))
            q, k = (self.rotate(t, c["head_dim"], c["rope_theta"], c["rope_scaling"]) for t in (q, k))
            o = self.softmax_attention(q, k, v, m["dim"] ** -0.5).flatten(1)
            x = x + self.lin(o, p + "self_attn.o_proj.weight", width)
            y = self.rms(x, p + "post_attention_layernorm.weight", eps)
            parts = []
            for part in y.split(16384):
                u = torch.nn.functional.silu(self.lin(part, p + "mlp.gate_proj.weight", c["intermediate_size"]))
                u *= self.lin(part, p + "mlp.up_proj.weight", c["intermediate_size"])
                parts.append(self.lin(u, p + "mlp.down_proj.weight", width))
            x = x + torch.cat(parts)
        y = self.rms(x[rows], "model.norm.weight", eps)
        return y @ table.T if c["tie_word_embeddings"] else self.lin(y, "lm_head.weight", c["vocab_size"])

    def other(self, model, tokens, rows):
        c, eps = self.cfg, self.cfg["norm"]["eps"]
        table = _tensor("embed", (c["vocab"], WIDTH), "table", model in ROUTED).double()
        x = table[tokens]
        at = torch.cat([torch.arange(b - a, device="cuda", dtype=torch.float64) for a, b in self.spans])
        if model == "muvetar":
            angle = at[:, None] * 10000.0 ** (-torch.arange(0, WIDTH, 2, device="cuda", dtype=torch.float64) / WIDTH)
            x = x + torch.stack([angle.sin(), angle.cos()], -1).flatten(1)
        if model == "pupinex":
            rows_of = torch.cat([torch.tensor([0]).to(tokens), tokens[:-1]]) * 1000003 + tokens * 31
            x = x + self.w("bigram", 65522, WIDTH, role="table")[torch.where(at == 0, 65521, rows_of % 65521)]
        if model == "bumisun":
            x = self.rms(x, "embed.norm", eps)
        history, memo, streams = [x], {}, [x] * 4
        for i, layer in enumerate(c["layers"]):
            p, m, kind = f"l{i}.", layer["mixer"], layer["type"]
            if model == "dobelix":
                h = x + self.conv(x, p + "canon1")
                y = (self.lightning if kind == "lightning" else self.sigmoid_attention)(h, p + "mix.", m, eps)
                x = x + self.rms(y, p + "norm1", eps)
                gelu = lambda g, u: torch.nn.functional.gelu(g, approximate="tanh") * u
                x = x + self.rms(self.gated(x, p + "mlp.", FF, gelu), p + "norm2", eps)
            elif model == "bamipel":
                h = self.rms(x, p + "norm1", eps)
                y = (self.delta_mixer(h, p + "mix.", m, eps) if kind == "delta" else self.unit_attention(h, p + "mix.", m, eps)
                     if kind == "attention" else self.latent_attention(h, p + "mix.", m, eps, False))
                x = x + self.rms(y, p + "norm1b", eps)
                x = x + self.rms(self.squared(self.rms(x, p + "norm2", eps), p + "mlp."), p + "norm2b", eps)
            elif model == "muvetar":
                h = self.rms(x, p + "norm1", eps)
                x = x + (self.mingru(h, p + "mix.", m, eps) if kind == "mingru" else
                         self.far_attention(h, p + "mix.left.", m["left"]) + self.selective_scan(h, p + "mix.right.", m["right"]))
                x = x + self.experts(self.rms(x, p + "norm2", eps), p + "mlp.", model)
                history.append(x)
                x = sum(a * b for a, b in zip(self.w(p + "dwa", i + 2, role="average"), history))
            elif model == "pupinex":
                h = self.layer_norm(x, p + "norm1", eps)
                x = x + (self.sink_attention(h, p + "mix.", m, eps) if kind == "attention" else self.gla(h, p + "mix.", m, eps)
                         if kind == "gla" else self.normed_attention(h, p + "mix.left.", m["left"], eps)
                         + self.matrix_memory(h, p + "mix.right.", m["right"], eps))
                h = self.layer_norm(x, p + "norm2", eps)
                x = x + (self.gated(h, p + "mlp.", FF, self.clamped) if layer["mlp"]["kind"] == "dense"
                         else self.experts(h, p + "mlp.", model))
            elif model == "fokalorn":
                for hc, norm in (("hc1", "norm1"), ("hc2", "norm2")):
                    h = sum(a * s for a, s in zip(self.w(f"{p}{hc}.in", 4), streams))
                    h = self.rms(h, None, eps, 2) * self.w(p + norm, WIDTH, role="scale")
                    if hc == "hc1":
                        mu = self.w(p + "shift", WIDTH)
                        h = self.each(lambda s: s + (torch.nn.functional.pad(s, (0, 0, 1, 0))[:-1] - s) * mu, h)
                        y = (self.channel_delta(h, p + "mix.", m, eps) if kind == "channel_delta"
                             else self.latent_attention(h, p + "mix.", m, eps, True))
                    else:
                        y = self.squared(h, p + "mlp.")
                    mix, out = self.w(f"{p}{hc}.mix", 4, 4), self.w(f"{p}{hc}.out", 4)
                    streams = [sum(mix[s, t] * streams[s] for s in range(4)) + out[t] * y for t in range(4)]
                x = sum(streams)
            else:
                h = self.rms(x, p + "norm1", eps)
                x = x + 0.5 * (self.kept_attention(h, p + "mix.", m, memo) if kind == "attention" else self.mamba2(h, p + "mix.", m, eps))
                h = self.rms(x, p + "norm2", eps)
                relu = lambda g, u: torch.relu(g) * u
                x = x + 0.5 * (self.gated(h, p + "mlp.", FF, relu) if kind == "attention" else self.experts(h, p + "mlp.", model))
        if model == "pupinex":
            return self.layer_norm(x[rows], "final.norm", eps) @ table.T
        y = self.rms(x[rows], None, eps, 2 if model == "fokalorn" else 1) * self.w("final.norm", WIDTH, role="scale")
        y = self.lin(y, "head", c["vocab"])
        return 30.0 * torch.tanh(y / 30.0) if model == "muvetar" else y


def exact(case, seed):
    rng = np.random.default_rng(seed)
    cfg = _config(case)
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    lengths = _lengths(case)
    if sum(lengths) * case["layers"] * (5 if case["model"] == "llama-8b" else 1) > 1_700_000:
        return None                                                   # minutes of products
    prompts = [rng.integers(0, vocab, size=n) for n in lengths]
    decode = case["kind"] == "decode"
    feed = rng.integers(0, vocab, size=(CONTEXT - case["prompt"] if decode else case["steps"], case["requests"]))
    feed = feed[:case["steps"]]
    seqs = [np.concatenate([p, feed[:, j]]) for j, p in enumerate(prompts)]
    ends = np.cumsum([len(s) for s in seqs]).tolist()
    spans = [(e - len(s), e) for e, s in zip(ends, seqs)]
    first = case["steps"] if decode else 0                            # decode: the step's logits alone
    rows = [a + n - 1 + t for t in range(first, case["steps"] + 1) for (a, _), n in zip(spans, lengths)]
    tokens = torch.from_numpy(np.concatenate(seqs)).to("cuda")
    plain = _Plain(cfg, spans)
    with torch.no_grad():
        logits = plain.llama(tokens, rows) if case["model"].startswith("llama") else plain.other(case["model"], tokens, rows)
    out = list(logits.split(case["requests"]))
    return out[0] if decode else out
