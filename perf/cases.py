"""What a user of this engine has it do, as cases that can be timed and compared.

A case is one call of ``LLM.generate``: a number of requests with prompts of some lengths, each followed by some new
tokens, on one model with random weights.  Portions of prompts run beside decoded rows, pages are allocated and given
back, decode steps are recorded and replayed as graphs, next tokens are chosen on the GPU: everything that serving does.
The continuations are given (``_Scorer``): with random weights the two largest logits lie so close that a rounding
difference would send two correct engines down different continuations.  The sampler runs all the same, and the logits
of every row that it was given come back; in 32 bits, where ties do not matter, so do the tokens that it chose.

``exact`` restates the models in 64 bits with plain torch operations.
"""
from __future__ import annotations

import hashlib
import json
import math
import random

import torch

from allpaca_b200 import LLM, EngineConfig, SamplingParams, bench_designs
from allpaca_b200.config.presets import preset_config
from allpaca_b200.engine.runner import ModelRunner
from allpaca_b200.models import DecoderModel, resolve
from allpaca_b200.parts import BuildEnv, Workspace
from allpaca_b200.sampling.sampler import Pending, Sampler

F64 = torch.float64
PAGE = 16
BUDGET = 2048                       # rows of a step, the entry point's default
DESIGNS = ("viresun", "bivatar", "gezozen", "merusun")
PRESETS = ("llama-3.1-8b", "llama-3.2-1b")


def _case(name, model, requests, shortest, longest, new, portion=512, sampling="greedy", dtype="bfloat16", size=""):
    return {"name": name, "model": model, "size": size, "dtype": dtype, "requests": requests, "shortest": shortest,
            "longest": longest, "new": new, "portion": portion, "sampling": sampling}


def listed():
    return [
        # a question to a small model: the latency of single rows, launches one after another
        _case("1b one short", "llama-3.2-1b", 1, 23, 23, 64),
        # many users of a small model: ragged prompts cut into portions beside rows that decode
        _case("1b mixed", "llama-3.2-1b", 24, 16, 4096, 32, sampling="default"),
        # the 32-bit path, used to check a checkpoint or a conversion
        _case("1b float32", "llama-3.2-1b", 4, 20, 90, 8, sampling="default", dtype="float32"),
        # one conversation with some history: weight streaming at batch 1
        _case("8b one", "llama-3.1-8b", 1, 2048, 2048, 32),
        # the benchmark's middle point: batch 8 behind prompts of 2048 tokens
        _case("8b eight", "llama-3.1-8b", 8, 2048, 2048, 32, portion=2048),
        # a busy server: 64 conversations, short ragged prompts, sampling with the default options
        _case("8b sixty-four", "llama-3.1-8b", 64, 32, 512, 24, sampling="default"),
        # a long document read for a few tokens of answer
        _case("8b document", "llama-3.1-8b", 1, 8191, 8191, 3, portion=2048),
        # the other decoders at the sizes of their benchmark: state-space mixers and routed experts, ...
        _case("viresun base", "viresun", 8, 100, 700, 24, size="base"),
        # ... attention through a shared latent, ...
        _case("bivatar base", "bivatar", 16, 64, 1024, 16, size="base"),
        # ... linear attention beside softmax attention, experts with a shared expert, ...
        _case("gezozen base", "gezozen", 4, 300, 1500, 24, size="base"),
        # ... matrix memory and windowed latents, one prompt of 2048 tokens then single rows, ...
        _case("merusun base", "merusun", 1, 2048, 2048, 32, portion=2048, size="base"),
        # ... and the same at its largest size with many short requests
        _case("merusun wide", "merusun", 32, 48, 300, 12, size="wide", sampling="default"),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    model = rng.choices(PRESETS + DESIGNS, (3, 4, 2, 2, 2, 2))[0]
    c = _case("", model, _log_uniform(rng, 1, 64), 8, _log_uniform(rng, 8, 4096), _log_uniform(rng, 4, 48),
              rng.choice((256, 512, 2048)), rng.choice(("greedy", "default")))
    c["shortest"] = _log_uniform(rng, 8, c["longest"])
    if model in DESIGNS:
        c["size"] = rng.choices(("small", "base", "wide"), (2, 4, 1))[0]
    elif model == "llama-3.2-1b" and rng.random() < 0.25:
        c["dtype"] = "float32"
    # no more than a few seconds of the largest listed case's kind of work, whatever was drawn
    most = 12000 if c["dtype"] == "bfloat16" else 600
    while sum(_lengths(c)) + c["requests"] * c["new"] > most:
        if c["requests"] > 4 and rng.random() < 0.5:
            c["requests"] = c["requests"] * 2 // 3
        else:
            c["longest"] = max(8, c["longest"] * 2 // 3)
            c["shortest"] = min(c["shortest"], c["longest"])
            c["new"] = max(2, c["new"] * 3 // 4)
    if model == "llama-3.1-8b":
        c["new"] = min(c["new"], 24)
    if c["dtype"] == "float32":
        c["new"] = min(c["new"], 12)
    del c["name"]
    return c


# ---- the model of a case ------------------------------------------------------------------------
def _config(case):
    if case["model"] in PRESETS:
        return preset_config(case["model"])
    return getattr(bench_designs, case["model"] + "_config")(case["size"])


def _lengths(case):
    """Prompt lengths, spread over their logarithm: a matter of the case, not of the seed."""
    rng = random.Random(json.dumps([case["requests"], case["shortest"], case["longest"]]))
    return [_log_uniform(rng, case["shortest"], case["longest"]) for _ in range(case["requests"])]


def _tensor(case, name, shape, dtype):
    """One weight, the same on every call, drawn as decoders are commonly initialised before training: matrices
    N(0, 0.02) for the Llama shapes and of unit gain for the others, those that write to the residual stream smaller, so
    that no layer drowns the ones before it; norm weights around 1, decays that neither die at once nor keep everything."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int.from_bytes(hashlib.sha256(("%s %s %s" % (case["model"], case["size"], name)).encode()).digest()[:7],
                                   "little"))
    shape, leaf = tuple(shape), name.rsplit(".", 1)[-1]
    n = torch.empty(shape, dtype=torch.float32, device="cuda")
    if case["model"] in PRESETS:
        std = 0.02
        if name.endswith(("o_proj.weight", "down_proj.weight")):
            std /= math.sqrt(2.0 * _config(case)["num_hidden_layers"])
        elif "embed_tokens" in name:
            std = 0.1 if _config(case).get("tie_word_embeddings") else 1.0
        t = n.fill_(1.0) if len(shape) == 1 else n.normal_(0.0, std, generator=gen)
    elif leaf == "A_log":
        t = torch.log(0.02 + 0.3 * n.uniform_(0.0, 1.0, generator=gen))
    elif leaf in ("r1", "r2"):
        t = n.uniform_(0.05, 0.55, generator=gen) + (0.45 if leaf == "r1" else 0.0)
    elif leaf == "dt_bias":
        t = n.normal_(-0.5, 1.0, generator=gen)
    elif leaf.startswith("norm") or leaf == "D":
        t = n.normal_(1.0, 0.2, generator=gen)
    elif leaf == "conv":
        t = n.normal_(0.0, 0.5, generator=gen)
    elif name.endswith("a2.b") or name.endswith("f.b"):
        t = n.normal_(2.0, 1.0, generator=gen)
    elif len(shape) <= 1:
        t = n.normal_(0.0, 0.3, generator=gen)
    else:
        gain = 0.5 if leaf in ("o", "down") else 1.0
        t = n.normal_(0.0, 1.0 if name == "embed" else gain * shape[-1] ** -0.5, generator=gen)
    # every value a number of 16 bits, as in a checkpoint
    return t.to(torch.bfloat16).to(dtype)


def _tokens(case, seed):
    """(prompts, continuations) as lists of token ids."""
    gen = torch.Generator().manual_seed(int(seed))
    cfg = _config(case)
    vocab = int(cfg.get("vocab_size") or cfg["vocab"])
    lengths, new = _lengths(case), case["new"]
    prompts = [torch.randint(0, vocab, (n,), generator=gen).tolist() for n in lengths]
    return prompts, torch.randint(0, vocab, (len(lengths), new), generator=gen).tolist()


_engines = {}


def _engine(case):
    """The loaded model with its caches: a program keeps it from call to call, and so does this file (one at a time)."""
    key = json.dumps({k: v for k, v in case.items() if k not in ("name", "sampling")}, sort_keys=True)
    if key not in _engines:
        _engines.clear()
        torch.cuda.empty_cache()
        raw, lengths = _config(case), _lengths(case)
        longest = max(lengths) + case["new"]
        pages = sum(-(-(n + case["new"]) // PAGE) for n in lengths) + 4
        engine = EngineConfig(dtype=case["dtype"], page_size=PAGE, num_pages=pages, max_num_seqs=case["requests"],
                              max_num_batched_tokens=BUDGET, prefill_chunk=case["portion"], max_model_len=longest)
        engine.validate()
        env = BuildEnv(dtype=engine.dtype, device=torch.device("cuda:0"), workspace=Workspace(torch.device("cuda:0")),
                       page_size=PAGE, max_seqs=engine.max_num_seqs)
        arch = resolve(raw)
        cfg = arch.config_class.from_dict(raw)
        model = DecoderModel(arch.spec_builder(cfg), env)
        tied = bool(raw.get("tie_word_embeddings"))
        model.load_weights({name: _tensor(case, name, spec.shape, engine.dtype)
                            for name, (spec, _, local) in model.weight_targets().items()
                            if not (local == "head" and tied)})
        _engines[key] = ModelRunner(None, engine, model=model, model_config=cfg)
    return _engines[key]


class _Scorer(Sampler):
    """The engine's sampler, with every request continued by its given tokens whatever was chosen; keeps the logits of
    every row it is given, and the chosen tokens."""

    def __init__(self, device, params, continuations, vocab):
        super().__init__(device, len(params))
        B, new = len(params), len(continuations[0])
        self.row_of = {id(p): i for i, p in enumerate(params)}
        self.continuations, self.new = continuations, new
        self.logits = torch.empty((B * new, vocab), dtype=torch.float32, device=device)
        self.chosen = torch.empty(B * new, dtype=torch.int32, device=device)
        steps = B * new + 1                                  # no more launches than rows
        self.host = torch.empty((steps, 2, B), dtype=torch.int64, pin_memory=True)
        self.begin()

    def begin(self):
        self.step, self.done = 0, [0] * len(self.continuations)

    def launch(self, logits, params, uniforms):
        pending = super().launch(logits, params, uniforms)
        if not params:
            return pending                                   # a portion of a prompt that nobody wants logits of
        rows = [self.row_of[id(p)] for p in params]
        tokens = [self.continuations[r][self.done[r]] for r in rows]
        host = self.host[self.step].view(-1)[:2 * len(rows)].view(2, len(rows))
        host.numpy()[:] = [tokens, [r * self.new + self.done[r] for r in rows]]
        for r in rows:
            self.done[r] += 1
        self.step += 1
        given = host.to(self.device, non_blocking=True)
        self.logits.index_copy_(0, given[1], logits)
        self.chosen.index_copy_(0, given[1], pending.device[:len(rows)])
        mine = Pending(given[0].to(torch.int32), pending.host, pending.event, pending.rows)
        mine.tokens = tokens
        return mine

    def fetch(self, pending):
        super().fetch(pending)
        return getattr(pending, "tokens", [])


def prepare(case, seed):
    runner = _engine(case)
    prompts, continuations = _tokens(case, seed)
    if case["sampling"] == "greedy":
        params = [SamplingParams.greedy_params(max_tokens=case["new"]) for _ in prompts]
    else:
        params = [SamplingParams(max_tokens=case["new"], seed=int(seed) + i) for i in range(len(prompts))]
    scorer = _Scorer(runner.device, params, continuations, runner.vocab_size)
    return {"llm": LLM(runner=runner, sampler=scorer), "scorer": scorer, "prompts": prompts, "params": params,
            "tokens": case["dtype"] == "float32"}


def run(state):
    scorer = state["scorer"]
    scorer.begin()
    state["llm"].generate(state["prompts"], state["params"])
    return {"logits": scorer.logits, "chosen": scorer.chosen} if state["tokens"] else {"logits": scorer.logits}


# ---- how much a pass is, and how exact ----------------------------------------------------------
def _kept(layer, cfg):
    """(values a token keeps in pages, how many tokens back they are read) of one layer."""
    m = layer["mixer"]
    pair = m.get("left", m)
    window = (pair.get("mask") or {}).get("size") or 1 << 30
    if layer["type"] == "latent_attention":
        return m["kv_rank"] + m.get("rot_dim", 0), window
    if "kv_heads" in pair and layer["type"] != "delta":
        return pair["kv_heads"] * (pair["dim"] + pair["vdim"]), window
    return 0, 0


def work(case):
    """Bytes: the weights that a row needs once for every step (a step depends on the one before it and the weights are
    larger than any cache), the kept keys and values once for every step of a request, the logits.  Operations: the
    products of every row, the attention of every row over what it sees."""
    cfg, lengths, new, B = _config(case), _lengths(case), case["new"], case["requests"]
    arch = resolve(cfg)
    env = BuildEnv(dtype=torch.float32, device=torch.device("cpu"), workspace=Workspace(torch.device("cpu")))
    targets = DecoderModel(arch.spec_builder(arch.config_class.from_dict(cfg)), env).weight_targets()
    item = 4 if case["dtype"] == "float32" else 2
    dense = expert = head = 0
    for name, (spec, _, local) in targets.items():
        n = math.prod(spec.shape)
        if local == "head":
            head = n
        elif ".mlp.e" in name:
            expert += n
        elif local != "embedding" and len(spec.shape) > 1:
            dense += n
    share, layers = 0.0, cfg.get("layers") or []
    for r in (L["mlp"]["router"] for L in layers if (L.get("mlp") or {}).get("kind") == "moe"):
        share = r["top"] / r["experts"]
    if layers:
        kept = [_kept(L, cfg) for L in layers]
    else:
        hd = cfg.get("head_dim") or cfg["hidden_size"] // cfg["num_attention_heads"]
        kept = [(2 * cfg["num_key_value_heads"] * hd, 1 << 30)] * cfg["num_hidden_layers"]
    rows = sum(lengths) + B * (new - 1)
    prompt_steps = max(-(-sum(lengths) // BUDGET), max(-(-n // case["portion"]) for n in lengths))
    touched = expert * (1.0 - (1.0 - share) ** B)
    moved = prompt_steps * (dense + expert) + (new - 1) * (dense + touched) + new * head
    moved += sum(v * min(w, n) * new for n in lengths for v, w in kept) + rows * sum(v for v, _ in kept)
    heads = layers[0]["mixer"].get("heads", 16) if layers else cfg["num_attention_heads"]
    group = heads * 2 if any(L["type"] == "latent_attention" for L in layers) else 4
    seen = sum(v * sum(min(w, j) for j in (n / 4, 3 * n / 4)) / 2 * (n + new) for n in lengths for v, w in kept)
    return {"bytes": moved * item + B * new * head // (cfg.get("hidden_size") or cfg["width"]) * 4,
            "flops": 2.0 * rows * (dense + share * expert) + 2.0 * B * new * head + 2.0 * group * seen}


def tolerance(case):
    if case["dtype"] == "float32":
        # 7e-6 off the 64-bit logits
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.01}
    # the same prompts in portions of 128 tokens instead (other kernels, other orders of sums) give logits that are off
    # by 0.008 to 0.013 of themselves for the Llama shapes, by 0.002 to 0.006 for the others, single values by 0.3 where
    # a rounding sends a row to another expert
    return {"rel": 0.03 if case["model"] in PRESETS else 0.02, "max": 0.9}


# ---- the models in 64 bits ----------------------------------------------------------------------
class _Rows:
    """The rows of all requests one under another, and where each request's lie."""

    def __init__(self, lengths):
        self.lengths = lengths
        self.starts = [sum(lengths[:i]) for i in range(len(lengths))]
        self.positions = torch.cat([torch.arange(n) for n in lengths]).to("cuda", F64)
        self.longest = max(lengths)
        self.seq = torch.cat([torch.full((n,), i) for i, n in enumerate(lengths)]).cuda()
        self.pos = self.positions.long()

    def pad(self, x):
        """[rows, ...] -> [longest, requests, ...] with zeros behind the shorter ones."""
        out = torch.zeros((self.longest, len(self.lengths)) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
        out[self.pos, self.seq] = x
        return out

    def unpad(self, x):
        return x[self.pos, self.seq]


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(rows, q, k, v, scale, window=None, keep=0, bias=None, cap=None, one=False, block=512):
    """q [N, H, D], k [N, G, D], v [N, G, E], every request on its own; ``bias(distance [a, b]) -> [H, a, b]`` is added to
    the scores, ``cap`` bounds them, ``one`` adds one to the denominator."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=F64, device=q.device)
    for s, n in zip(rows.starts, rows.lengths):
        kk, vv = (t[s:s + n].transpose(0, 1).unsqueeze(1) for t in (k, v))                    # [G, 1, n, .]
        for a in range(0, n, block):
            b = min(n, a + block)
            lo = 0 if window is None or keep else max(0, a - window + 1)
            qq = q[s + a:s + b].transpose(0, 1).reshape(G, H // G, b - a, -1)
            z = (qq @ kk[:, :, lo:b].transpose(-1, -2)).reshape(H, b - a, b - lo) * scale
            j = torch.arange(lo, b, device=q.device)[None, :]
            dist = torch.arange(a, b, device=q.device)[:, None] - j
            if cap:
                z = cap * torch.tanh(z / cap)
            if bias is not None:
                z = z + bias(dist.clamp(min=0).to(F64))
            seen = dist >= 0
            if window is not None:
                seen = seen & ((dist < window) | (j < keep))
            z = z.masked_fill(~seen, -math.inf)
            if one:
                z = torch.cat([z, torch.zeros_like(z[..., :1])], dim=-1)
            p = torch.softmax(z, dim=-1)[..., :b - lo].reshape(G, H // G, b - a, b - lo)
            out[s + a:s + b] = (p @ vv[:, :, lo:b]).reshape(H, b - a, -1).transpose(0, 1)
    return out


def _angles(positions, dims, base, scaling=None):
    """Cosine and sine [N, dims/2] of a rotation; ``scaling`` stretches the slow pairs."""
    f, grow = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if scaling and scaling.get("rope_type") == "llama3":
        n0, lo, hi = (float(scaling[x]) for x in ("original_max_position_embeddings", "low_freq_factor", "high_freq_factor"))
        for i, x in enumerate(f):
            s = min(max((n0 * x / (2.0 * math.pi) - lo) / (hi - lo), 0.0), 1.0)
            f[i] = (1.0 - s) * x / float(scaling["factor"]) + s * x
    elif scaling:
        s, n = float(scaling["factor"]), float(scaling["original"])
        at = [dims * math.log(n / (2.0 * math.pi * float(scaling[t]))) / (2.0 * math.log(base)) for t in ("fast", "slow")]
        lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
        for i, x in enumerate(f):
            r = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            f[i] = x / s * r + x * (1.0 - r)
        grow = 0.1 * math.log(s) + 1.0
    a = positions[:, None] * torch.tensor(f, dtype=F64, device="cuda")[None, :]
    return torch.cos(a) * grow, torch.sin(a) * grow


def _rotate(x, angles, neighbours=False):
    """x [N, heads, dim]: pair i is (i, i + dims/2), or (2i, 2i + 1) among neighbours; coordinates beyond ``dims`` pass."""
    c, s = angles[0][:, None, :], angles[1][:, None, :]
    half = c.shape[-1]
    if neighbours:
        u, v = x[..., 0:2 * half:2], x[..., 1:2 * half:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., 2 * half:]], -1)
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def _recurrence(rows, q, k, v, decay, beta=None):
    """``S <- decay S + k u^T``, read out by q; u is v, or ``beta (v - S^T k)`` (delta rule).  Per head; ``decay`` [N, H, D]
    or [N, H, 1]."""
    q, k, v, decay = (rows.pad(t) for t in (q, k, v, decay))
    beta = rows.pad(beta) if beta is not None else None
    S = torch.zeros(v.shape[1:3] + (k.shape[-1], v.shape[-1]), dtype=F64, device="cuda")
    out = torch.empty_like(v)
    for t in range(rows.longest):
        S = decay[t].unsqueeze(-1) * S
        u = v[t]
        if beta is not None:
            u = beta[t].unsqueeze(-1) * (u - (k[t].unsqueeze(-2) @ S).squeeze(-2))
        S = S + k[t].unsqueeze(-1) * u.unsqueeze(-2)
        out[t] = (q[t].unsqueeze(-2) @ S).squeeze(-2)
    return rows.unpad(out)


def _conv(rows, x, w, bias=0.0):
    """Every channel filtered along time, the last tap on the row itself; then SiLU."""
    p, taps = rows.pad(x), w.shape[1]
    y = torch.zeros_like(p)
    for j in range(taps):
        back = taps - 1 - j
        y[back:] += p[:p.shape[0] - back] * w[:, j]
    return _silu(rows.unpad(y) + bias)


class _Plain:
    """One decoder over whole sequences; ``W(name, *shape)`` is a weight, ``lin`` a product with one."""

    def __init__(self, case, cfg, rows):
        self.case, self.cfg, self.rows = case, cfg, rows

    def W(self, name, *shape):
        return _tensor(self.case, name, shape, F64)

    def lin(self, name, x, out, bias=False):
        y = x @ self.W(name, out, x.shape[-1]).T
        return y + self.W(name + ".b", out) if bias else y

    def heads(self, name, x, heads, dim, bias=False):
        return self.lin(name, x, heads * dim, bias).reshape(-1, heads, dim)

    def rot(self, r):
        return _angles(self.rows.positions, int(r["dims"]), float(r["base"]), r.get("scaling"))

    def llama(self, tokens, wanted):
        c, R = self.cfg, self.rows
        eps, H, G = float(c["rms_norm_eps"]), c["num_attention_heads"], c["num_key_value_heads"]
        D, F, Wd, V = c["head_dim"], c["intermediate_size"], c["hidden_size"], c["vocab_size"]
        angles = _angles(R.positions, D, float(c["rope_theta"]), c.get("rope_scaling"))
        table = self.W("model.embed_tokens.weight", V, Wd)
        x = table[tokens]
        for i in range(c["num_hidden_layers"]):
            p = "model.layers.%d." % i
            h = _rms(x, eps)
            q, k = (_rotate(self.heads(p + "self_attn.%s_proj.weight" % n, h, m, D), angles) for n, m in (("q", H), ("k", G)))
            v = self.heads(p + "self_attn.v_proj.weight", h, G, D)
            x = x + self.lin(p + "self_attn.o_proj.weight", _attend(R, q, k, v, D ** -0.5).flatten(1), Wd)
            h = _rms(x, eps)
            h = _silu(self.lin(p + "mlp.gate_proj.weight", h, F)) * self.lin(p + "mlp.up_proj.weight", h, F)
            x = x + self.lin(p + "mlp.down_proj.weight", h, Wd)
        head = table if c.get("tie_word_embeddings") else self.W("lm_head.weight", V, Wd)
        return _rms(x[wanted], eps) @ head.T

    def experts(self, p, mlp, h, chosen, share, act, scaled_input=False):
        """Routed experts; ``act(prefix, rows)`` is one expert."""
        out = torch.zeros_like(h)
        for e in range(int(mlp["router"]["experts"])):
            row, place = (chosen == e).nonzero(as_tuple=True)
            if len(row):
                s = share[row, place][:, None]
                out[row] += act("%se%d" % (p, e), h[row] * s) if scaled_input else s * act("%se%d" % (p, e), h[row])
        return out

    # -- Viresun
    def viresun(self, tokens, wanted):
        c, R = self.cfg, self.rows
        eps, Wd, V = float(c["norm"]["eps"]), c["width"], c["vocab"]
        co, si = _angles(R.positions, Wd, 10000.0)
        x = self.W("embed", V, Wd)[tokens] + torch.stack([si, co], -1).flatten(1)
        x = _rms(x, eps) * self.W("embed.norm")
        for i, L in enumerate(c["layers"]):
            p, m = "l%d." % i, L["mixer"]
            h = _rms(x, eps) * self.W(p + "norm1")
            x = x + (self.biased(p + "mix.", m, h, eps) if L["type"] == "attention" else self.mamba(p + "mix.", m, h, eps))
            h = _rms(x, eps) * self.W(p + "norm2")
            p, mlp = p + "mlp.", L["mlp"]
            if mlp["kind"] == "dense":
                x = x + self.lin(p + "down", torch.relu(self.lin(p + "gate", h, mlp["ff"])) * self.lin(p + "up", h, mlp["ff"]), Wd)
                continue
            E, F, limit = mlp["router"]["experts"], mlp["expert"]["ff"], mlp["expert"]["limit"]
            best, chosen = (self.lin(p + "router", h, E) + self.W(p + "router.b", E)).topk(mlp["router"]["top"], dim=1)

            def one(q, rows):
                g = self.lin(q + ".gate", rows, F).clamp(max=limit)
                u = self.lin(q + ".up", rows, F).clamp(-limit, limit)
                return self.lin(q + ".down", g * torch.sigmoid(1.702 * g) * (u + 1.0), Wd)
            x = x + self.experts(p, mlp, h, chosen, torch.softmax(best, 1), one)
        return self.lin("head", _rms(x[wanted], eps) * self.W("final.norm"), V)

    def biased(self, p, m, h, eps):
        H, G, D, E = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k = _rms(self.heads(p + "q", h, H, D), eps), _rms(self.heads(p + "k", h, G, D), eps)
        turn = torch.floor((self.rows.positions + 1) / m["q_temp"]["every"]) + 1
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(turn))[:, None, None]
        r1, r2 = self.W(p + "r1", H)[:, None, None], self.W(p + "r2", H)[:, None, None]
        o = _attend(self.rows, q, k, self.heads(p + "v", h, G, E), m["scale"], m["mask"]["size"],
                    bias=lambda d: -r1 * torch.log1p(r2 * d))
        return self.lin(p + "o", o.flatten(1), h.shape[1])

    def mamba(self, p, m, h, eps):
        H, E, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, gn = H * E, G * N
        z, xbc, dt = self.lin(p + "in", h, 2 * inner + 2 * gn + H).split([inner, inner + 2 * gn, H], 1)
        xbc = _conv(self.rows, xbc, self.W(p + "conv", inner + 2 * gn, m["conv"]), self.W(p + "conv.b", inner + 2 * gn))
        x, B, C = xbc.split([inner, gn, gn], 1)
        x = x.reshape(-1, H, E)
        B, C = (t.reshape(-1, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        dt = torch.nn.functional.softplus(dt + self.W(p + "dt_bias", H), threshold=100.0)
        y = _recurrence(self.rows, C, dt.unsqueeze(-1) * B, x, torch.exp(-torch.exp(self.W(p + "A_log", H)) * dt).unsqueeze(-1))
        y = (y + self.W(p + "D", H)[:, None] * x).flatten(1) * _silu(z)
        y = _rms(y.reshape(y.shape[0], m["norm_groups"], -1), eps).flatten(1) * self.W(p + "norm", inner)
        return self.lin(p + "o", y, h.shape[1])

    # -- Bivatar
    def bivatar(self, tokens, wanted):
        c, R = self.cfg, self.rows
        eps, Wd, V, mult = float(c["norm"]["eps"]), c["width"], c["vocab"], float(c["residual_mult"])
        x, kept = self.W("embed", V, Wd)[tokens] * float(c["embedding"]["scale"]), {}
        for i, L in enumerate(c["layers"]):
            p, m = "l%d.mix." % i, L["mixer"]
            H, D, E = m["heads"], m["dim"], m["vdim"]
            if L["type"] == "latent_attention":
                src, rank, rd, angles = m.get("kv_from", i), m["kv_rank"], m["rot_dim"], self.rot(m["rot"])
                if src == i:
                    down = self.lin(p + "dkv", x, rank + rd)
                    kept[i] = _rms(down[:, :rank], eps) * self.W(p + "dkv.norm", rank), _rotate(down[:, None, rank:], angles)
                latent, turned = kept[src]
                q = _rms(self.lin(p + "dq", x, m["q_rank"]), eps) * self.W(p + "dq.norm", m["q_rank"])
                q = self.heads(p + "uq", q, H, D + rd)
                q = torch.cat([q[..., :D], _rotate(q[..., D:], angles)], -1)
                k = torch.cat([self.heads(p + "uk", latent, H, D), turned.expand(-1, H, -1)], -1)
                y = _attend(R, q, k, self.heads(p + "uv", latent, H, E), m["scale"])
            else:
                G = m["kv_heads"]
                q = _rms(self.heads(p + "q", x, H, D), eps) * self.W(p + "q.norm", D)
                k = _rms(self.heads(p + "k", x, G, D), eps) * self.W(p + "k.norm", D)
                slope = torch.tensor([2.0 ** (-8.0 * (a + 1) / H) for a in range(H)], dtype=F64, device="cuda")[:, None, None]
                y = _attend(R, q, k, self.heads(p + "v", x, G, E), m["scale"], m["mask"]["size"], m["mask"]["keep_first"],
                            lambda d: -slope * d)
            y = self.lin(p + "o", (y * torch.sigmoid(self.lin(p + "g", x, H))[:, :, None]).flatten(1), Wd)
            x = x + mult * _rms(y, eps) * self.W("l%d.norm1" % i, Wd)
            p, F = "l%d.mlp." % i, L["mlp"]["ff"]
            y = torch.nn.functional.gelu(self.lin(p + "gate", x, F), approximate="tanh") * self.lin(p + "up", x, F)
            x = x + mult * _rms(self.lin(p + "down", y, Wd), eps) * self.W("l%d.norm2" % i, Wd)
        return self.lin("head", _rms(x[wanted], eps) * self.W("final.norm", Wd), V)

    # -- Gezozen
    def gezozen(self, tokens, wanted):
        c = self.cfg
        eps, Wd, V, n = float(c["norm"]["eps"]), c["width"], c["vocab"], int(c["norm"]["groups"])

        def norm(x, name):
            return _rms(x.reshape(x.shape[0], n, -1), eps).flatten(1) * self.W(name, Wd)
        x = self.W("embed", V, Wd)[tokens]
        for i, L in enumerate(c["layers"]):
            p, m = "l%d." % i, L["mixer"]
            if L["type"] == "delta":
                y = self.delta(p + "mix.", m, x, eps)
            else:
                y = m["left_scale"] * self.left(p + "mix.left.", m["left"], x, eps, L["type"] == "parallel_2")
                y = y + m["right_scale"] * self.right(p + "mix.right.", m["right"], x, eps)
            x = norm(c["postln_alpha"] * x + torch.sigmoid(self.lin(p + "rg1", x, Wd, True)) * y, p + "norm1")
            mlp, q = L["mlp"], p + "mlp."
            E, F, S = mlp["router"]["experts"], mlp["expert"]["ff"], mlp["shared"]["ff"]
            share, chosen = torch.sigmoid(self.lin(q + "router", x, E)).topk(mlp["router"]["top"], dim=1)

            def one(name, rows, ff=F):
                return self.lin(name + ".down", _silu(self.lin(name + ".gate", rows, ff)) * self.lin(name + ".up", rows, ff), Wd)
            y = self.experts(q, mlp, x, chosen, share, one, scaled_input=True)
            y = y + torch.sigmoid(self.lin(q + "shared.sg", x, 1)) * one(q + "shared", x, S)
            x = norm(c["postln_alpha"] * x + torch.sigmoid(self.lin(p + "rg2", x, Wd, True)) * y, p + "norm2")
        return self.lin("head", norm(x[wanted], "final.norm"), V)

    def delta(self, p, m, h, eps):
        H, G, D, E, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
        q, k, v = (_conv(self.rows, self.lin(p + n, h, a * b), self.W(p + n + ".conv", a * b, taps)).reshape(-1, a, b)
                   for n, a, b in (("q", G, D), ("k", G, D), ("v", H, E)))
        q, k = ((t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for t in (q, k))
        step = torch.nn.functional.softplus(self.lin(p + "a", h, H) + self.W(p + "dt_bias", H), threshold=100.0)
        forget = torch.exp(-torch.exp(self.W(p + "A_log", H)) * step)
        o = _recurrence(self.rows, q * D ** -0.5, k, v, forget.unsqueeze(-1), torch.sigmoid(self.lin(p + "b", h, H)))
        o = (_rms(o, eps) * self.W(p + "norm", E)).flatten(1)
        return self.lin(p + "o", o * _silu(self.lin(p + "g", h, H * E)), h.shape[1])

    def left(self, p, m, h, eps, biased):
        H, G, D, E = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        angles = self.rot(m["rot"])
        q, k = (_rotate(_rms(self.heads(p + n, h, a, D, biased), eps) * self.W(p + n + ".norm", D), angles)
                for n, a in (("q", H), ("k", G)))
        o = _attend(self.rows, q, k, self.heads(p + "v", h, G, E, biased), m["scale"], (m.get("mask") or {}).get("size"),
                    cap=m.get("softcap"))
        return self.lin(p + "o", o.flatten(1), h.shape[1])

    def right(self, p, m, h, eps):
        H, D, E = m["heads"], m["dim"], m["vdim"]
        q, k, v = self.heads(p + "q", h, H, D), self.heads(p + "k", h, H, D), self.heads(p + "v", h, H, E)
        if "tau" in m:
            z = self.lin(p + "a2", self.lin(p + "a1", h, m["rank"]), H * D, True)
            o = _recurrence(self.rows, q * D ** -0.5, k, v,
                            torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(-1, H, D))
            o = _rms(o, eps) * self.W(p + "norm", E)
        else:
            angles = self.rot(m["rot"])
            decay = torch.tensor(m["decay"], dtype=F64, device="cuda")[None, :, None].expand(h.shape[0], -1, -1)
            o = _rms(_recurrence(self.rows, _rotate(q, angles), _rotate(k, angles) * D ** -0.5, v, decay), eps)
        return self.lin(p + "o", o.flatten(1) * _silu(self.lin(p + "g", h, H * E)), h.shape[1])

    # -- Merusun
    def merusun(self, tokens, wanted):
        c = self.cfg
        eps, Wd, V = float(c["norm"]["eps"]), c["width"], c["vocab"]
        x, kept = self.W("embed", V, Wd)[tokens] * float(c["embedding"]["scale"]), {}
        for i, L in enumerate(c["layers"]):
            p, m = "l%d." % i, L["mixer"]
            h, q = _rms(x, eps) * self.W(p + "norm1", Wd), p + "mix."
            H, D, E = m["heads"], m["dim"], m["vdim"]
            if L["type"] == "mlstm":
                y = self.memory(q, m, h, eps)
            elif L["type"] == "latent_attention":
                rank, rd, angles = m["kv_rank"], m["rot_dim"], self.rot(m["rot"])
                down = self.lin(q + "dkv", h, rank + rd)
                latent = _rms(down[:, :rank], eps) * self.W(q + "dkv.norm", rank)
                turned = _rotate(down[:, None, rank:], angles, True)
                k = torch.cat([self.heads(q + "uk", latent, H, D), turned.expand(-1, H, -1)], -1)
                a = self.heads(q + "q", h, H, D + rd)
                a = torch.cat([a[..., :D], _rotate(a[..., D:], angles, True)], -1)
                y = self.lin(q + "o", _attend(self.rows, a, k, self.heads(q + "uv", latent, H, E), m["scale"],
                                              m["mask"]["size"]).flatten(1), Wd)
            else:
                src, G = m.get("kv_from", i), m["kv_heads"]
                if src == i:
                    kept[i] = _rms(self.heads(q + "k", h, G, D, True), eps), self.heads(q + "v", h, G, E, True)
                a = _rms(self.heads(q + "q", h, H, D, True), eps)
                y = self.lin(q + "o", _attend(self.rows, a, *kept[src], m["scale"], m["mask"]["size"], one=True).flatten(1), Wd)
            x = x + _rms(y, eps) * self.W(p + "norm1b", Wd)
            h, q, mlp = _rms(x, eps) * self.W(p + "norm2", Wd), p + "mlp.", L["mlp"]
            r, F = mlp["router"], mlp["expert"]["ff"]
            n, groups = r["experts"], r["groups"]
            s = torch.softmax(self.lin(q + "router", h, n), -1)
            best = s.reshape(-1, groups["count"], n // groups["count"]).amax(-1).topk(groups["keep"], -1).indices
            shut = torch.ones(len(s), groups["count"], dtype=torch.bool, device="cuda").scatter(1, best, False)
            chosen = s.masked_fill(shut.repeat_interleave(n // groups["count"], 1), -1.0).topk(r["top"], -1).indices

            def one(name, rows, ff=F):
                return self.lin(name + ".down", torch.relu(self.lin(name + ".up", rows, ff)).square(), Wd)
            y = self.experts(q, mlp, h, chosen, s.gather(1, chosen) * r["scale"], one) + one(q + "shared", h, mlp["shared"]["ff"])
            x = x + _rms(y, eps) * self.W(p + "norm2b", Wd)
        return self.lin("head", _rms(x[wanted], eps) * self.W("final.norm", Wd), V)

    def memory(self, p, m, h, eps):
        H, D, E, cap = m["heads"], m["dim"], m["vdim"], float(m["gate_cap"])
        q, k, v = self.heads(p + "q", h, H, D) * D ** -0.5, self.heads(p + "k", h, H, D), self.heads(p + "v", h, H, E)
        i, f = (cap * torch.tanh(self.lin(p + n, h, H, True) / cap) for n in ("i", "f"))
        i, f = self.rows.pad(i), self.rows.pad(torch.nn.functional.logsigmoid(f))
        top, keep, write, floor = torch.zeros_like(i[0]), [], [], []
        for t in range(self.rows.longest):
            new = torch.maximum(f[t] + top, i[t])
            keep.append(torch.exp(f[t] + top - new))
            write.append(torch.exp(i[t] - new))
            floor.append(torch.exp(-new))
            top = new
        keep, write, floor = (self.rows.unpad(torch.stack(t)) for t in (keep, write, floor))
        # the vector beside the matrix is one more value column, of ones
        wide = torch.cat([v, torch.ones_like(v[..., :1])], -1)
        o = _recurrence(self.rows, q, write.unsqueeze(-1) * k, wide, keep.unsqueeze(-1))
        o = o[..., :E] / (torch.maximum(o[..., E].abs(), floor) + 1e-6).unsqueeze(-1)
        o = _rms(o, eps).flatten(1)
        return self.lin(p + "o", o * self.W(p + "norm", H * E) * torch.sigmoid(self.lin(p + "g", h, H * E)), h.shape[1])


def exact(case, seed):
    prompts, continuations = _tokens(case, seed)
    new = case["new"]
    sequences = [p + c[:new - 1] for p, c in zip(prompts, continuations)]
    rows = _Rows([len(s) for s in sequences])
    tokens = torch.tensor([t for s in sequences for t in s], device="cuda")
    wanted = torch.cat([torch.arange(s + len(p) - 1, s + len(p) - 1 + new) for s, p in zip(rows.starts, prompts)]).cuda()
    plain = _Plain(case, _config(case), rows)
    kind = "llama" if case["model"] in PRESETS else case["model"]
    logits = getattr(plain, kind)(tokens, wanted)
    if case["dtype"] != "float32":
        return {"logits": logits}
    return {"logits": logits, "chosen": logits.argmax(-1).to(torch.int32) if case["sampling"] == "greedy" else None}
