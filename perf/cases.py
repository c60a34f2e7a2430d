"""What a program that serves models with this library has it do, as cases that can be timed and compared.

A case is one round of work on an engine that a program keeps: requests come in, their prompts run through
`Engine.step` (whole, or in portions), then every sequence is carried on token by token with given tokens, as trace
replay, scoring and any server's loop above the step function do it, and the slots are given back.  The outputs are the
logits of every step.  One case goes through `Engine.generate` (greedy, float32, where the tokens are determined) and
scores what came out, as `tq run` and `tq perplexity` do.

The models are the shapes of real size that the package holds (`tq_kv_b200/config/shapes`: qwen2.5-0.5b, qwen2.5-7b,
zodosun-2k, rirudra-2k) and the Pavisun decoder of width 2,048 that `bench.py --design pavisun` runs (routed experts,
residual streams, windows; its routing is a table, so that no near tie decides it).  qwen2.5-32b runs the 7B shape's
kernels; through its 64 layers of random weights bfloat16 rounding alone moves the logits by 7 %, too much to compare.
Weights are random (the package's own generator, seed 0): nothing here depends on their values.  An engine is kept
between states, as a program keeps it; the prompts and the given tokens are a state's own and come from its seed.
"""
from __future__ import annotations

import gc
import math

import torch

import tq_kv_b200 as tq
from tq_kv_b200.config import spec_from_config_dict
from tq_kv_b200.engine.model import DecoderModel
from tq_kv_b200.weights.random_init import random_tensor

WEIGHT_SEED = 0


# ---- the cases -----------------------------------------------------------------------------------------------------
def _case(name, model, batch, prompt, new, *, dtype="bfloat16", ragged=False, portion=0, generate=False):
    """`batch` requests of `prompt` tokens (`ragged`: of half of it up to all of it), `new` tokens each; `portion`: the
    most prompt tokens of a sequence that one step takes (0: whole prompts); `generate`: through Engine.generate."""
    c = {"model": model, "dtype": dtype, "batch": batch, "prompt": prompt, "ragged": ragged, "new": new,
         "portion": portion, "generate": generate}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a short chat turn on the smallest model: a few hundred small launches a token, nothing else
        _case("chat turn 0.5B", "qwen2.5-0.5b", 1, 40, 24),
        # a chat turn with some history on the usual model: every token reads all weights once
        _case("chat turn 7B", "qwen2.5-7b", 1, 300, 24),
        # a small service: eight requests of unequal length, prompts of a page or two of text
        _case("eight requests 7B", "qwen2.5-7b", 8, 1200, 32, ragged=True),
        # a full batch of short unequal requests
        _case("full batch 7B", "qwen2.5-7b", 64, 320, 12, ragged=True),
        # a document read in portions, so that other work gets in between, then a short answer
        _case("document in portions 7B", "qwen2.5-7b", 1, 6000, 6, portion=2048),
        # the true 32-bit path: greedy generation, then every position's logits
        _case("generate and score 0.5B float32", "qwen2.5-0.5b", 2, 150, 16, dtype="float32", generate=True),
        # a long prompt on the decoders with recurrent states: the chain of states is the prompt's time
        _case("long prompt Zodosun", "zodosun-2k", 1, 3000, 24),
        _case("long prompt Rirudra", "rirudra-2k", 1, 3000, 24),
        # many unequal requests on the same: states and pages of many sequences
        _case("thirty-two requests Zodosun", "zodosun-2k", 32, 300, 24, ragged=True),
        # a full batch whose prompts come in odd portions
        _case("full batch in portions Rirudra", "rirudra-2k", 64, 210, 24, ragged=True, portion=77),
        # the 32-bit path of a decoder with states
        _case("four requests Rirudra float32", "rirudra-2k", 4, 250, 16, dtype="float32", ragged=True),
        # routed experts and windows, an ordinary batch
        _case("sixteen requests Pavisun", "pavisun-2k", 16, 500, 24, ragged=True),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        model = rng.choice(["qwen2.5-0.5b", "qwen2.5-7b", "qwen2.5-7b", "zodosun-2k", "rirudra-2k", "pavisun-2k"])
        dtype = "float32" if model != "qwen2.5-7b" and rng.random() < 0.2 else "bfloat16"
        batch = _log_int(rng, 1, 64)
        prompt = _log_int(rng, 16, 512 if dtype == "float32" else 6000)
        portion = _log_int(rng, 48, max(48, prompt // 2)) if prompt >= 128 and rng.random() < 0.25 else 0
        generate = model == "qwen2.5-0.5b" and dtype == "float32" and batch * prompt <= 600 and rng.random() < 0.5
        c = _case(None, model, batch, prompt, _log_int(rng, 2, 40), dtype=dtype,
                  ragged=batch > 1 and rng.random() < 0.75, portion=0 if generate else portion, generate=generate)
        steps = (-(-prompt // portion) if portion else 1) + c["new"]
        if _cost(c) <= most and steps <= 60 and batch * prompt <= 40000:
            return c


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (6e13 if case["dtype"] == "float32" else 1.6e15))


def _config(model):
    if model != "pavisun-2k":
        return tq.named_shape(model)
    mlp = {"kind": "moe", "expert": {"ff": 2816}, "router": {"experts": 8, "top": 2}}
    unit = {"type": "attention_2", "mlp": mlp, "mixer": {
        "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 1.0, "mask": {"size": 1024, "keep_first": 4}}}
    turned = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
        "mask": {"size": 1024},
        "rot": {"base": 1e6, "dims": 128, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    return {"architecture": "Pavisun", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "streams": 4,
            "logit_softcap": 30.0, "max_positions": 8192, "layers": [unit, turned, unit, turned]}


def _lengths(case):
    B, P = case["batch"], case["prompt"]
    return [P - (i * 7919) % (P // 2 + 1) if case["ragged"] else P for i in range(B)]


def _steps(case):
    """The steps of a pass: lists of (sequence, first token, end, whether the last token's logits are wanted)."""
    lens, out = _lengths(case), []
    size, at = case["portion"] or max(lens), 0
    while at < max(lens):
        out.append([(i, at, min(n, at + size), at + size >= n) for i, n in enumerate(lens) if at < n])
        at += size
    for k in range(case["new"]):
        out.append([(i, n + k, n + k + 1, True) for i, n in enumerate(lens)])
    return out


# ---- what a program holds before the call, and the call ----------------------------------------------------------------
_kept: dict = {}         # the one engine that is kept, by what it was made for


def _engine(case):
    B, total = case["batch"], case["prompt"] + case["new"]
    context = max(2048, -(-(total + 1) // 512) * 512)
    key = (case["model"], case["dtype"], B, context, total, case["portion"])
    if key not in _kept:
        _kept.clear()
        gc.collect()
        torch.cuda.empty_cache()
        _kept[key] = tq.Engine.from_random(
            _config(case["model"]), seed=WEIGHT_SEED, dtype=case["dtype"], max_slots=B, max_context=context,
            max_tokens=B * (-(-(total + 1) // 64) * 64), window_chunk=max(64, case["portion"]))
    return _kept[key]


def _tokens(case, seed):
    """Per sequence: its prompt and the tokens it goes on with."""
    vocab = _config(case["model"]).get("vocab_size") or _config(case["model"])["vocab"]
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (n + case["new"],), generator=g).tolist() for n in _lengths(case)]


def prepare(case, seed):
    return {"case": case, "engine": _engine(case), "tokens": _tokens(case, seed), "steps": _steps(case)}


def run(state):
    case, engine, tokens = state["case"], state["engine"], state["tokens"]
    if case["generate"]:
        prompts = [t[:n] for t, n in zip(tokens, _lengths(case))]
        results = engine.generate(prompts, tq.GenerationParams.greedy(case["new"], stop_token_ids=()))
        slots = [engine.new_sequence() for _ in prompts]
        whole = [p + r.tokens for p, r in zip(prompts, results)]
        logits = engine.step([tq.StepRow(s, t, list(range(len(t)))) for s, t in zip(slots, whole)])
        for s in slots:
            engine.release(s)
        return {"tokens": torch.tensor([r.tokens for r in results]), "logits": logits}
    slots = [engine.new_sequence() for _ in tokens]
    out = []
    for rows in state["steps"]:
        logits = engine.step([tq.StepRow(slots[i], tokens[i][a:b], [b - a - 1] if want else [])
                              for i, a, b, want in rows])
        if logits is not None:
            out.append(logits)
    for s in slots:
        engine.release(s)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
_sizes_of: dict = {}


def _sizes(model):
    """Per model: matrix entries that every token uses, of all experts and of those a token uses, of the head; values
    cached per token, entries of state per sequence, operations per query and visible key, operations on the states per
    token, the window."""
    if model in _sizes_of:
        return _sizes_of[model]
    c = _config(model)
    spec = spec_from_config_dict(c)[2]
    specs = DecoderModel(spec).weight_specs()
    count = {n: math.prod(s.shape) for n, s in specs.items()}
    embed = next(n for n in count if n in ("embed", "model.embed_tokens.weight"))
    head = next((n for n in count if n in ("head", "lm_head.weight")), embed)
    experts = sum(v for n, v in count.items() if ".mlp.e" in n)
    every = sum(v for n, v in count.items()
                if n not in (embed, head) and ".mlp.e" not in n and not n.endswith(".table"))
    cached = state = pair = chain = 0
    if "num_hidden_layers" in c:
        L, H, G, d = c["num_hidden_layers"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        cached, pair = 2 * L * G * d, 4 * L * H * d
    for layer in c.get("layers", ()):
        m, kind = layer["mixer"], layer["type"]
        if kind == "general_delta":
            state, chain = state + m["heads"] * m["dim"] ** 2, chain + 8 * m["heads"] * m["dim"] ** 2
        elif kind == "parallel":
            a, b = m["left"], m["right"]
            cached, pair = cached + a["kv_heads"] * (a["dim"] + a["vdim"]), pair + 2 * a["heads"] * (a["dim"] + a["vdim"])
            state, chain = state + b["heads"] * b["dim"] * b["vdim"], chain + 5 * b["heads"] * b["dim"] * b["vdim"]
        elif kind == "latent_attention":
            cached, pair = cached + m["kv_rank"] + m["rot_dim"], pair + 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif kind in ("mamba2", "delta"):
            n = m["heads"] * m["vdim"] * (m["state"] if kind == "mamba2" else m["dim"])
            state, chain = state + n, chain + (5 if kind == "mamba2" else 7) * n
        else:                                                   # attention, attention_2
            values = m["kv_heads"] * (m["dim"] * (2 if kind == "attention_2" else 1) + m["vdim"] * (kind == "attention"))
            cached, pair = cached + values, pair + 2 * m["heads"] * (m["dim"] + m["vdim"])
    out = {"every": every, "experts": experts, "used": experts // 4, "head": count[head], "vocab": specs[head].shape[0],
           "width": specs[embed].shape[1], "cached": cached, "state": state, "pair": pair, "chain": chain,
           "window": 1024 if model == "pavisun-2k" else 1 << 30}
    _sizes_of[model] = out
    return out


def work(case):
    z = _sizes(case["model"])
    es = 4 if case["dtype"] == "float32" else 2
    steps = _steps(case)
    if case["generate"]:        # prompts, new - 1 single tokens, and one step over everything with all logits wanted
        lens = _lengths(case)
        steps = steps[:1] + steps[1:case["new"]] + [[(i, 0, n + case["new"], True) for i, n in enumerate(lens)]]
    nbytes = flops = 0
    for k, rows in enumerate(steps):
        scored = case["generate"] and k == len(steps) - 1
        n = sum(b - a for _, a, b, _ in rows)
        wanted = n if scored else sum(w for _, _, _, w in rows)
        share = min(1.0, 0.25 * n) if z["experts"] else 0.0
        nbytes += es * (z["every"] + share * z["experts"] + (z["head"] if wanted else 0) + n * (z["width"] + z["cached"]))
        nbytes += 4 * wanted * z["vocab"] + 8 * len(rows) * z["state"]
        flops += 2 * n * (z["every"] + z["used"]) + 2 * wanted * z["head"] + n * z["chain"]
        for _, a, b, _ in rows:
            nbytes += es * z["cached"] * min(a, z["window"])
            full = max(0, b - max(a, z["window"]))              # queries whose window is full
            ramp = (b - a) - full
            flops += z["pair"] * (full * z["window"] + ramp * (a + 1 + a + ramp) / 2)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # against 64 bits the path measures 3.6e-6 (float32); 0.007 (Rirudra), 0.02 (Zodosun), 0.04 (7B, 28 layers) to 0.05
    # (Pavisun) in bfloat16, and up to 0.014 from itself where sums meet in another order
    return {"rel": 1.5e-5, "differ": 0.0} if case["dtype"] == "float32" else {"rel": 0.03}


# ---- the same in 64 bits, plain torch ----------------------------------------------------------------------------------
def exact(case, seed):
    z = _sizes(case["model"])
    B, T = case["batch"], case["prompt"] + case["new"]
    if 2.0 * (z["every"] + z["experts"]) * B * T > 3.5e14:
        return None
    tokens, lens = _tokens(case, seed), _lengths(case)
    with torch.no_grad():
        model = _Plain(_config(case["model"]))
        if case["generate"]:
            seqs = [t[:n] for t, n in zip(tokens, lens)]
            for _ in range(case["new"]):
                rows = model.logits(seqs, [(i, len(s) - 1) for i, s in enumerate(seqs)])
                seqs = [s + [int(t)] for s, t in zip(seqs, rows.argmax(-1).tolist())]
            out = {"tokens": torch.tensor([s[n:] for s, n in zip(seqs, lens)]),
                   "logits": model.logits(seqs, [(i, t) for i, s in enumerate(seqs) for t in range(len(s))])}
        else:
            steps = [[(i, b - 1) for i, _, b, want in rows if want] for rows in _steps(case)]
            steps = [s for s in steps if s]
            got = model.logits(tokens, [p for s in steps for p in s])
            out = list(got.split([len(s) for s in steps]))
    return out


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _unit(x):
    return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _rates(dims, base, scaling=None):
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    f = base ** (-2.0 * i / dims)
    if not scaling:
        return f, 1.0

    def index_of(turns):
        return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(index_of(scaling["fast"])), 0), min(math.ceil(index_of(scaling["slow"])), dims - 1)
    r = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / scaling["factor"] * r + f * (1 - r), 0.1 * math.log(scaling["factor"]) + 1.0


def _turn(x, dims, base, *, pairs, scaling=None):
    """x [B, T, heads, n] rotated by position over its first `dims` entries, in neighbouring pairs or in halves."""
    rate, m = _rates(dims, base, scaling)
    ang = torch.arange(x.shape[1], dtype=torch.float64, device="cuda").reshape(-1, 1, 1) * rate
    c, s = m * torch.cos(ang), m * torch.sin(ang)
    ia, ib = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    out, a, b = x.clone(), x[..., ia], x[..., ib]
    out[..., ia], out[..., ib] = a * c - b * s, b * c + a * s
    return out


def _attend(q, k, v, weights_of):
    """q [B, T, H, d], k, v [B, T, G, .]: weights_of(scores [h, T, T], first head) gives the weights of the masked scores'
    heads; returns [B, T, H * e]."""
    B, T, H, _ = q.shape
    n = H // k.shape[2]
    out = q.new_empty(B, T, H, v.shape[-1])
    some = max(1, int(2e9 // (8 * T * T)))                       # heads at a time: bounds the scores' memory
    for b in range(B):
        for h in range(0, H, some):
            heads = torch.arange(h, min(H, h + some), device="cuda")
            s = torch.einsum("thd,shd->hts", q[b, :, heads], k[b, :, heads // n])
            out[b, :, heads] = torch.einsum("hts,shd->thd", weights_of(s, heads), v[b, :, heads // n])
    return out.reshape(B, T, -1)


class _Plain:
    """The decoders over whole padded sequences in float64 (padding follows the tokens, and everything is causal)."""

    def __init__(self, config):
        self.c = config
        self.specs = DecoderModel(spec_from_config_dict(config)[2]).weight_specs()

    def w(self, name):
        s = self.specs[name]
        t = random_tensor(name, tuple(s.shape), s.role, WEIGHT_SEED, torch.bfloat16, "cuda")
        return t.double() if t.is_floating_point() else t.long()

    def mul(self, x, name):
        return x @ self.w(name).T

    def logits(self, seqs, places):
        T = max(len(s) for s in seqs)
        tok = torch.tensor([s + [0] * (T - len(s)) for s in seqs], device="cuda")
        far = torch.arange(T, device="cuda")
        self.dist = far.reshape(-1, 1) - far.reshape(1, -1)      # query minus key
        x, head = getattr(self, "_" + (self.c.get("architecture") or "qwen2").lower())(tok)
        b, t = (torch.tensor(p, device="cuda") for p in zip(*places))
        cap = self.c.get("logit_softcap")
        out = self.mul(x[b, t], head) * self.c.get("logit_scale", 1.0)
        return cap * torch.tanh(out / cap) if cap else out

    def ff(self, x, p, gate="gate", up="up", down="down"):
        return self.mul(_silu(self.mul(x, p + gate)) * self.mul(x, p + up), p + down)

    def softmax(self, s, mask=None):
        return s.masked_fill_(self.dist < 0 if mask is None else ~mask, -math.inf).softmax(-1)

    # Qwen2
    def _qwen2(self, tok):
        c = self.c
        H, G, d, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
        x = self.w("model.embed_tokens.weight")[tok]
        B, T, _ = x.shape
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            n = _rms(x, eps) * self.w(p + "input_layernorm.weight")
            q, k, v = (self.mul(n, f"{p}self_attn.{a}_proj.weight") + self.w(f"{p}self_attn.{a}_proj.bias") for a in "qkv")
            q, k, v = q.reshape(B, T, H, d), k.reshape(B, T, G, d), v.reshape(B, T, G, d)
            q, k = (_turn(a, d, c["rope_theta"], pairs=False) for a in (q, k))
            o = _attend(q, k, v, lambda s, h: self.softmax(s / math.sqrt(d)))
            x = x + self.mul(o, p + "self_attn.o_proj.weight")
            n = _rms(x, eps) * self.w(p + "post_attention_layernorm.weight")
            x = x + self.ff(n, p + "mlp.", "gate_proj.weight", "up_proj.weight", "down_proj.weight")
        return (_rms(x, eps) * self.w("model.norm.weight"),
                "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight")

    # Zodosun
    def _zodosun(self, tok):
        c, eps, W = self.c, self.c["norm"]["eps"], self.c["width"]
        T = tok.shape[1]
        ang = torch.arange(T, dtype=torch.float64, device="cuda").reshape(-1, 1) * _rates(W, 10000.0)[0]
        x = self.w("embed")[tok] + torch.stack([torch.sin(ang), torch.cos(ang)], -1).reshape(T, W)
        for i, layer in enumerate(c["layers"]):
            p = f"l{i}."
            n = self.grouped(x, eps) * self.w(p + "norm1")
            if layer["type"] == "parallel":
                a = self.sigmoid_attention(n, p + "mix.left.", layer["mixer"]["left"], eps)
                b = self.decayed_sum(n, p + "mix.right.", layer["mixer"]["right"], eps)
                x = x + 0.5 * (_rms(a, eps) * self.w(p + "mix.left.out") + _rms(b, eps) * self.w(p + "mix.right.out"))
            else:
                x = x + self.delta_rule(n, p + "mix.", layer["mixer"], eps)
            x = x + self.ff(self.grouped(x, eps) * self.w(p + "norm2"), p + "mlp.")
        return self.grouped(x, eps) * self.w("final.norm"), "head"

    def grouped(self, x, eps):
        g = self.c["norm"]["groups"]
        return _rms(x.reshape(*x.shape[:-1], g, -1), eps).reshape(x.shape)

    def sigmoid_attention(self, n, p, m, eps):
        B, T, _ = n.shape
        H, G, d, e, t = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["q_temp"]
        q, k, v = (self.mul(n, p + a) + self.w(p + a + ".b") for a in "qkv")
        q, k = _rms(q, eps) * self.w(p + "q.norm"), _rms(k, eps) * self.w(p + "k.norm")
        at = torch.arange(T, device="cuda")
        q = q * (1.0 + t["coef"] * torch.log(((at + 1) // t["every"] + 1).double())).reshape(-1, 1)
        table, half, far = self.w(p + "rel"), m["bias_rows"] // 2, m["bias_max"]
        row = [j if j < half else min(2 * half - 1, half + int(math.floor(math.log(j / half) / math.log(far / half) * half)))
               for j in range(T)]
        row = torch.tensor(row, device="cuda")[self.dist.clamp(min=0)]
        offset = self.w(p + "pb")

        def weights(s, h):
            s = torch.sigmoid(s * m["scale"] + table[row][..., h].permute(2, 0, 1) + offset[h].reshape(-1, 1, 1))
            return s.masked_fill_(self.dist < 0, 0.0)

        o = _attend(q.reshape(B, T, H, d), k.reshape(B, T, G, d), v.reshape(B, T, G, e), weights)
        o = o.reshape(B, T, H, e) * torch.sigmoid(self.mul(n, p + "g")).unsqueeze(-1)
        return self.mul(o.reshape(B, T, H * e), p + "o")

    def decayed_sum(self, n, p, m, eps):
        B, T, _ = n.shape
        H, d, e = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(self.mul(n, p + a)).reshape(B, T, H, -1) for a in "qkv")
        decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda").reshape(1, H, 1, 1)
        S, o = n.new_zeros(B, H, d, e), n.new_empty(B, T, H, e)
        for t in range(T):
            S = torch.addcmul(decay * S, k[:, t].unsqueeze(-1), v[:, t].unsqueeze(-2))
            o[:, t] = (q[:, t].unsqueeze(-2) @ S).squeeze(-2)
        o = _rms(o.reshape(B, T, H * e), eps) * self.w(p + "norm")
        return self.mul(o * torch.sigmoid(self.mul(n, p + "g")), p + "o")

    def delta_rule(self, n, p, m, eps):
        B, T, _ = n.shape
        H, d = m["heads"], m["dim"]
        r, k, v = (self.mul(n, p + a).reshape(B, T, H, d) for a in "rkv")
        low = torch.tanh(self.mul(n, p + "w1")) @ self.w(p + "w2").T + self.w(p + "w0")
        keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(low)).reshape(B, T, H, d, 1)
        u = _unit(k)
        off = (torch.sigmoid(self.mul(n, p + "a") + self.w(p + "a.b")).reshape(B, T, H, d) * u).unsqueeze(-1)
        S, o = n.new_zeros(B, H, d, d), n.new_empty(B, T, H, d)
        for t in range(T):
            uS = u[:, t].unsqueeze(-2) @ S
            S = torch.addcmul(keep[:, t] * S - off[:, t] * uS, k[:, t].unsqueeze(-1), v[:, t].unsqueeze(-2))
            o[:, t] = (r[:, t].unsqueeze(-2) @ S).squeeze(-2)
        o = _rms(o, eps).reshape(B, T, H * d) * self.w(p + "norm")
        return self.mul(o * torch.sigmoid(self.mul(n, p + "g")), p + "o")

    # Rirudra
    def _rirudra(self, tok):
        c, eps = self.c, self.c["norm"]["eps"]
        x = self.w("embed")[tok] * c["embedding"]["scale"]
        mixers = {"delta": self.gated_delta, "mamba2": self.state_space, "latent_attention": self.latent_attention}
        for i, layer in enumerate(c["layers"]):
            p = f"l{i}."
            n = _rms(x, eps) * (1.0 + self.w(p + "norm1"))
            x = x + c["residual_mult"] * (mixers[layer["type"]](n, p + "mix.", layer["mixer"], eps) + self.ff(n, p + "mlp."))
        return _rms(x, eps) * (1.0 + self.w("final.norm")), "embed"

    def conv(self, x, name, bias=None):
        taps, T = self.w(name), x.shape[1]
        K = taps.shape[1]
        padded = torch.nn.functional.pad(x, (0, 0, K - 1, 0))
        y = sum(padded[:, j:j + T] * taps[:, j] for j in range(K))
        return _silu(y + self.w(bias) if bias else y)

    def gated_delta(self, n, p, m, eps):
        B, T, _ = n.shape
        H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (self.conv(self.mul(n, p + a), p + a + ".conv") for a in "qkv")
        q, k = (_unit(a.reshape(B, T, G, d)).repeat_interleave(H // G, 2) for a in (q, k))
        q, v = q * d ** -0.5, v.reshape(B, T, H, e)
        beta = torch.sigmoid(self.mul(n, p + "b")).unsqueeze(-1)
        step = torch.nn.functional.softplus(self.mul(n, p + "a") + self.w(p + "dt_bias"), threshold=30.0)
        g = torch.exp(-torch.exp(self.w(p + "A_log")) * step).reshape(B, T, H, 1, 1)
        S, o = n.new_zeros(B, H, d, e), n.new_empty(B, T, H, e)
        for t in range(T):
            S = g[:, t] * S
            u = beta[:, t] * (v[:, t] - (k[:, t].unsqueeze(-2) @ S).squeeze(-2))
            S = torch.addcmul(S, k[:, t].unsqueeze(-1), u.unsqueeze(-2))
            o[:, t] = (q[:, t].unsqueeze(-2) @ S).squeeze(-2)
        o = (_rms(o, eps) * self.w(p + "norm")).reshape(B, T, H * e)
        return self.mul(o * _silu(self.mul(n, p + "g")), p + "o")

    def state_space(self, n, p, m, eps):
        B, T, _ = n.shape
        H, e, N, G, R = m["heads"], m["vdim"], m["state"], m["groups"], m["norm_groups"]
        z, xbc, dt = self.mul(n, p + "in").split([H * e, H * e + 2 * G * N, H], -1)
        x, b, c = self.conv(xbc, p + "conv", p + "conv.b").split([H * e, G * N, G * N], -1)
        x = x.reshape(B, T, H, e)
        b, c = (a.reshape(B, T, G, N).repeat_interleave(H // G, 2) for a in (b, c))
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias"), threshold=30.0)
        decay = torch.exp(-torch.exp(self.w(p + "A_log")) * dt).reshape(B, T, H, 1, 1)
        b = (dt.unsqueeze(-1) * b).unsqueeze(-1)
        S, y = n.new_zeros(B, H, N, e), n.new_empty(B, T, H, e)
        for t in range(T):
            S = torch.addcmul(decay[:, t] * S, b[:, t], x[:, t].unsqueeze(-2))
            y[:, t] = (c[:, t].unsqueeze(-2) @ S).squeeze(-2)
        y = (y + self.w(p + "D").unsqueeze(-1) * x).reshape(B, T, H * e) * _silu(z)
        y = _rms(y.reshape(B, T, R, -1), eps).reshape(B, T, H * e) * self.w(p + "norm")
        return self.mul(y, p + "o")

    def latent_attention(self, n, p, m, eps):
        B, T, _ = n.shape
        H, d, r, e, k = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        q = self.mul(_rms(self.mul(n, p + "dq"), eps) * self.w(p + "dq.norm"), p + "uq").reshape(B, T, H, d + r)
        kv = self.mul(n, p + "dkv")
        lat = _rms(kv[..., :k], eps) * self.w(p + "dkv.norm")
        turned = [_turn(a, m["rot"]["dims"], m["rot"]["base"], pairs=True) for a in (q[..., d:], kv[..., None, k:])]
        keys = self.mul(lat, p + "uk").reshape(B, T, H, d)
        o = _attend(torch.cat([q[..., :d], turned[0]], -1), torch.cat([keys, turned[1].expand(B, T, H, r)], -1),
                    self.mul(lat, p + "uv").reshape(B, T, H, e), lambda s, h: self.softmax(s * m["scale"]))
        return self.mul(o * torch.sigmoid(self.mul(n, p + "g")), p + "o")

    # Pavisun
    def _pavisun(self, tok):
        c, eps = self.c, self.c["norm"]["eps"]
        xs = torch.stack([self.w("embed")[tok]] * c["streams"])
        for i, layer in enumerate(c["layers"]):
            p = f"l{i}."
            mixer = self.turned_attention if layer["type"] == "attention" else self.unit_attention
            for hc, norm, sub in ((p + "hc1.", p + "norm1", lambda n: mixer(n, p + "mix.", layer["mixer"], eps)),
                                  (p + "hc2.", p + "norm2", lambda n: self.experts(n, tok, p + "mlp.", layer["mlp"]))):
                y = sub(_rms(torch.einsum("s,sbtw->btw", self.w(hc + "in"), xs), eps) * self.w(norm))
                xs = torch.einsum("sr,sbtw->rbtw", self.w(hc + "mix"), xs) + self.w(hc + "out").reshape(-1, 1, 1, 1) * y
        return _rms(xs.sum(0), eps) * self.w("final.norm"), "head"

    def turned_attention(self, n, p, m, eps):
        B, T, _ = n.shape
        q, v = (self.mul(n, p + a).reshape(B, T, -1, m["dim"]) for a in "qk")
        rot = m["rot"]
        q, k = (_turn(a, rot["dims"], rot["base"], pairs=False, scaling=rot["scaling"]) for a in (q, v))
        seen = (self.dist >= 0) & (self.dist < m["mask"]["size"])
        cap = m["softcap"]
        o = _attend(q, k, v, lambda s, h: self.softmax(cap * torch.tanh(s * (m["scale"] / cap)), seen))
        return self.mul(o, p + "o")

    def unit_attention(self, n, p, m, eps):
        B, T, _ = n.shape
        H = m["heads"]
        q, k = (_rms(self.mul(n, p + a).reshape(B, T, -1, m["dim"]), eps) for a in "qk")
        v = self.mul(n, p + "v").reshape(B, T, -1, m["vdim"])
        first = torch.arange(T, device="cuda").reshape(1, -1) < m["mask"]["keep_first"]
        seen = (self.dist >= 0) & ((self.dist < m["mask"]["size"]) | first)
        o = _attend(q, k, v, lambda s, h: self.softmax(
            s * m["scale"] - (2.0 ** (-8.0 * (h + 1.0) / H)).double().reshape(-1, 1, 1) * self.dist, seen))
        return self.mul(o * torch.sigmoid(self.mul(n, p + "g")), p + "o")

    def experts(self, n, tok, p, m):
        named = self.w(p + "table")[tok]                         # [B, T, top]
        out = torch.zeros_like(n)
        for e in range(m["router"]["experts"]):
            b, t, _ = torch.nonzero(named == e, as_tuple=True)
            if b.numel():
                out[b, t] += self.ff(n[b, t], f"{p}e{e}.") / m["router"]["top"]
        return out
