"""What a user of this library has it do, as cases that can be timed and checked.

A case is one script of steps through the public entry points: ``Model.from_config`` and
``Model.new_session`` in ``prepare``; ``acquire``, ``step`` and ``release`` (or
``Generator.generate``) in ``run``.  The token ids of every step are given, as in a replay of a
trace, so that the logits of two implementations can be compared place by place; only the
``generate`` cases draw their own tokens, in float32, where draws are reproducible.

The kinds of script:

    serve      all prompts in one step, then ``new`` steps of one token a sequence
    score      whole texts in one step, the logits of every place wanted
    portions   ``batch`` - 1 sequences decode while one prompt comes in portions beside them
    generate   ``Generator.generate`` with the default sampling options

The models are the shapes this repository's own benchmark and tests run.  The designs with routed
experts are left out: in bfloat16 a router's close calls turn on the last bit of a sum, so two
right implementations differ by far more than their arithmetic does.  What they do besides routing
(the products, norms, attention and recurrences) is made of the same kernels.
"""
from __future__ import annotations

import math

import numpy as np
import torch

_QWEN2_7B = {
    "architectures": ["Qwen2ForCausalLM"], "vocab_size": 152064, "hidden_size": 3584,
    "num_hidden_layers": 28, "num_attention_heads": 28, "num_key_value_heads": 4,
    "intermediate_size": 18944, "rope_theta": 1e6, "rms_norm_eps": 1e-6,
    "tie_word_embeddings": False, "use_sliding_window": False, "max_position_embeddings": 32768}
_QWEN2_05B = dict(_QWEN2_7B, vocab_size=151936, hidden_size=896, num_hidden_layers=24,
                  num_attention_heads=14, num_key_value_heads=2, intermediate_size=4864,
                  tie_word_embeddings=True)
_QWEN2_14B = dict(_QWEN2_7B, hidden_size=5120, num_hidden_layers=48, num_attention_heads=40,
                  num_key_value_heads=8, intermediate_size=13824, rms_norm_eps=1e-5)
_QWEN2_TINY = dict(_QWEN2_7B, vocab_size=256, hidden_size=64, num_hidden_layers=2,
                   num_attention_heads=4, num_key_value_heads=1, intermediate_size=128,
                   rope_theta=1e4, tie_word_embeddings=True, max_position_embeddings=128)

# the other designs at width 2,048, as the benchmark runs them
_FURITAR = {
    "architecture": "Furitar", "vocab": 32000, "width": 2048, "max_positions": 8192,
    "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "logit_scale": 1.0,
    "layers": [{"type": "attention", "mlp": {"kind": "dense", "ff": 8448},
                "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128,
                          "scale": 128 ** -0.5 * 4.0, "mask": {"size": 1024}}}] * 8}
_BUDANEX = {
    "architecture": "Budanex", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-5},
    "logit_softcap": 30.0, "loop": {"start": 3, "stop": 6, "times": 2},
    "layers": [
        {"type": "mamba2", "mlp": None,
         "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}},
        {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 5632},
         "mixer": {"heads": 16, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 96,
                   "scale": 96 ** -0.5, "mask": {"size": 1024},
                   "rot": {"base": 500000.0, "dims": 32,
                           "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}},
        {"type": "attention", "mlp": {"kind": "dense", "ff": 5632},
         "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                   "softcap": 50.0, "rot": {"base": 1000000.0, "dims": 64}}}] * 2}
_PAZATAR_ATT = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
_PAZATAR = {
    "architecture": "Pazatar", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "loop": None,
    "layers": [
        {"type": "attention", "mlp": {"kind": "dense", "ff": 8448},
         "mixer": dict(_PAZATAR_ATT, mask={"size": 8192},
                       rot={"base": 500000.0, "dims": 128,
                            "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}})},
        {"type": "parallel", "mlp": {"kind": "dense", "ff": 8448},
         "mixer": {"left": dict(_PAZATAR_ATT, softcap=50.0, conv=4, mask={"size": 1024},
                                rot={"base": 500000.0, "dims": 64,
                                     "scaling": {"factor": 8.0, "original": 8192, "low": 1.0, "high": 4.0}}),
                   "right": {"heads": 8, "dim": 128, "vdim": 256, "tau": 16.0, "decay_rank": 16}}}] * 3}

_MODELS = {"qwen2-tiny": _QWEN2_TINY, "qwen2-0.5b": _QWEN2_05B, "qwen2-7b": _QWEN2_7B,
           "qwen2-14b": _QWEN2_14B, "furitar": _FURITAR, "budanex": _BUDANEX, "pazatar": _PAZATAR}


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def _case(name, kind, model, batch, low, high, new=0, portion=0, dtype="bfloat16"):
    """Prompts of ``low`` to ``high`` tokens (the longest has ``high``)."""
    c = {"kind": kind, "model": model, "dtype": dtype, "batch": batch, "low": low, "high": high,
         "new": new, "portion": portion}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call there is: three short prompts through a toy model, sampled; what
        # counts is the host and the launches
        _case("tiny-generate", "generate", "qwen2-tiny", 3, 5, 13, new=32, dtype="float32"),
        # the 32-bit engine, used to check a model: two texts scored at every place
        _case("0.5b-score-32bit", "score", "qwen2-0.5b", 2, 130, 255, dtype="float32"),
        # one user and a small model: short chat turn, every token waits for the one before
        _case("0.5b-one", "serve", "qwen2-0.5b", 1, 37, 37, new=32),
        # a small model serving many unequal requests
        _case("0.5b-ragged64", "serve", "qwen2-0.5b", 64, 16, 1024, new=24),
        # one user and the headline model: a chat turn
        _case("7b-one", "serve", "qwen2-7b", 1, 333, 333, new=32),
        # the headline: eight sequences at about 2,000 tokens of context
        _case("7b-batch8", "serve", "qwen2-7b", 8, 1801, 2048, new=24),
        # a full batch of short requests
        _case("7b-batch64", "serve", "qwen2-7b", 64, 19, 300, new=16),
        # one long document and a short answer (the largest)
        _case("7b-long", "serve", "qwen2-7b", 1, 20011, 20011, new=8),
        # the largest model: a prompt that comes in portions beside three sequences that decode
        _case("14b-portions", "portions", "qwen2-14b", 4, 700, 3001, portion=512),
        # the other designs: eight prompts of about a thousand tokens and their decoding
        _case("furitar-batch8", "serve", "furitar", 8, 601, 1300, new=24),
        _case("budanex-batch8", "serve", "budanex", 8, 601, 1300, new=24),
        _case("pazatar-batch8", "serve", "pazatar", 8, 601, 1300, new=24),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.99)))))))


def _seconds(case):
    """A rough cost of a case, to keep drawn ones below the largest listed."""
    w = work(case)
    rate = 1.0e15 if case["dtype"] == "bfloat16" else 3.0e13
    return w["flops"] / rate + w["bytes"] / 5e12 + 4e-4 * len(_steps(case))


def draw(rng):
    """Any of the kinds, over batches of 1 to 64 and prompts of 8 to 20,000 tokens."""
    while True:
        kind = rng.choice(["serve"] * 7 + ["portions"] * 2 + ["score", "generate"])
        model = rng.choice(["qwen2-0.5b"] * 3 + ["qwen2-7b"] * 4 + ["qwen2-14b", "furitar", "budanex", "pazatar"])
        dtype, new, portion = "bfloat16", 0, 0
        batch = _log_uniform(rng, 1, 64)
        high = _log_uniform(rng, 8, 20000)
        low = max(4, int(high * rng.choice([1.0, 0.9, 0.5, 0.05])))
        if kind == "serve":
            new = rng.randint(4, 32)
        elif kind == "portions":
            batch, portion = max(2, batch), rng.choice([128, 256, 500, 512, 1024, 2048])
            high = int(portion * rng.uniform(1.2, 12.0))
            low = max(4, high // rng.choice([1, 2, 20]))
        elif kind == "score":
            batch, high = min(batch, 4), min(high, 400)
            low = min(low, high)
            dtype = rng.choice(["bfloat16", "float32"])
            if model.startswith("qwen2") and dtype == "float32":
                model = "qwen2-0.5b"
        else:
            model, dtype, new = "qwen2-tiny", "float32", rng.randint(4, 60)
            batch, high = min(batch, 16), min(high, 64)
            low = min(low, high)
        if model == "furitar" and high + new > 8192:
            continue
        case = _case(None, kind, model, batch, low, high, new, portion, dtype)
        cache = batch * (high + new + 64) * _token_bytes(case)
        if _seconds(case) <= _seconds(_LARGEST) and cache <= 12e9:
            return case


_LARGEST = _case(None, "serve", "qwen2-7b", 1, 20011, 20011, new=8)


# ------------------------------------------------------------------------------------------------
# the steps of a case: [(row, first place, one past the last, wanted places)] each
# ------------------------------------------------------------------------------------------------
def _lengths(case):
    """Prompt lengths, spread evenly over the logarithm of their range; the last is the longest."""
    n, low, high = case["batch"], case["low"], case["high"]
    return [int(round(low * (high / low) ** (((i + 1) * 0.6180339887498949) % 1.0))) for i in range(n - 1)] + [high]


def _steps(case):
    lengths = _lengths(case)
    n = len(lengths)
    if case["kind"] == "score":
        return [[(b, 0, lengths[b], list(range(lengths[b]))) for b in range(n)]]
    if case["kind"] in ("serve", "generate"):
        first = [(b, 0, lengths[b], [lengths[b] - 1]) for b in range(n)]
        return [first] + [[(b, lengths[b] + t, lengths[b] + t + 1, [0]) for b in range(n)]
                          for t in range(case["new"] - (case["kind"] == "generate"))]
    size, last = case["portion"], n - 1
    steps = [[(b, 0, lengths[b], [lengths[b] - 1]) for b in range(last)]]
    for t, at in enumerate(range(0, lengths[last], size)):
        end = min(at + size, lengths[last])
        steps.append([(b, lengths[b] + t, lengths[b] + t + 1, [0]) for b in range(last)]
                     + [(last, at, end, [end - at - 1])])
    return steps


def _totals(case):
    """Tokens of every row over all steps."""
    ends = [0] * case["batch"]
    for step in _steps(case):
        for b, _, end, _ in step:
            ends[b] = max(ends[b], end)
    return ends


def _ids(case, seed):
    cfg = _MODELS[case["model"]]
    rng = np.random.default_rng([int(seed), 7])
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    return [rng.integers(0, vocab, n).tolist() for n in _totals(case)]


def _model(case, seed):
    from minfer_b200 import Model
    # the wide models' weights are drawn smaller than the default of 0.02: a product's gain
    # (std * sqrt(width)) then stays below 1, as a trained model's does, and rounding errors are
    # not amplified from layer to layer
    std = {"qwen2-7b": 0.01, "qwen2-14b": 0.008}.get(case["model"])
    return Model.from_config(_MODELS[case["model"]], seed=int(seed), dtype=case["dtype"], device="cuda:0",
                             norm_std=0.05, make_on="device", weight_std=std)


# ------------------------------------------------------------------------------------------------
# what is measured
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """A loaded model with its session (or generator) and the requests' token ids on the host."""
    model, ids = _model(case, seed), _ids(case, seed)
    if case["kind"] == "generate":
        from minfer_b200 import Generator, SamplingParams
        room = sum(-(-(n + case["new"]) // 64) * 64 for n in _lengths(case))
        return {"generator": Generator(model, max_tokens=room, max_batch=case["batch"]),
                "prompts": [row[:n] for row, n in zip(ids, _lengths(case))], "new": case["new"],
                "sampling": SamplingParams(seed=int(seed))}
    session = model.new_session(max_seqs=case["batch"], max_positions=-(-max(_totals(case)) // 64) * 64)
    script = [([b for b, _, _, _ in step], [ids[b][at:end] for b, at, end, _ in step],
               [want for _, _, _, want in step]) for step in _steps(case)]
    return {"session": session, "script": script, "rows": case["batch"]}


def run(state):
    """One script from fresh slots to released ones; the logits of every step."""
    if "generator" in state:
        out = state["generator"].generate(state["prompts"], state["new"], state["sampling"], stop_token_ids=[])
        return [torch.tensor(r.tokens) for r in out]
    session = state["session"]
    slots = [session.acquire() for _ in range(state["rows"])]
    logits = [session.step([slots[b] for b in rows], tokens, want) for rows, tokens, want in state["script"]]
    for s in slots:
        session.release(s)
    return logits


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _runs(cfg):
    """The layers in the order in which they run."""
    loop, layers = cfg.get("loop"), cfg["layers"]
    if not loop:
        return list(range(len(layers)))
    return (list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"]
            + list(range(loop["stop"], len(layers))))


def _layer_costs(name):
    """Per layer run: (numbers in matrices, [(numbers read per visible key, flops per visible pair,
    span, by window)], recurrent state's numbers and its flops a token)."""
    cfg = _MODELS[name]
    if name.startswith("qwen2"):
        w, heads, kv = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        d = w // heads
        numbers = 2 * w * w + 2 * w * kv * d + 3 * w * cfg["intermediate_size"]
        return [(numbers, [(2 * kv * d, 4 * heads * d, 0, False)], 0, 0)] * cfg["num_hidden_layers"]
    out = []
    for i in _runs(cfg):
        layer, w = cfg["layers"][i], cfg["width"]
        m, ff = layer["mixer"], (layer["mlp"] or {"ff": 0})["ff"]
        numbers, reads, state, per_token = (3 if name == "budanex" else 2) * w * ff, [], 0, 0
        if layer["type"] == "mamba2":
            inner = m["heads"] * m["vdim"]
            numbers += w * (2 * inner + 2 * m["groups"] * m["state"] + m["heads"]) + inner * w
            state = inner * m["state"]
            per_token = 5 * state
        elif layer["type"] == "latent_attention":
            rank, wide = m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"])
            numbers += w * (wide + rank + 2 * m["heads"] * m["vdim"]) + m["heads"] * (m["dim"] + m["vdim"]) * m["kv_rank"]
            reads.append((rank, 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["mask"]["size"], True))
        else:
            a = m.get("left", m)
            shared = name == "pazatar" and layer["type"] == "attention"     # values are the keys
            q, k = a["heads"] * a["dim"], a["kv_heads"] * a["dim"]
            numbers += w * (2 * q + (1 if shared else 2) * k)
            reads.append(((1 if shared else 2) * k, 4 * q, (a.get("mask") or {"size": 0})["size"], False))
            if "right" in m:
                r = m["right"]
                nk, nv = r["heads"] * r["dim"], r["heads"] * r["vdim"]
                numbers += w * (2 * nk + 3 * nv + r["decay_rank"]) + nk * r["decay_rank"]
                state = r["heads"] * r["dim"] * r["vdim"]
                per_token = 5 * state
        out.append((numbers, reads, state, per_token))
    return out


def _pairs(at, end, span, window):
    """(visible keys of all queries together, distinct keys they see) for queries at..end-1."""
    if not span:
        return (at + 1 + end) * (end - at) / 2, end
    p = np.arange(at, end)
    seen = np.minimum(p + 1, span) if window else p % span + 1
    first = max(0, at - span + 1) if window else at - at % span
    return float(seen.sum()), end - first


def _token_bytes(case):
    """Cached bytes of a token over all layers."""
    size = 2 if case["dtype"] == "bfloat16" else 4
    return sum(r[0] for _, reads, _, _ in _layer_costs(case["model"]) for r in reads) * size


def work(case):
    """Per step: every matrix read once, a key read once for each sequence that sees it, states read
    and written, new keys and the logits written; a recurrent state in 32 bits."""
    cfg, layers = _MODELS[case["model"]], _layer_costs(case["model"])
    size = 2 if case["dtype"] == "bfloat16" else 4
    w, vocab = cfg.get("hidden_size") or cfg["width"], cfg.get("vocab_size") or cfg["vocab"]
    # a looped layer's weights are read on each pass: the layers between do not fit the chip
    numbers = sum(layer[0] for layer in layers)
    total_bytes = total_flops = 0.0
    for step in _steps(case):
        tokens = sum(end - at for _, at, end, _ in step)
        wanted = sum(len(want) for _, _, _, want in step)
        total_bytes += (numbers + w * vocab) * size + tokens * (w * size + 4) + wanted * vocab * 4
        total_flops += 2.0 * numbers * tokens + 2.0 * w * vocab * wanted
        for _, at, end, _ in step:
            for _, reads, state, per_token in layers:
                total_bytes += 2 * 4 * state
                total_flops += per_token * (end - at)
                for per_key, per_pair, span, window in reads:
                    pairs, keys = _pairs(at, end, span, window)
                    total_bytes += per_key * size * (keys if at else end)
                    total_flops += per_pair * pairs
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if case["kind"] == "generate":
        return {"rel": 0.0, "differ": 0.01}
    # measured against ``exact``: 3.5e-6 in 32 bits, 0.005 to 0.01 in bfloat16; about four times that
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 1.5e-4}
    return {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits: the designs' equations in plain torch, all sequences' tokens side by side
# ------------------------------------------------------------------------------------------------
class _Plain:
    """Sequences of tokens laid end to end, a model's weights by name, and the equations."""

    def __init__(self, weights, eps, lengths):
        self.w, self.eps, self.lengths = weights, eps, lengths
        self.spans, at = [], 0
        for n in lengths:
            self.spans.append((at, at + n))
            at += n
        self.places = torch.cat([torch.arange(n, device="cuda", dtype=torch.float64) for n in lengths])

    def __getitem__(self, name):
        return self.w[name].to("cuda", torch.float64)

    def times(self, x, name, bias=None):
        y = x @ self[name].T
        return y if bias is None else y + self[bias]

    def unit(self, x):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + self.eps)

    def norm(self, x, name):
        return self.unit(x) * self[name]

    def padded(self, x):
        """[tokens, ..] -> [sequences, longest, ..], zeros behind the shorter ones."""
        out = x.new_zeros((len(self.lengths), max(self.lengths)) + x.shape[1:])
        for b, (lo, hi) in enumerate(self.spans):
            out[b, :hi - lo] = x[lo:hi]
        return out

    def packed(self, x):
        return torch.cat([x[b, :n] for b, n in enumerate(self.lengths)])

    def before(self, x, steps):
        """Every token's predecessor ``steps`` places earlier, zeros before the start."""
        out = torch.zeros_like(x)
        for lo, hi in self.spans:
            out[lo + steps:hi] = x[lo:hi - steps] if hi - lo > steps else x[lo:lo]
        return out

    def conv(self, x, name):
        taps = self[name]
        n = taps.shape[1]
        return sum((x if j == n - 1 else self.before(x, n - 1 - j)) * taps[:, j] for j in range(n))

    def turn(self, x, freqs, halves=True, magnitude=1.0):
        """Rotates the first 2 len(freqs) numbers of every head: pairs (i, i + half) or (2i, 2i + 1)."""
        n = len(freqs)
        ang = self.places[:, None] * torch.tensor(freqs, device="cuda", dtype=torch.float64)
        c, s = magnitude * torch.cos(ang)[:, None], magnitude * torch.sin(ang)[:, None]
        out = x.clone()
        i0, i1 = (slice(0, n), slice(n, 2 * n)) if halves else (slice(0, 2 * n, 2), slice(1, 2 * n, 2))
        out[..., i0] = x[..., i0] * c - x[..., i1] * s
        out[..., i1] = x[..., i1] * c + x[..., i0] * s
        return out

    def attend(self, q, k, v, scale, window=0, chunk=0, softcap=0.0, sink=None, distance=None):
        """q [tokens, H, D], k and v [tokens, G, ..]; ``sink`` [H]: scores without a value;
        ``distance`` (r1, r2) [H]: a score falls by r1 ln(1 + r2 (i - j))."""
        heads, groups = q.shape[1], k.shape[1]
        out = q.new_empty(q.shape[0], heads, v.shape[2])
        for lo, hi in self.spans:
            kk, vv = k[lo:hi].movedim(1, 0), v[lo:hi].movedim(1, 0)              # [G, T, ..]
            block = max(1, min(2048, int(1.5e8 / (heads * (hi - lo)))))
            for a in range(0, hi - lo, block):
                b = min(a + block, hi - lo)
                first = max(0, a - window + 1) if window else (a - a % chunk if chunk else 0)
                qq = q[lo + a:lo + b].view(b - a, groups, heads // groups, -1).permute(1, 2, 0, 3)
                s = torch.einsum("gpqd,gkd->gpqk", qq, kk[:, first:b]) * scale
                gap = torch.arange(a, b, device="cuda")[:, None] - torch.arange(first, b, device="cuda")
                if softcap:
                    s = softcap * torch.tanh(s / softcap)
                if distance is not None:
                    r1, r2 = (r.view(groups, -1, 1, 1) for r in distance)
                    s = s - r1 * torch.log1p(r2 * gap.clamp(min=0))
                hidden = gap < 0
                if window:
                    hidden |= gap >= window
                if chunk:
                    hidden |= (torch.arange(a, b, device="cuda")[:, None] // chunk
                               != torch.arange(first, b, device="cuda") // chunk)
                s = s.masked_fill_(hidden, -math.inf)
                if sink is not None:
                    s = torch.cat([s, sink.view(groups, -1, 1, 1).expand(-1, -1, b - a, 1)], -1)
                p = torch.softmax(s, -1)
                o = torch.einsum("gpqk,gkd->gpqd", p[..., :b - first], vv[:, first:b])
                out[lo + a:lo + b] = o.permute(2, 0, 1, 3).reshape(b - a, heads, -1)
        return out


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.clamp(x, min=0) + torch.log1p(torch.exp(-x.abs()))


def _frequencies(rot):
    return [rot["base"] ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)]


def _yarn(rot):
    f, dims, base = rot["scaling"], rot["dims"], rot["base"]
    at = [dims * math.log(f["original"] / (2 * math.pi * f[n])) / (2 * math.log(base)) for n in ("fast", "slow")]
    lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return ([x / f["factor"] * r + x * (1 - r) for x, r in zip(_frequencies(rot), ramp)],
            0.1 * math.log(f["factor"]) + 1.0)


def _banded(rot):
    f, out = rot["scaling"], []
    for x in _frequencies(rot):
        turns = f["original"] * x / (2 * math.pi)
        s = min(max((turns - f["low"]) / (f["high"] - f["low"]), 0.0), 1.0)
        out.append((1 - s) * x / f["factor"] + s * x)
    return out


def _plain_qwen2(cfg, m, ids):
    heads, kv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    d = cfg["hidden_size"] // heads
    freqs = _frequencies({"base": cfg["rope_theta"], "dims": d})
    x = m["model.embed_tokens.weight"][ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        y = m.norm(x, p + "input_layernorm.weight")
        q, k, v = (m.times(y, f"{p}self_attn.{n}_proj.weight", f"{p}self_attn.{n}_proj.bias").view(len(ids), h, d)
                   for n, h in (("q", heads), ("k", kv), ("v", kv)))
        o = m.attend(m.turn(q, freqs), m.turn(k, freqs), v, d ** -0.5)
        x = x + m.times(o.reshape(len(ids), -1), p + "self_attn.o_proj.weight")
        y = m.norm(x, p + "post_attention_layernorm.weight")
        y = _silu(m.times(y, p + "mlp.gate_proj.weight")) * m.times(y, p + "mlp.up_proj.weight")
        x = x + m.times(y, p + "mlp.down_proj.weight")
    head = "model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"
    return lambda rows: m.times(m.norm(x[rows], "model.norm.weight"), head)


def _plain_furitar(cfg, m, ids):
    x = m["embed"][ids] * cfg["embedding"]["scale"] + m["pos"][m.places.long()]
    for i, layer in enumerate(cfg["layers"]):
        p, a = f"l{i}.", layer["mixer"]
        h = m.norm(x, p + "norm1")
        u = h + (m.before(h, 1) - h) * m[p + "shift"]
        q, k, v = (m.times(u, f"{p}mix.{n}").view(len(ids), g, d)
                   for n, g, d in (("q", a["heads"], a["dim"]), ("k", a["kv_heads"], a["dim"]),
                                   ("v", a["kv_heads"], a["vdim"])))
        o = m.attend(m.unit(q), m.unit(k), v, a["scale"], chunk=a["mask"]["size"],
                     sink=torch.zeros(a["heads"], device="cuda", dtype=torch.float64),
                     distance=(m[p + "mix.r1"], m[p + "mix.r2"]))
        x = x + m.times(o.reshape(len(ids), -1), p + "mix.o")
        z, (up, down) = m.times(m.norm(x, p + "norm2"), p + "mlp.up"), _softplus(m[p + "mlp.act"])
        z = torch.where(z > 0, up * z * z, (0.5 + down) * (torch.expm1(z.clamp(max=0)) - z)) + 0.5 * z
        x = x + m.times(z, p + "mlp.down")
    return lambda rows: m.times(m.norm(x[rows], "final.norm"), "head") * cfg["logit_scale"]


def _mamba2(m, u, p, a):
    heads, wide, n, groups = a["heads"], a["vdim"], a["state"], a["groups"]
    inner = heads * wide
    z, xbc, dt = m.times(u, p + "in").split([inner, inner + 2 * groups * n, heads], -1)
    xbc = _silu(m.conv(xbc, p + "conv") + m[p + "conv.b"])
    dt = _softplus(dt + m[p + "dt_bias"])
    x, b, c = xbc.split([inner, groups * n, groups * n], -1)
    x = x.view(-1, heads, wide)
    b, c = (m.padded(t.view(-1, groups, n).repeat_interleave(heads // groups, 1)) for t in (b, c))
    keep, add = m.padded(torch.exp(-torch.exp(m[p + "A_log"]) * dt)), m.padded(dt[..., None] * x)
    state, out = x.new_zeros(len(m.lengths), heads, n, wide), torch.empty_like(add)
    for t in range(add.shape[1]):
        state = keep[:, t, :, None, None] * state + b[:, t, :, :, None] * add[:, t, :, None, :]
        out[:, t] = torch.einsum("bhnp,bhn->bhp", state, c[:, t])
    y = (m.packed(out) + m[p + "D"][:, None] * x).reshape(-1, inner) * _silu(z)
    y = m.unit(y.view(-1, a["norm_groups"], inner // a["norm_groups"])).reshape(-1, inner)
    return m.times(y * m[p + "norm"], p + "o")


def _latent_attention(m, u, p, a):
    heads, d, rank = a["heads"], a["dim"], a["kv_rank"]
    q, ckr = m.times(u, p + "q").view(-1, heads, d + a["rot_dim"]), m.times(u, p + "dkv")
    c = m.norm(ckr[:, :rank], p + "dkv.norm")
    freqs, magnitude = _yarn(a["rot"])
    kr = m.turn(ckr[:, None, rank:], freqs, False, magnitude).expand(-1, heads, -1)
    q = torch.cat([q[..., :d], m.turn(q[..., d:], freqs, False, magnitude)], -1)
    k = torch.cat([m.times(c, p + "uk").view(-1, heads, d), kr], -1)
    o = m.attend(q, k, m.times(c, p + "uv").view(-1, heads, a["vdim"]), a["scale"],
                 window=a["mask"]["size"], sink=m[p + "sink"])
    return m.times(o.reshape(len(u), -1) * torch.sigmoid(m.times(u, p + "g")), p + "o")


def _capped_attention(m, u, p, a):
    q, k = (m.norm(m.times(u, p + n, p + n + ".b"), p + n + ".norm").view(len(u), -1, a["dim"]) for n in "qk")
    v = m.times(u, p + "v", p + "v.b").view(len(u), -1, a["vdim"])
    freqs = _frequencies(a["rot"])
    o = m.attend(m.turn(q, freqs), m.turn(k, freqs), v, a["scale"], softcap=a["softcap"])
    return m.times(o.reshape(len(u), -1), p + "o")


def _plain_budanex(cfg, m, ids):
    mixers = {"mamba2": _mamba2, "latent_attention": _latent_attention, "attention": _capped_attention}
    x = start = m.norm(m["embed"][ids], "embed.norm")
    passes = 0
    for i in _runs(cfg):
        if i == cfg["loop"]["start"]:
            x = x + (start if passes else 0.0) + m["loop.step"][passes]
            passes += 1
        p, layer = f"l{i}.", cfg["layers"][i]
        x = x + mixers[layer["type"]](m, m.norm(x, p + "norm1"), p + "mix.", layer["mixer"])
        if layer["mlp"] is not None:
            y = m.norm(x, p + "norm2")
            y = torch.nn.functional.gelu(m.times(y, p + "mlp.gate"), approximate="tanh") * m.times(y, p + "mlp.up")
            x = x + m.times(y, p + "mlp.down")
    cap = cfg["logit_softcap"]
    return lambda rows: cap * torch.tanh(m.times(m.norm(x[rows], "final.norm"), "head") / cap)


def _gated_linear(m, y, p, a):
    heads, d = a["heads"], a["dim"]
    z = m.times(m.times(y, p + "a1"), p + "a2", p + "a2.b")
    keep = m.padded(torch.exp(-_softplus(-z) / a["tau"]).view(-1, heads, d))
    q = m.padded(m.times(y, p + "q").view(-1, heads, d) * d ** -0.5)
    k, v = m.padded(m.times(y, p + "k").view(-1, heads, d)), m.padded(m.times(y, p + "v").view(-1, heads, a["vdim"]))
    state, out = y.new_zeros(len(m.lengths), heads, d, a["vdim"]), torch.empty_like(v)
    for t in range(v.shape[1]):
        state = keep[:, t, :, :, None] * state + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = torch.einsum("bhd,bhdj->bhj", q[:, t], state)
    o = m.norm(m.packed(out), p + "norm").reshape(len(y), -1)
    return m.times(o * _silu(m.times(y, p + "g")), p + "o")


def _conv_attention(m, y, p, a):
    q, k, v = (m.conv(m.times(y, p + n), f"{p}{n}.conv").view(len(y), -1, a["dim"]) for n in "qkv")
    freqs = _banded(a["rot"])
    q, k = m.turn(m.norm(q, p + "q.norm"), freqs), m.turn(m.norm(k, p + "k.norm"), freqs)
    o = m.attend(q, k, v, a["scale"], chunk=a["mask"]["size"], softcap=a["softcap"],
                 sink=torch.zeros(a["heads"], device="cuda", dtype=torch.float64))
    return m.times(o.reshape(len(y), -1), p + "o")


def _keys_as_values(m, y, p, a):
    k = m.times(y, p + "k")
    v = k.view(len(y), -1, a["dim"])
    freqs, magnitude = _yarn(a["rot"])
    q, k = (m.turn(m.norm(t, p + n).view(len(y), -1, a["dim"]), freqs, False, magnitude)
            for t, n in ((m.times(y, p + "q"), "q.norm"), (k, "k.norm")))
    return m.times(m.attend(q, k, v, a["scale"], chunk=a["mask"]["size"]).reshape(len(y), -1), p + "o")


def _plain_pazatar(cfg, m, ids):
    x = m["embed"][ids]
    for i in _runs(cfg):
        p, a = f"l{i}.", cfg["layers"][i]["mixer"]
        y = m.norm(x, p + "norm1")
        if "right" in a:
            y = 0.5 * (m.norm(_conv_attention(m, y, p + "mix.left.", a["left"]), p + "mix.left.out")
                       + m.norm(_gated_linear(m, y, p + "mix.right.", a["right"]), p + "mix.right.out"))
        else:
            y = _keys_as_values(m, y, p + "mix.", a)
        x = x + m.norm(y, p + "norm1b")
        y = torch.clamp(m.times(m.norm(x, p + "norm2"), p + "mlp.up"), min=0) ** 2
        x = x + m.norm(m.times(y, p + "mlp.down"), p + "norm2b")
    return lambda rows: m.times(m.norm(x[rows], "final.norm"), "embed")


def exact(case, seed):
    """``run``'s logits by the designs' equations; the weights are the model's own numbers."""
    if case["kind"] == "generate" or work(case)["flops"] > 4e14:      # drawn tokens; over 20 seconds
        return None
    cfg, lengths = _MODELS[case["model"]], _totals(case)
    plain = {"furitar": _plain_furitar, "budanex": _plain_budanex,
             "pazatar": _plain_pazatar}.get(case["model"], _plain_qwen2)
    eps = cfg["rms_norm_eps"] if "rms_norm_eps" in cfg else cfg["norm"]["eps"]
    m = _Plain(_model(case, seed).export_state_dict(), eps, lengths)
    ids = torch.tensor([t for row in _ids(case, seed) for t in row], device="cuda")
    with torch.no_grad():
        logits = plain(cfg, m, ids)
        return [logits(torch.tensor([m.spans[b][0] + at + place for b, at, _, want in step for place in want],
                                    device="cuda")) for step in _steps(case)]
