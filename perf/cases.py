"""Cases of real use whose time is measured, with their inputs, their work and what they return in 64 bits.

A case is one pass of a loaded model: a prompt step (whole prompts, or a long prompt in portions; the logits behind each
prompt come back) or a single-token step of a batch of sequences (each one's logits come back), through ``Runner.step``
as a server's loop calls it.  Weights are random with the sizes of the configurations in ``rustyllm_b200/configs`` and
``rustyllm_b200/bench_designs.py``.

``exact`` is a plain statement of the models in float64: whole sequences, no cache, weights drawn by the rule that random
weights are defined by (twelve uniform 16-bit integers from splitmix64 over a counter, seeded by seed and tensor name).
"""
import json
import math
import os
import zlib

import torch

import rustyllm_b200
from rustyllm_b200 import Runner
from rustyllm_b200.bench_designs import SIZES, forilorn_config, mogutar_config, mosurax_config

DEV = "cuda:0"
F64 = torch.float64
PAGE = 64
GROW = 2048        # single tokens a sequence may gain before its context starts over
# Most tokens of one prompt, and of all prompts of a pass, that are asked of a model
MOST_PROMPT = {"llama31_8b": 2048, "llama32_1b": 8192, "llama32_1b float32": 512, "mosurax": 2048, "mogutar": 2048, "forilorn": 2048}
# Most sequences in a batch of single tokens, and the longest context there
MOST_BATCH = {"llama31_8b": 8, "llama32_1b": 64, "llama32_1b float32": 8, "mosurax": 64, "mogutar": 32, "forilorn": 64}
MOST_CONTEXT = {"llama31_8b": 2048, "llama32_1b": 2048, "llama32_1b float32": 700, "mosurax": 1536, "mogutar": 1024, "forilorn": 1536}


def _case(name, model, kind, seqs, shortest, longest, dtype="bfloat16", portion=0):
    """``seqs`` sequences whose lengths spread evenly over the logarithm from ``shortest`` to ``longest`` tokens: prompts
    (``kind`` "prompt"; ``portion``: at most so many tokens of each a step, 0: all) or contexts that one more token is
    fed to ("decode")."""
    c = {"model": model, "dtype": dtype, "kind": kind, "seqs": seqs, "shortest": shortest, "longest": longest, "portion": portion}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user at a small model, right behind a short question: the smallest call, a chain of launches
        _case("1b-decode-1", "llama32_1b", "decode", 1, 131, 131),
        # the headline: eight users of an 8B model at contexts of every length
        _case("8b-decode-8", "llama31_8b", "decode", 8, 128, 2047),
        # a full batch of a small model: the cache is as large as the weights
        _case("1b-decode-64", "llama32_1b", "decode", 64, 256, 2047),
        # a document as a prompt, an 8B model
        _case("8b-prompt-2048", "llama31_8b", "prompt", 1, 2048, 2048),
        # a chat turn as a prompt
        _case("8b-prompt-293", "llama31_8b", "prompt", 1, 293, 293),
        # requests of every length that came in together
        _case("1b-16-prompts", "llama32_1b", "prompt", 16, 33, 1201),
        # a long document taken in portions, so that a step's memory stays bounded
        _case("1b-8000-in-portions", "llama32_1b", "prompt", 1, 8000, 8000, portion=3000),
        # the 32-bit path, both directions
        _case("1b-float32-prompt-500", "llama32_1b", "prompt", 1, 500, 500, dtype="float32"),
        _case("1b-float32-decode-4", "llama32_1b", "decode", 4, 96, 700, dtype="float32"),
        # the other designs by what they are made of: experts, and attention with a sink and a gate,
        _case("mosurax-decode-48", "mosurax", "decode", 48, 160, 1500),
        # recurrences with a matrix state (and experts, filters, a window),
        _case("mogutar-prompt-1500", "mogutar", "prompt", 1, 1500, 1500),
        # attention through a latent (and a chunked mask, a hashed pair table)
        _case("forilorn-2-prompts", "forilorn", "prompt", 2, 600, 1400),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    key = rng.choice(["llama31_8b", "llama32_1b", "llama32_1b", "llama32_1b float32", "mosurax", "mogutar", "forilorn"])
    model, _, dtype = key.partition(" ")
    dtype = dtype or "bfloat16"
    if rng.random() < 0.5:
        seqs = _log_int(rng, 1, MOST_BATCH[key])
        a, b = sorted(_log_int(rng, 16, MOST_CONTEXT[key]) for _ in range(2))
        return _case(None, model, "decode", seqs, b if seqs == 1 else a, b, dtype)
    seqs = _log_int(rng, 1, 12)
    b = _log_int(rng, 17 * seqs, MOST_PROMPT[key]) // seqs
    a = b if seqs == 1 else _log_int(rng, max(9, b // 8), b)
    portion = _log_int(rng, max(16, b // 4), b) if rng.random() < 0.25 else 0
    return _case(None, model, "prompt", seqs, a, b, dtype, portion)


# --------------------------------------------------------------------------------------------- inputs
def _config(model):
    if model.startswith("llama"):
        with open(os.path.join(os.path.dirname(rustyllm_b200.__file__), "configs", model + ".json")) as f:
            return json.load(f)
    s = SIZES["w2048"]
    if model == "mogutar":
        cfg = mogutar_config(s)
        for layer in cfg["layers"]:        # every token takes all of four experts: behind layers that norm what they add and carry
            layer["mlp"]["router"] = {"experts": 4, "top": 4}        # a state, one close choice would change every later token
        return cfg
    return mosurax_config(s, True) if model == "mosurax" else forilorn_config(s)


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _lengths(case):
    n, a, b = case["seqs"], case["shortest"], case["longest"]
    if n == 1:
        return [b]
    lens = [int(round(a * (b / a) ** (i / (n - 1)))) for i in range(n)]
    return lens[::2] + lens[1::2][::-1]        # neither sorted nor all long ones at one end


def _tokens(case, seed):
    """The sequences' tokens and, for single tokens, what is fed next, in turn."""
    g = torch.Generator().manual_seed(seed)
    V = _vocab(_config(case["model"]))
    prompts = [torch.randint(0, V, (n,), generator=g).tolist() for n in _lengths(case)]
    fed = torch.randint(0, V, (32, case["seqs"], 1), generator=g).tolist() if case["kind"] == "decode" else []
    return prompts, fed


def _begin(state):
    """The sequences' contexts into the cache, in steps of up to 8,192 tokens."""
    r = state["runner"]
    for s in state["slots"]:
        r.engine.free_slot(s)
    state["slots"] = [r.engine.alloc_slot() for _ in state["prompts"]]
    at, state["fed_at"] = 0, 0
    while at < len(state["slots"]):
        n, end = 0, at
        while end < len(state["slots"]) and (end == at or n + len(state["prompts"][end]) <= 8192):
            n += len(state["prompts"][end])
            end += 1
        r.step(state["slots"][at:end], state["prompts"][at:end], None)
        at = end
    state["length"] = max(len(p) for p in state["prompts"])
    state["limit"] = state["length"] + GROW


def prepare(case, seed):
    cfg = _config(case["model"])
    prompts, fed = _tokens(case, seed)
    n, grow = case["seqs"], GROW if case["kind"] == "decode" else 0
    room = sum(-(-(len(p) + grow + 1) // PAGE) * PAGE for p in prompts)
    runner = Runner.from_config(cfg, seed=seed, dtype=case["dtype"], device=DEV, norm_noise=True, max_batch=n, max_cache_tokens=room)
    state = {"runner": runner, "kind": case["kind"], "portion": case["portion"], "prompts": prompts, "fed": fed, "slots": []}
    if case["kind"] == "decode":
        runner.warm_up([n])
        _begin(state)
    return state


def run(state):
    r = state["runner"]
    if state["kind"] == "decode":
        if state["length"] >= state["limit"]:
            _begin(state)
        fed = state["fed"][state["fed_at"] % len(state["fed"])]
        state["fed_at"] += 1
        state["length"] += 1
        return r.step(state["slots"], fed, "last")
    prompts, portion = state["prompts"], state["portion"]
    slots = [r.engine.alloc_slot() for _ in prompts]
    if portion:
        logits = {}
        for at in range(0, max(len(p) for p in prompts), portion):
            live = [i for i, p in enumerate(prompts) if len(p) > at]
            last = [i for i in live if len(prompts[i]) <= at + portion]
            want = [[len(prompts[i]) - at - 1] if i in last else [] for i in live]
            rows = r.step([slots[i] for i in live], [prompts[i][at:at + portion] for i in live], want if last else None)
            logits.update({i: rows[k] for k, i in enumerate(last)})
        out = torch.stack([logits[i] for i in range(len(prompts))])
    else:
        out = r.step(slots, prompts, "last")
    for s in slots:
        r.engine.free_slot(s)
    return out


# --------------------------------------------------------------------------------------------- work
def _expert_share(experts, top, tokens):
    """Share of the experts that some token chooses, if the choices are even."""
    return 1.0 - (1.0 - top / experts) ** tokens


def work(case):
    """Bytes: every weight that the pass uses once, the cache or state it reads and writes once, the logits.  Operations:
    two a multiply-add of the products (each token's own experts), of the visible scores and weighted values, and of the
    recurrences."""
    cfg, lens = _config(case["model"]), _lengths(case)
    size = 4 if case["dtype"] == "float32" else 2
    decode = case["kind"] == "decode"
    T = len(lens) if decode else sum(lens)
    V, n = _vocab(cfg), len(lens)

    def pairs(limit=None):        # visible (query, key) pairs of all sequences
        total = 0
        for L in lens:
            if decode:
                total += min(L + 1, limit or L + 1)
            else:
                w = min(L, limit or L)
                total += w * (w + 1) // 2 + (L - w) * w
        return total

    def cached(per, limit=None):        # bytes of cached rows read (single tokens) and written
        return size * per * ((sum(min(L, limit or L) for L in lens) if decode else 0) + T)
    nbytes, flops = 0.0, 0.0

    def product(k, m, rows=None, used=1.0):
        nonlocal nbytes, flops
        nbytes += size * k * m * used
        flops += 2.0 * (T if rows is None else rows) * k * m
    if "num_hidden_layers" in cfg:
        d, I, H, G, hd = (cfg[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
        for _ in range(cfg["num_hidden_layers"]):
            product(d, (H + 2 * G) * hd)
            product(H * hd, d)
            product(d, 2 * I)
            product(I, d)
            flops += 4.0 * H * hd * pairs()
            nbytes += cached(2 * G * hd)
    else:
        d = cfg["width"]
        for layer in cfg["layers"]:
            m, mlp = layer["mixer"], layer.get("mlp")
            if layer["type"] in ("attention", "parallel"):
                a = m["left"] if layer["type"] == "parallel" else m
                H, G, hd = a["heads"], a["kv_heads"], a["dim"]
                gate, own = (H * hd, 1) if case["model"] == "forilorn" else (H * hd if case["model"] == "mosurax" else 0, 2)
                product(d, (H + own * G) * hd + gate)
                product(H * hd, d)
                window = (a.get("mask") or {}).get("size")
                flops += 4.0 * H * hd * pairs(window)
                nbytes += cached(2 * G * hd, window)
            if layer["type"] == "parallel":
                s = m["right"]
                inner, N, gr = s["heads"] * s["vdim"], s["state"], s["groups"]
                product(d, 2 * inner + 2 * gr * N + s["heads"])
                product(inner, d)
                flops += 4.0 * T * inner * N
                nbytes += n * 4 * inner * N * (2 if decode else 1)
            if layer["type"] == "lightning":
                H, dk, dv = m["heads"], m["dim"], m["vdim"]
                product(d, 2 * H * (dk + dv))
                product(H * dv, d)
                flops += 4.0 * T * H * dk * dv
                nbytes += n * 4 * H * dk * dv * (2 if decode else 1)
            if layer["type"] == "latent_attention":
                H, hd, rd, vd, r, qr = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
                product(d, qr + r + rd + H)
                product(qr, H * (hd + rd))
                product(r, H * (hd + vd))
                product(H * vd, d)
                flops += 2.0 * H * (hd + rd + vd) * pairs(m["mask"]["size"])
                nbytes += cached(r + rd, m["mask"]["size"])
            if mlp is not None and mlp["kind"] == "dense":
                product(d, mlp["ff"] * (1 if case["model"] == "forilorn" else 2))
                product(mlp["ff"], d)
            elif mlp is not None:
                E, top, ff = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
                product(d, E)
                product(d, 3 * ff * E, rows=T * top / E, used=_expert_share(E, top, T))
                if mlp.get("shared"):
                    product(d, 3 * mlp["shared"]["ff"])
            if "token_side" in cfg:
                product(d, 2 * cfg["token_side"]["dim"])
    product(d, V, rows=n)
    nbytes += 4.0 * n * V + size * T * d
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # four times the distance from ``exact``: 32-bit sums 1e-5, bfloat16 activations 0.004 (forilorn, 8 layers) to 0.05 (32 layers;
    # mosurax, where single tokens take another expert at a close call), where 0.03 is stated
    if case["dtype"] == "float32":
        return {"rel": 4e-5, "max": 1e-3}
    return {"rel": 1.6e-2 if case["model"] == "forilorn" else 3e-2, "max": 0.9}


# --------------------------------------------------------------------------------------------- in 64 bits
def _mix64(z):
    """splitmix64's output for the counter values ``z`` (int64 that wraps)."""
    def right(x, n):
        return (x >> n) & ((1 << (64 - n)) - 1)
    z = z + (0x9E3779B97F4A7C15 - (1 << 64))
    z = (z ^ right(z, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ right(z, 27)) * (0x94D049BB133111EB - (1 << 64))
    return z ^ right(z, 31)


class _Weights:
    """Tensors of a random model, in float64 on the GPU, drawn when asked for."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = seed, torch.float32 if dtype == "float32" else torch.bfloat16

    def __call__(self, name, *shape, mean=0.0):
        seed = (self.seed * 0x9E3779B97F4A7C15 + zlib.crc32(name.encode("utf-8")) * 0x100000001B3 + 0x1234567) % (1 << 63)
        n = math.prod(shape)
        out = torch.empty(n, dtype=F64, device=DEV)
        step = torch.tensor(0.02, dtype=torch.float32) * 2.0 ** -16
        for at in range(0, n, 1 << 24):
            i = torch.arange(at, min(n, at + (1 << 24)), dtype=torch.int64, device=DEV)
            total = torch.zeros_like(i)
            for r in range(3):
                h = _mix64(i * 3 + (seed + r))
                for shift in (0, 16, 32, 48):
                    total += (h >> shift) & 0xFFFF
            z = (total - 393210).to(torch.float32)
            out[at:at + i.numel()] = (z * step.item() + mean).to(self.dtype).to(F64)
        return out.view(*shape)


def _rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)
    return y if w is None else y * w


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _plain_freqs(dims, base):
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64)


def _llama3_freqs(dims, base, s):
    f = _plain_freqs(dims, base)
    if s:
        turns = s["original_max_position_embeddings"] * f / (2.0 * math.pi)
        blend = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0.0, 1.0)
        f = (1.0 - blend) * f / s["factor"] + blend * f
    return f


def _stretched_freqs(dims, base, s):
    """Frequencies stretched by parts, and the factor on cosine and sine."""
    def dim_of(turns):
        return dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(dim_of(s["fast"])), 0), min(math.ceil(dim_of(s["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f = _plain_freqs(dims, base)
    return f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _turn(x, freqs, neighbours=False, mult=1.0):
    """x [T, ..., width]: row t at position t; pairs (i, i + n / 2) or neighbours of the first n dimensions turn.  An
    angle is the 32-bit product of position and 32-bit frequency, as the reference defines it."""
    n = 2 * freqs.numel()
    t = torch.arange(x.shape[0], device=DEV, dtype=torch.float32)
    a = (t[:, None] * freqs.to(DEV, torch.float32)[None, :]).to(F64).view(x.shape[0], *[1] * (x.dim() - 2), -1)
    c, s = torch.cos(a) * mult, torch.sin(a) * mult
    out = x.clone()
    i, j = (slice(0, n, 2), slice(1, n, 2)) if neighbours else (slice(0, n // 2), slice(n // 2, n))
    u, v = x[..., i], x[..., j]
    out[..., i], out[..., j] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, visible=None, cap=None, sink=False):
    """q [T, H, dk], k [T, G, dk], v [T, G, dv] of one sequence; ``visible(i, j)`` limits the keys j <= i of position i."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=DEV)
    j = torch.arange(T, device=DEV)[None, :]
    kt, vt = k.permute(1, 2, 0), v.transpose(0, 1)
    for at in range(0, T, 512):
        i = torch.arange(at, min(T, at + 512), device=DEV)[:, None]
        end = at + i.shape[0]
        see = j[:, :end] <= i
        if visible is not None:
            see &= visible(i, j[:, :end])
        qb = q[at:end].view(end - at, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, -1, q.shape[2])
        s = (qb @ kt[:, :, :end]) * scale
        s = s.view(G, H // G, end - at, end)
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~see, -math.inf)
        top = s.amax(dim=-1, keepdim=True)
        if sink:
            top = top.clamp(min=0.0)
        p = torch.exp(s - top)
        p = p / (p.sum(dim=-1, keepdim=True) + (torch.exp(-top) if sink else 0.0))
        o = p.view(G, -1, end) @ vt[:, :end]
        out[at:end] = o.view(H, end - at, -1).transpose(0, 1)
    return out


def _filter(u, taps):
    """A causal filter over time, a row of ``taps`` a channel; its last column meets the current token."""
    n = taps.shape[1]
    pad = torch.cat([torch.zeros(n - 1, u.shape[1], dtype=F64, device=DEV), u])
    return sum(taps[:, j] * pad[j:j + u.shape[0]] for j in range(n))


def _recur(decay, k, v, q):
    """S_t = decay_t S_{t-1} + k_t v_t^T, o_t = S_t^T q_t a head: decay [T, H], k and q [T, H, dk], v [T, H, dv]."""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], dtype=F64, device=DEV)
    out = torch.empty_like(v)
    for t in range(k.shape[0]):
        S = torch.baddbmm(S * decay[t][:, None, None], k[t][:, :, None], v[t][:, None, :])
        out[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    return out


def _experts(h, w, p, scores, weights, top, ff):
    """The ``top`` experts of each row by ``scores``, summed by their weights."""
    ids = scores.topk(top, dim=-1).indices
    wt = weights(ids)
    out = torch.zeros_like(h)
    for e in range(scores.shape[1]):
        row, at = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            out.index_add_(0, row, wt[row, at][:, None] * _gated(h[row], w, f"{p}e{e}.", ff))
    return out


def _gated(h, w, p, ff):
    d = h.shape[1]
    return (_silu(h @ w(p + "gate", ff, d).T) * (h @ w(p + "up", ff, d).T)) @ w(p + "down", d, ff).T


def _llama(cfg, w, seqs):
    d, I, H, G, hd = (cfg[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
    eps, V = cfg["rms_norm_eps"], cfg["vocab_size"]
    freqs = _llama3_freqs(hd, cfg["rope_theta"], cfg.get("rope_scaling"))
    table = w("model.embed_tokens.weight", V, d)
    x = torch.cat([table[s] for s in seqs])
    head = table if cfg.get("tie_word_embeddings") else None
    del table
    lens = [len(s) for s in seqs]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w(p + "input_layernorm.weight", d, mean=1.0), eps)
        q, k, v = (h @ w(p + f"self_attn.{n}_proj.weight", m * hd, d).T for n, m in (("q", H), ("k", G), ("v", G)))
        o = [_attend(_turn(a.view(-1, H, hd), freqs), _turn(b.view(-1, G, hd), freqs), c.view(-1, G, hd), hd ** -0.5).flatten(1)
             for a, b, c in zip(q.split(lens), k.split(lens), v.split(lens))]
        x = x + torch.cat(o) @ w(p + "self_attn.o_proj.weight", d, H * hd).T
        h = _rms(x, w(p + "post_attention_layernorm.weight", d, mean=1.0), eps)
        g = _silu(h @ w(p + "mlp.gate_proj.weight", I, d).T) * (h @ w(p + "mlp.up_proj.weight", I, d).T)
        x = x + g @ w(p + "mlp.down_proj.weight", d, I).T
    x = _rms(_last(x, lens), w("model.norm.weight", d, mean=1.0), eps)
    return x @ (w("lm_head.weight", V, d) if head is None else head).T


def _last(x, lens):
    return torch.stack([c[-1] for c in x.split(lens)])


def _mosurax(cfg, w, seqs):
    d, V, eps = cfg["width"], cfg["vocab"], cfg["norm"]["eps"]
    table, places = w("embed", V, d), w("pos", cfg["max_positions"], d)
    x = torch.cat([table[s] + places[:len(s)] for s in seqs])
    lens = [len(s) for s in seqs]
    for i, layer in enumerate(cfg["layers"]):
        m, mlp, p = layer["mixer"], layer["mlp"], f"l{i}.mix."
        H, G, hd = m["heads"], m["kv_heads"], m["dim"]
        h = _rms(x, w(f"l{i}.norm1", d, mean=1.0), eps)
        q, k, v = ((h @ w(p + n, r * hd, d).T).view(-1, r, hd).split(lens) for n, r in (("q", H), ("k", G), ("v", G)))
        o = torch.cat([_attend(*qkv, m["scale"], sink=True).flatten(1) for qkv in zip(q, k, v)])
        x = x + (o * torch.sigmoid(h @ w(p + "g", H * hd, d).T)) @ w(p + "o", d, H * hd).T
        h, p = _rms(x, w(f"l{i}.norm2", d, mean=1.0), eps), f"l{i}.mlp."
        if mlp["kind"] == "dense":
            x = x + _gated(h, w, p, mlp["ff"])
            continue
        z = h @ w(p + "router", mlp["router"]["experts"], d).T
        x = x + _experts(h, w, p, z, lambda ids: torch.softmax(z.gather(1, ids), dim=-1), mlp["router"]["top"], mlp["expert"]["ff"]) \
            + _gated(h, w, p + "shared.", mlp["shared"]["ff"])
    z = _rms(_last(x, lens), w("final.norm", d, mean=1.0), eps) @ w("head", V, d).T
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _mogutar(cfg, w, seqs):
    d, V, eps, side = cfg["width"], cfg["vocab"], cfg["norm"]["eps"], cfg["token_side"]["dim"]
    x = torch.cat([w("embed", V, d)[s] for s in seqs])
    beside = w("side.embed", V, len(cfg["layers"]) * side)[torch.cat(seqs)]
    lens = [len(s) for s in seqs]

    def attention(x, m, p):
        H, G, hd = m["heads"], m["kv_heads"], m["dim"]
        window, keep = m["mask"]["size"], m["mask"]["keep_first"]
        freqs, mult = _stretched_freqs(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
        out, part = [], {}
        for n, r in (("q", H), ("k", G), ("v", G)):
            taps = w(p + n + ".conv", r * hd, m["conv"])
            u = x @ w(p + n, r * hd, d).T + w(p + n + ".b", r * hd)
            part[n] = [_filter(c, taps).view(-1, r, hd) for c in u.split(lens)]
        qn, kn = w(p + "q.norm", hd, mean=1.0), w(p + "k.norm", hd, mean=1.0)
        for q, k, v in zip(part["q"], part["k"], part["v"]):
            q, k = (_turn(_rms(c, n, eps), freqs, mult=mult) for c, n in ((q, qn), (k, kn)))
            out.append(_attend(q, k, v, m["scale"], lambda i, j: (i - j < window) | (j < keep), m["softcap"]).flatten(1))
        return torch.cat(out) @ w(p + "o", d, H * hd).T

    def state_space(x, m, p):
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, C = H * P, H * P + 2 * G * N
        proj = x @ w(p + "in", inner + C + H, d).T
        taps, skip = w(p + "conv", C, m["conv"]), w(p + "D", H, mean=1.0)
        out = []
        for c in proj.split(lens):
            u = _silu(_filter(c[:, inner:inner + C], taps))
            b, q = (u[:, inner + s:inner + s + G * N].view(-1, G, N).repeat_interleave(H // G, dim=1) for s in (0, G * N))
            v = u[:, :inner].view(-1, H, P)
            step = torch.nn.functional.softplus(c[:, inner + C:])
            y = _recur(torch.exp(-step), b * step[:, :, None], v, q) + skip[:, None] * v
            y = (y.flatten(1) * _silu(c[:, :inner])).view(-1, m["norm_groups"], inner // m["norm_groups"])
            out.append(_rms(y, None, eps).flatten(1))
        return (torch.cat(out) * w(p + "norm", inner, mean=1.0)) @ w(p + "o", d, inner).T

    def linear_attention(x, m, p):
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        decay = torch.tensor(m["decay"], dtype=F64, device=DEV)
        q, k, v = (_silu(x @ w(p + n, H * r, d).T).view(-1, H, r).split(lens) for n, r in (("q", dk), ("k", dk), ("v", dv)))
        o = torch.cat([_recur(decay.expand(c.shape[0], H), b, c, a).flatten(1) for a, b, c in zip(q, k, v)])
        y = _rms(o, w(p + "norm", H * dv, mean=1.0), eps) * torch.sigmoid(x @ w(p + "g", H * dv, d).T)
        return y @ w(p + "o", d, H * dv).T

    for i, layer in enumerate(cfg["layers"]):
        m, r, p = layer["mixer"], layer["mlp"]["router"], f"l{i}."
        if layer["type"] == "parallel":
            y = m["left_scale"] * attention(x, m["left"], p + "mix.left.") + m["right_scale"] * state_space(x, m["right"], p + "mix.right.")
        else:
            y = linear_attention(x, m, p + "mix.")
        x = x + _rms(y, w(p + "norm1", d, mean=1.0), eps)
        s = torch.sigmoid(x @ w(p + "mlp.router", r["experts"], d).T)
        y = _experts(x, w, p + "mlp.", s, lambda ids: s.gather(1, ids), r["top"], layer["mlp"]["expert"]["ff"])
        x = x + _rms(y, w(p + "norm2", d, mean=1.0), eps)
        y = (_gelu(x @ w(p + "side.gate", side, d).T) * beside[:, i * side:(i + 1) * side]) @ w(p + "side.proj", d, side).T
        x = x + _rms(y, w(p + "side.norm", d, mean=1.0), eps)
    return _rms(_last(x, lens), w("final.norm", d, mean=1.0), eps) @ w("head", V, d).T


def _forilorn(cfg, w, seqs):
    d, V, eps, bg = cfg["width"], cfg["vocab"], cfg["norm"]["eps"], cfg["embedding"]["bigram"]
    table, pair = w("embed", V, d), w("bigram", bg["buckets"] + 1, d)
    rows = [torch.cat([torch.tensor([bg["buckets"]], device=DEV), (s[:-1] * bg["mul_prev"] + s[1:] * bg["mul_cur"]) % bg["buckets"]]) for s in seqs]
    x = torch.cat([table[s] * cfg["embedding"]["scale"] + pair[r] for s, r in zip(seqs, rows)])
    lens = [len(s) for s in seqs]

    def attention(x, m, p):
        H, G, hd, size = m["heads"], m["kv_heads"], m["dim"], m["mask"]["size"]
        freqs = _plain_freqs(m["rot"]["dims"], m["rot"]["base"])
        q, k = ((x @ w(p + n, r * hd, d).T).view(-1, r, hd).split(lens) for n, r in (("q", H), ("k", G)))
        o = [_attend(_rms(_turn(a, freqs, True), None, eps), _rms(_turn(b, freqs, True), None, eps), b, m["scale"],
                     lambda i, j: i // size == j // size).flatten(1) for a, b in zip(q, k)]
        return (torch.cat(o) * torch.sigmoid(x @ w(p + "g", H * hd, d).T)) @ w(p + "o", d, H * hd).T

    def latent(x, m, p):
        H, hd, rd, vd, r, qr, size = *(m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank")), m["mask"]["size"]
        freqs = _plain_freqs(m["rot"]["dims"], m["rot"]["base"])
        cq = _rms(x @ w(p + "dq", qr, d).T, w(p + "dq.norm", qr, mean=1.0), eps)
        q = (cq @ w(p + "uq", H * (hd + rd), qr).T).view(-1, H, hd + rd)
        low = x @ w(p + "dkv", r + rd, d).T
        c = _rms(low[:, :r], w(p + "dkv.norm", r, mean=1.0), eps)
        k, v = (c @ w(p + "uk", H * hd, r).T).view(-1, H, hd), (c @ w(p + "uv", H * vd, r).T).view(-1, H, vd)
        o = []
        for a, b, e, z in zip(q.split(lens), k.split(lens), v.split(lens), low[:, r:].split(lens)):
            a = torch.cat([a[..., :hd], _turn(a[..., hd:], freqs, True)], dim=-1)
            b = torch.cat([b, _turn(z[:, None], freqs, True).expand(-1, H, -1)], dim=-1)
            o.append(_attend(a, b, e, m["scale"], lambda i, j: i - j < size))
        gate = torch.sigmoid(x @ w(p + "g", H, d).T)
        return (torch.cat(o) * gate[:, :, None]).flatten(1) @ w(p + "o", d, H * vd).T

    for i, layer in enumerate(cfg["layers"]):
        p, ff = f"l{i}.", layer["mlp"]["ff"]
        y = (attention if layer["type"] == "attention" else latent)(x, layer["mixer"], p + "mix.")
        x = x + cfg["residual_mult"] * _rms(y, 1.0 + w(p + "norm1", d), eps)
        y = _gelu(x @ w(p + "mlp.up", ff, d).T) @ w(p + "mlp.down", d, ff).T
        x = x + cfg["residual_mult"] * _rms(y, 1.0 + w(p + "norm2", d), eps)
    return _rms(_last(x, lens), 1.0 + w("final.norm", d), eps) @ table.T


def exact(case, seed):
    cfg = _config(case["model"])
    prompts, fed = _tokens(case, seed)
    seqs = [torch.tensor(p + (fed[0][b] if fed else []), device=DEV) for b, p in enumerate(prompts)]
    model = _llama if case["model"].startswith("llama") else {"mosurax": _mosurax, "mogutar": _mogutar, "forilorn": _forilorn}[case["model"]]
    return model(cfg, _Weights(seed, case["dtype"]), seqs)
