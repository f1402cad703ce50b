"""The work that users of the engine have it do, as cases that can be timed and checked.

A case is one model with random weights and one call pattern of ``Engine.step``, the function that generation, the
scheduler and trace replay all go through:

* ``rows`` requests that decode one token each, with between ``low`` and ``high`` tokens in the cache (drawn per
  request from the seed), and
* a new request's prompt of ``prompt`` tokens, in portions of at most ``PORTION`` tokens, whose last ``want`` positions'
  logits are wanted (1: generation, more: scoring and replay).

A case with rows alone is a decode step, one with a prompt alone a prefill, one with both the mixed batch that a server
runs while a request comes in.  The requests that decode grow by a token a pass, as they do in use.

Models: Qwen3 at the layer sizes of 0.6B (all layers) and of 8B (fewer layers), in bfloat16 and in the true 32-bit mode,
and three designs that between them reach the other kinds of kernels: Kefetar (soft-capped attention behind short
convolutions, decay retention), Bevuvik (differences of two attention maps over a window, soft-capped attention beside
a gated delta rule) and Mukenex (latent attention, attention over blocks of positions, lightning retention, experts
named by a token table, several residual streams).  Designs whose router ranks computed logits are left out: a choice
between two experts within rounding of each other moves a token's logits by more than any tolerance.
"""
import math
import random
import zlib

import torch

from llm_infer_rust_b200 import Engine, StepEntry

VOCAB = 151936
PORTION = 8192                # the engine's default bound of prompt tokens a step
ROOM = 4096                   # tokens that a decoding request may grow by before it starts again


# ------------------------------------------------------------------------------------------------------------ models
def _qwen3(width, heads, kv_heads, inter, layers, tied):
    return dict(model_type="qwen3", architectures=["Qwen3ForCausalLM"], rope_theta=1e6, rms_norm_eps=1e-6,
                torch_dtype="bfloat16", eos_token_id=None, num_hidden_layers=layers, hidden_size=width,
                num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=128, intermediate_size=inter,
                vocab_size=VOCAB, tie_word_embeddings=tied, max_position_embeddings=40960)


def _kefetar(width, heads, kv_heads, inter, layers):
    attn = {"type": "attention", "mlp": {"kind": "dense", "ff": inter * 3 // 2},
            "mixer": {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "conv": 3, "scale": 128 ** -0.5,
                      "softcap": 50.0, "v_mix": True, "rot": {"base": 1e6, "dims": 128, "scaling": {"factor": 4.0}}}}
    ret = {"type": "retention", "mlp": {"kind": "dense", "ff": inter * 3 // 2},
           "mixer": {"heads": heads, "dim": 128, "vdim": 128, "rot": {"base": 1e6, "dims": 64},
                     "decay": [1.0 - 2.0 ** (-5 - 3 * h / max(1, heads - 1)) for h in range(heads)]}}
    return {"architecture": "Kefetar", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "canon": {"taps": 3},
            "layers": [attn if i % 2 == 0 else ret for i in range(layers)]}


def _bevuvik(width, heads, kv_heads, inter, layers):
    mlp = {"kind": "dense", "ff": inter, "limit": 7.0}
    pair = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0,
                 "rot": {"base": 1e6, "dims": 64}},
        "right": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}}
    diff = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": heads, "kv_heads": kv_heads, "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "diff": 0.4,
        "rot": {"base": 1e6, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}},
        "mask": {"size": 1024}}}
    return {"architecture": "Bevuvik", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "residual_mult": 0.3,
            "layers": [pair if i % 4 == 0 else diff for i in range(layers)], "loop": {"start": 1, "stop": 3, "times": 2}}


def _mukenex(width, heads, kv_heads, inter, layers):
    moe = {"kind": "moe", "expert": {"ff": inter // 2}, "router": {"experts": 8, "top": 2}}
    lightning = {"type": "lightning", "mlp": {"kind": "dense", "ff": inter * 3 // 2},
                 "mixer": {"heads": heads, "dim": 128, "vdim": 128,
                           "decay": [1.0 - 2.0 ** (-5 - 3 * h / max(1, heads - 1)) for h in range(heads)]}}
    latent = {"type": "latent_attention", "mlp": moe,
              "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 256, "scale": 192 ** -0.5,
                        "rot": {"base": 1e6, "dims": 64}, "mask": {"size": 1024}}}
    blocks = {"type": "attention", "mlp": moe,
              "mixer": {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                        "mask": {"size": 1024}}}
    return {"architecture": "Mukenex", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "streams": 4,
            "logit_softcap": 30.0, "layers": [(lightning, latent, blocks)[i % 3] for i in range(layers)]}


def config_of(case):
    model = case["model"]
    if model == "qwen3-0.6b":
        return _qwen3(1024, 16, 8, 3072, 28, True)
    if model == "qwen3-8b":
        return _qwen3(4096, 32, 8, 12288, 8, False)
    return {"kefetar": _kefetar, "bevuvik": _bevuvik, "mukenex": _mukenex}[model](1024, 16, 8, 3072, 6)


# ------------------------------------------------------------------------------------------------------------- cases
def _case(model, dtype="bfloat16", rows=0, low=0, high=0, prompt=0, want=1, graphs=False):
    return {"model": model, "dtype": dtype, "rows": rows, "low": low, "high": high, "prompt": prompt,
            "want": min(want, prompt), "graphs": graphs}


def listed():
    return [dict(c, name=n) for n, c in (
        # one user talks to a small model: latency and the count of launches
        ("decode-1", _case("qwen3-0.6b", rows=1, low=300, high=300, graphs=True)),
        # the headline benchmark: eight requests at 4,096 tokens
        ("decode-8-long", _case("qwen3-0.6b", rows=8, low=4096, high=4096, graphs=True)),
        # a server under load: many requests of all lengths, wide layers
        ("decode-45-ragged", _case("qwen3-8b", rows=45, low=100, high=2000, graphs=True)),
        # a question of no special length: no shape comes twice, so no graph of its step exists
        ("prompt-777", _case("qwen3-0.6b", prompt=777)),
        # the benchmark's prompt at wide layers, the benchmark's options
        ("prompt-2048-wide", _case("qwen3-8b", prompt=2048, graphs=True)),
        # a document, in portions
        ("prompt-document", _case("qwen3-0.6b", prompt=11111)),
        # a request comes in while others decode: a shape that does not come again
        ("mixed", _case("qwen3-0.6b", rows=20, low=50, high=1500, prompt=1000)),
        # the exact mode: a trace's prompt with the logits of its places, and steps of generation
        ("float32-prompt", _case("qwen3-0.6b", "float32", prompt=300, want=16)),
        ("float32-decode", _case("qwen3-0.6b", "float32", rows=4, low=200, high=900)),
        # the designs: prompts on their attention and recurrence kernels, and a step of a few requests
        ("kefetar-prompt", _case("kefetar", prompt=1500)),
        ("bevuvik-prompt", _case("bevuvik", prompt=2048)),
        ("mukenex-decode", _case("mukenex", rows=8, low=600, high=2000, graphs=True)),
    )]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case: a prompt of 16 to 8,192 tokens, a step of 1 to 64 requests of up to 4,096 tokens, or both.  The
    32-bit mode and the designs are used with shorter prompts."""
    kind = rng.choice(("prompt", "decode", "mixed"))
    model, dtype = rng.choice((("qwen3-0.6b", "bfloat16"), ("qwen3-0.6b", "bfloat16"), ("qwen3-8b", "bfloat16"),
                               ("qwen3-0.6b", "float32"), ("kefetar", "bfloat16"), ("bevuvik", "bfloat16"),
                               ("mukenex", "bfloat16")))
    longest = 400 if dtype == "float32" else 3000 if model != "qwen3-0.6b" else 8192
    prompt = _log_int(rng, 16, longest if kind == "prompt" else min(longest, 2000)) if kind != "decode" else 0
    rows = high = low = 0
    if kind != "prompt":
        rows = _log_int(rng, 1, 16 if dtype == "float32" else 64)
        high = _log_int(rng, 64, min(4096, 40000 // rows))
        low = rng.randint(max(1, high // 8), high)
    return _case(model, dtype, rows, low, high, prompt, rng.choice((1, 1, 5)), rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------------ the timed call
class _State:
    def __init__(self, case, seed):
        self.case = case
        self.contexts, self.next_tokens, self.prompt = _inputs(case, seed)
        limit = max(case["high"] + ROOM, case["prompt"] + 1)
        self.engine = Engine(None, random_weights_config=config_of(case), random_weights_seed=seed % 1000, dtype=case["dtype"],
                             max_running_req=2 * case["rows"] + 2, max_seq_len=limit,
                             max_total_tokens=case["rows"] * limit + 2 * case["prompt"] + 64 * (case["rows"] + 2),
                             cuda_graph_bs=case["rows"] if case["graphs"] and not case["prompt"] else 0,
                             prefill_cuda_graph_max_tokens=2048 if case["graphs"] and case["prompt"] else 0,
                             log_level="warn")
        self.limit = limit
        self.fill()

    def fill(self):
        for r, ids in enumerate(self.contexts):
            self.engine.open_request(r + 1)
            for at in range(0, len(ids), PORTION):
                self.engine.step([StepEntry(r + 1, ids[at:at + PORTION], [])])


def _inputs(case, seed):
    """Token ids of the requests that decode, the token each decodes next, and the new prompt."""
    rng, gen = random.Random(seed), torch.Generator().manual_seed(seed)
    lengths = [rng.randint(case["low"], case["high"]) for _ in range(case["rows"])]

    def ids(n):
        return torch.randint(0, VOCAB, (n,), generator=gen).tolist()
    return [ids(n) for n in lengths], ids(len(lengths)), ids(case["prompt"])


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    engine, case = state.engine, state.case
    rows = [StepEntry(r + 1, [t], [0]) for r, t in enumerate(state.next_tokens)]
    if rows and max(engine.request_length(e.request) for e in rows) >= state.limit:
        for e in rows:                                # the longest conversation is full: all begin again
            engine.close_request(e.request)
        state.fill()
    if not state.prompt:
        return engine.step(rows)
    new, n, want = case["rows"] + 1, case["prompt"], case["want"]
    engine.open_request(new)
    for at in range(0, n, PORTION):
        part = state.prompt[at:at + PORTION]
        wanted = [i for i in range(len(part)) if at + i >= n - want]
        logits = engine.step([StepEntry(new, part, wanted)] + rows)
    engine.close_request(new)
    return logits


# -------------------------------------------------------------------------------------------------------------- bounds
def _layer_numbers(case):
    """Of the whole model: matrix weights that every token is multiplied with, weights that are read when ``tokens``
    tokens come, and per layer (bytes of cache a position, FLOPs a query and position, window), FLOPs of the
    recurrences a token and the bytes of their states a request."""
    raw, size = config_of(case), 4 if case["dtype"] == "float32" else 2
    if "architecture" not in raw:
        w, h, g, inter = raw["hidden_size"], raw["num_attention_heads"], raw["num_key_value_heads"], raw["intermediate_size"]
        per = w * 128 * (2 * h + 2 * g) + 3 * w * inter
        n = raw["num_hidden_layers"]
        return n * per, lambda tokens: n * per, [(2 * g * 128 * size, 4 * h * 128, None)] * n, 0, 0, w
    w, used, read, cache, scan, states = raw["width"], 0, [], [], 0, 0
    runs = list(range(len(raw["layers"])))
    if "loop" in raw:
        runs = runs[:3] + runs[1:]
        used += raw["loop"]["times"] * 2 * w * w
        read.append(lambda tokens: 2 * w * w)
    for at, i in enumerate(runs):
        layer = raw["layers"][i]
        m, mlp, kind = layer["mixer"], layer["mlp"], layer["type"]
        h = m["heads"] if "heads" in m else m["left"]["heads"]
        if kind in ("retention", "lightning"):
            mix = 5 * w * h * 128
            scan, states = scan + 4 * h * 128 * 128, states + h * 128 * 128 * 4
        elif kind == "parallel":
            g = m["left"]["kv_heads"]
            mix = w * 128 * (2 * h + 2 * g) + w * 128 * (2 * m["right"]["kv_heads"] + 3 * h)
            scan, states = scan + 8 * h * 128 * 128, states + h * 128 * 128 * 4
            cache.append((2 * g * 128 * size, 4 * h * 128, None))
        elif kind == "latent_attention":
            mix = w * (h * 192 + 256 + 64 + 2 * h * 128) + 2 * h * 128 * 256
            cache.append(((256 + 64) * size, 2 * h * (192 + 128), m["mask"]["size"]))
        else:
            g, maps = m["kv_heads"], 2 if "diff" in m else 1
            gate = h * 128 if "softcap" in m else 0
            mix = w * 128 * (2 * h + 2 * g) + w * gate
            cache.append((2 * g * 128 * size, 2 * h * (128 + 128 * maps), m["mask"]["size"] if "mask" in m else None))
        if mlp["kind"] == "moe":
            e, top, ff = mlp["router"]["experts"], mlp["router"]["top"], 3 * w * mlp["expert"]["ff"]
            used += mix + top * ff
            read.append(lambda tokens, mix=mix, e=e, top=top, ff=ff: mix + e * (1 - (1 - top / e) ** tokens) * ff)
        else:
            ff = (3 if raw["architecture"] == "Bevuvik" else 2) * w * mlp["ff"]
            used += mix + ff
            if i not in runs[:at]:
                read.append(lambda tokens, mix=mix, ff=ff: mix + ff)
    return used, lambda tokens: sum(f(tokens) for f in read), cache, scan, states, w


def work(case):
    used, read, cache, scan, states, width = _layer_numbers(case)
    size = 4 if case["dtype"] == "float32" else 2
    mean = (case["low"] + case["high"]) / 2
    tokens, logits = case["rows"] + case["prompt"], case["rows"] + case["want"]
    flops = 2.0 * tokens * used + 2.0 * logits * VOCAB * width + tokens * scan
    moved = size * (read(tokens) + VOCAB * width + tokens * width) + 4 * logits * VOCAB + 4 * tokens
    moved += 2 * states * (case["rows"] + (1 if case["prompt"] else 0))
    for position, flop, window in cache:
        n, s = case["prompt"], window or 1 << 30
        flops += flop * (case["rows"] * min(mean, s) + (n * (n + 1) / 2 if n <= s else s * (s + 1) / 2 + (n - s) * s))
        moved += position * (case["rows"] * min(mean, s) + tokens)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    # four times what was measured against exact(), and at most 0.03.  float32: sums of up to a few thousand terms in 32
    # bits, 2.1e-6.  bfloat16: every layer rounds its activations to 8 bits; 0.012 to 0.021 for Qwen3 (28 layers, and 8
    # wide ones), 0.005 to 0.0065 for six layers of the designs, whose streams are 32-bit.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 0.03 if case["model"].startswith("qwen3") else 0.024, "max": 0.4}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
_MASK = (1 << 64) - 1


def _mix_int(x):
    x &= _MASK
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & _MASK
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & _MASK
    return x ^ (x >> 31)


def _signed(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _mix(x):
    x = (x ^ ((x >> 30) & ((1 << 34) - 1))) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ ((x >> 27) & ((1 << 37) - 1))) * _signed(0x94D049BB133111EB)
    return x ^ ((x >> 31) & ((1 << 33) - 1))


class _Weights:
    """The random weights of a seed by checkpoint name: sums of eight 16-bit fields of hashed counters, as the
    random-weights mode documents them, rounded to the model's type and widened to 64 bits."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = seed, dtype

    def key(self, name):
        return _signed(_mix_int(_mix_int(self.seed) ^ (zlib.crc32(name.encode()) * 0x9E3779B97F4A7C15)))

    def __call__(self, name, *shape):
        key, n = self.key(name), math.prod(shape)
        out = torch.empty(n, dtype=self.dtype, device="cuda")
        for at in range(0, n, 1 << 24):
            i = torch.arange(at, min(n, at + (1 << 24)), device="cuda")
            total = torch.zeros_like(i)
            for word in (0, 1):
                h = _mix(key + i * 2 + word)
                for field in range(4):
                    total += (h >> (16 * field)) & 0xFFFF
            z = (total.float() - 8 * 32767.5) * (1.0 / math.sqrt(8 * (65536.0 ** 2 - 1.0) / 12.0))
            out[at:at + i.numel()] = (0.02 * z).to(self.dtype)
        return out.double().reshape(shape)

    def choices(self, name, rows, top, modulus):
        first = (_mix(self.key(name) + torch.arange(rows, device="cuda") * top) >> 49) & ((1 << 15) - 1)
        return (first[:, None] + torch.arange(top, device="cuda")) % modulus


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _silu(x):
    return x * torch.sigmoid(x)


def _taps(x, w):
    """Causal convolution of every channel: x [T, C], w [C, taps]."""
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(w[:, j] * padded[j:j + x.shape[0]] for j in range(taps))


def _turn(x, angles, gain=1.0, pairs=False):
    """Rotate the first 2 n coordinates of x [T, heads, d] by angles [T, n]: halves, or neighbouring pairs."""
    n = angles.shape[1]
    c, s = gain * torch.cos(angles)[:, None], gain * torch.sin(angles)[:, None]
    first, second = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if pairs else (slice(0, n), slice(n, 2 * n))
    out = x.clone()
    out[..., first] = x[..., first] * c - x[..., second] * s
    out[..., second] = x[..., second] * c + x[..., first] * s
    return out


def _angles(T, dims, base):
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device="cuda") / dims)
    return torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * f


def _attend(q, k, v, scale, cap=None, window=None, block=None, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv]: causal softmax attention, a piece of queries of a head at a time."""
    T, H = q.shape[:2]
    rep, out = H // k.shape[1], q.new_empty(q.shape[0], q.shape[1], v.shape[2])
    step, cols = 2048, torch.arange(T, device=q.device)
    for at in range(0, T, step):
        rows, end = cols[at:at + step, None], min(T, at + step)
        hidden = cols[None, :end] > rows
        if window:
            hidden |= rows - cols[None, :end] >= window
        if block:
            hidden |= rows // block != cols[None, :end] // block
        for h in range(H):
            s = (q[at:end, h] @ k[:end, h // rep].T) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(hidden, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[h].expand(len(s), 1)], 1)
            out[at:end, h] = torch.softmax(s, -1)[:, :end] @ v[:end, h // rep]
    return out


def _decayed(q, k, v, decay):
    """o_i = sum over j <= i of decay^(i - j) (q_i . k_j) v_j."""
    T, i = q.shape[0], torch.arange(q.shape[0], device=q.device)
    back = (i[:, None] - i[None, :]).double()
    return torch.stack([((q[:, h] @ k[:, h].T) * torch.where(back >= 0, decay[h] ** back.clamp(min=0), 0.0)) @ v[:, h]
                        for h in range(q.shape[1])], 1)


def _delta(q, k, v, g, beta):
    """S <- g S + k (beta (v - (g S)^T k))^T, o = S^T q; q k [T, H, d], v [T, H, dv], g beta [T, H]."""
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(q.shape[0]):
        S *= g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S += k[t][:, :, None] * u[:, None, :]
        out[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return out


def _layers_qwen3(raw, w, X, ids):
    W, H, G, F, eps = (raw[n] for n in ("hidden_size", "num_attention_heads", "num_key_value_heads", "intermediate_size",
                                        "rms_norm_eps"))
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        q, k, v = (w(p + f"self_attn.{n}_proj.weight", r * 128, W) for n, r in (("q", H), ("k", G), ("v", G)))
        o = w(p + "self_attn.o_proj.weight", W, H * 128)
        gate, up = (w(p + f"mlp.{n}_proj.weight", F, W) for n in ("gate", "up"))
        down = w(p + "mlp.down_proj.weight", W, F)
        for r, x in enumerate(X):
            T, h, a = len(x), _rms(x, eps), _angles(len(x), 128, 1e6)
            qs = _turn(_rms((h @ q.T).view(T, H, 128), eps), a)
            ks = _turn(_rms((h @ k.T).view(T, G, 128), eps), a)
            x = x + _attend(qs, ks, (h @ v.T).view(T, G, 128), 128 ** -0.5).reshape(T, -1) @ o.T
            h = _rms(x, eps)
            X[r] = x + (_silu(h @ gate.T) * (h @ up.T)) @ down.T


def _layers_kefetar(raw, w, X, ids):
    W, eps, first = raw["width"], raw["norm"]["eps"], {}
    for i, layer in enumerate(raw["layers"]):
        p, m, F = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        H, G = m["heads"], m.get("kv_heads", m["heads"])
        q, k, v, g = (w(p + "mix." + n, r * 128, W) for n, r in (("q", H), ("k", G), ("v", G), ("g", H)))
        o, up, down = w(p + "mix.o", W, H * 128), w(p + "mlp.up", F, W), w(p + "mlp.down", W, F)
        canon = [w(p + n, W, 3) for n in ("canon1", "canon2")]
        if layer["type"] == "attention":
            conv = [w(p + f"mix.{n}.conv", r * 128, 3) for n, r in (("q", H), ("k", G), ("v", G))]
            lam = w(p + "mix.vmix")
        for r, x in enumerate(X):
            T, h = len(x), _rms(x, eps)
            h = h + _taps(h, canon[0])
            if layer["type"] == "attention":
                qs, ks, vs = (_taps(h @ a.T, c) for a, c in zip((q, k, v), conv))
                a = _angles(T, 128, 1e6) / 4.0
                if r in first:
                    vs = (1.0 - lam) * vs + lam * first[r]
                else:
                    first[r] = vs
                y = _attend(_turn(qs.view(T, H, 128), a), _turn(ks.view(T, G, 128), a), vs.view(T, G, 128), m["scale"],
                            m["softcap"]).reshape(T, -1) * torch.sigmoid(h @ g.T)
            else:
                a = _angles(T, 64, 1e6)
                y = _decayed(_turn((h @ q.T).view(T, H, 128), a), _turn((h @ k.T).view(T, H, 128), a) * 128 ** -0.5,
                             (h @ v.T).view(T, H, 128), m["decay"])
                y = _rms(y, eps).reshape(T, -1) * _silu(h @ g.T)
            x = x + y @ o.T
            h = _rms(x, eps)
            z = (h + _taps(h, canon[1])) @ up.T
            X[r] = x + (_rms(z, eps) + _rms(z * z, eps) + _rms(z * z * z, eps) + 1.0) @ down.T


def _layers_bevuvik(raw, w, X, ids):
    W, eps, start = raw["width"], raw["norm"]["eps"], list(X)
    into = w("loop.in", W, 2 * W)
    blend = torch.arange(32, dtype=torch.float64, device="cuda")
    low, high = (64 * math.log(4096 / (2 * math.pi * n)) / (2 * math.log(1e6)) for n in (32.0, 1.0))
    low, high = max(math.floor(low), 0), min(math.ceil(high), 63)
    blend = ((blend - low) / max(high - low, 0.001)).clamp(0, 1)
    for i, first in [(0, False), (1, True), (2, False), (1, True), (2, False)] + [(i, False) for i in range(3, len(raw["layers"]))]:
        layer, p = raw["layers"][i], f"l{i}."
        m, F, limit = layer["mixer"], layer["mlp"]["ff"], layer["mlp"]["limit"]
        gate, up, down = w(p + "mlp.gate", F, W), w(p + "mlp.up", F, W), w(p + "mlp.down", W, F)
        p += "mix."
        for r, x in enumerate(X):
            if first:
                x = torch.cat([x, start[r]], -1) @ into.T
            T, h = len(x), _rms(x, eps)
            if layer["type"] == "attention":
                H, G = m["heads"], m["kv_heads"]
                q, k, v = (h @ w(p + n, c * 128, W).T + w(p + n + ".b", c * 128) for n, c in (("q", H), ("k", G), ("v", G)))
                q, k, v = q.view(T, H, 2, 64), k.view(T, G, 2, 64), v.view(T, G, 128)
                a, gain = _angles(T, 64, 1e6) * (blend / 4.0 + 1.0 - blend), 0.1 * math.log(4.0) + 1.0
                maps = [_attend(_turn(q[:, :, j], a, gain, True), _turn(k[:, :, j], a, gain, True), v, m["scale"],
                                window=m["mask"]["size"]) for j in (0, 1)]
                l1, l2 = (torch.exp((w(p + f"lq{j}", 64) * w(p + f"lk{j}", 64)).sum()) for j in (1, 2))
                y = _rms(maps[0] - (l1 - l2 + m["diff"]) * maps[1], eps) * (1.0 - m["diff"])
                y = y.reshape(T, -1) @ w(p + "o", W, H * 128).T + w(p + "o.b", W)
            else:
                H, G, L = m["left"]["heads"], m["left"]["kv_heads"], p + "left."
                a = _angles(T, 64, 1e6)
                q, k, v = ((h @ w(L + n, c * 128, W).T).view(T, c, 128) for n, c in (("q", H), ("k", G), ("v", G)))
                left = _attend(_turn(q, a), _turn(k, a), v, m["left"]["scale"], m["left"]["softcap"]).reshape(T, -1)
                left = left @ w(L + "o", W, H * 128).T
                G, R = m["right"]["kv_heads"], p + "right."
                q, k, v = (_silu(_taps(h @ w(R + n, c * 128, W).T, w(R + n + ".conv", c * 128, 4))).view(T, c, 128)
                           for n, c in (("q", G), ("k", G), ("v", H)))
                beta = torch.sigmoid(h @ w(R + "b", H, W).T)
                g = torch.exp(-torch.exp(w(R + "A_log", H)) * torch.nn.functional.softplus(h @ w(R + "a", H, W).T
                                                                                         + w(R + "dt_bias", H)))
                q, k = (_unit(z).repeat_interleave(H // G, 1) for z in (q, k))
                right = _rms(_delta(q * 128 ** -0.5, k, v, g, beta), eps).reshape(T, -1)
                right = (right * _silu(h @ w(R + "g", H * 128, W).T)) @ w(R + "o", W, H * 128).T
                y = 0.5 * (_rms(left, eps) + _rms(right, eps))
            a, b = (h @ gate.T).clamp(max=limit), (h @ up.T).clamp(-limit, limit)
            X[r] = x + raw["residual_mult"] * (y + (a * torch.sigmoid(1.702 * a) * (b + 1.0)) @ down.T)


def _layers_mukenex(raw, w, X, ids):
    # the streams' coefficients of the random-weights mode leave every stream e + (all sublayers so far), and a
    # sublayer reads their mean: one stream x with x <- x + y; the final sum of all four is undone by the last norm
    # but for its eps
    W, eps = raw["width"], raw["norm"]["eps"]
    for i, layer in enumerate(raw["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        H, G, M = m["heads"], m.get("kv_heads", m["heads"]), f"l{i}.mix."
        o = w(M + "o", W, H * 128)
        for r, x in enumerate(X):
            T, h = len(x), _rms(x, eps)
            if layer["type"] == "lightning":
                q, k, v = (_silu(h @ w(M + n, H * 128, W).T).view(T, H, 128) for n in ("q", "k", "v"))
                y = _rms(_decayed(q, k, v, m["decay"]).reshape(T, -1), eps) * torch.sigmoid(h @ w(M + "g", H * 128, W).T)
            elif layer["type"] == "attention":
                q, k, v = ((h @ w(M + n, c * 128, W).T + w(M + n + ".b", c * 128)).view(T, c, 128)
                           for n, c in (("q", H), ("k", G), ("v", G)))
                y = _attend(_rms(q, eps), _rms(k, eps), v, m["scale"], block=m["mask"]["size"]).reshape(T, -1)
            else:
                C, a = m["kv_rank"], _angles(T, 64, 1e6)
                q, down = (h @ w(M + "q", H * 192, W).T).view(T, H, 192), h @ w(M + "dkv", C + 64, W).T
                c = _rms(down[:, :C], eps)
                key = _turn(down[:, C:].reshape(T, 1, 64), a, pairs=True).expand(T, H, 64)
                q = torch.cat([q[..., :128], _turn(q[..., 128:], a, pairs=True)], -1)
                key = torch.cat([(c @ w(M + "uk", H * 128, C).T).view(T, H, 128), key], -1)
                y = _attend(q, key, (c @ w(M + "uv", H * 128, C).T).view(T, H, 128), m["scale"], window=m["mask"]["size"],
                            sink=w(M + "sink", H)).reshape(T, -1) * torch.sigmoid(h @ w(M + "g", H * 128, W).T)
            x = x + y @ o.T
            h = _rms(x, eps)
            if mlp["kind"] == "dense":
                X[r] = x + torch.nn.functional.gelu(h @ w(p + "mlp.up", mlp["ff"], W).T) @ w(p + "mlp.down", W, mlp["ff"]).T
                continue
            E, top, F = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
            chosen = w.choices(p + "mlp.table", VOCAB, top, E)[ids[r]]
            X[r] = x.clone()
            for e in range(E):
                at = (chosen == e).any(-1).nonzero()[:, 0]
                gate, up, down = (w(p + f"mlp.e{e}.{n}", *s) for n, s in (("gate", (F, W)), ("up", (F, W)), ("down", (W, F))))
                X[r][at] += ((_silu(h[at] @ gate.T) * (h[at] @ up.T)) @ down.T) / top


def exact(case, seed):
    raw, (contexts, following, prompt) = config_of(case), _inputs(case, seed)
    w = _Weights(seed % 1000, torch.float32 if case["dtype"] == "float32" else torch.bfloat16)
    qwen = "architecture" not in raw
    width = raw["hidden_size"] if qwen else raw["width"]
    # the order of step(): the new prompt, then the requests that decode
    sequences = ([(prompt, case["want"])] if prompt else []) + [(c + [t], 1) for c, t in zip(contexts, following)]
    embed = w("model.embed_tokens.weight" if qwen else "embed", VOCAB, width)
    ids = [torch.tensor(s, device="cuda") for s, _ in sequences]
    X = [embed[i] for i in ids]
    head = embed if qwen and raw["tie_word_embeddings"] else w("lm_head.weight" if qwen else "head", VOCAB, width)
    {"qwen3": _layers_qwen3, "kefetar": _layers_kefetar, "bevuvik": _layers_bevuvik,
     "mukenex": _layers_mukenex}["qwen3" if qwen else case["model"]](raw, w, X, ids)
    last = torch.cat([x[len(x) - n:] for x, (_, n) in zip(X, sequences)])
    streams = raw.get("streams", 1)
    logits = _rms(last * streams, raw["rms_norm_eps"] if qwen else raw["norm"]["eps"]) @ head.T
    cap = raw.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits
