"""The work that users of this engine have it do, as cases that can be timed and checked.

Three kinds of pass, all through the public engine (``batchspec_b200.engine``):

``decode``  one captured decode step of a live batch, host token ids in, float32 logits out: what ``Engine.generate`` and
            a decode session do for nearly all of their steps.  The position is not committed, so a pass can be repeated.
``prompt``  requests are admitted, their whole prompts run in one ``Engine.step``, and they are released: the time to a
            first token, or, with every row's logits wanted, the scoring of given texts.
``serve``   a short continuous-batching run through ``Engine.step``: prompts cut into portions beside requests that
            already decode, requests leaving when done.  Its decode steps are given tokens, so logits can be compared.

Models are the configurations that the package ships, with its seeded random weights drawn on the device.  Prompt
lengths of a case run geometrically from ``lo`` to ``hi`` over its requests; token ids and weights come from the seed.
``layers``: a stack of random layers lets the rounding of one grow in the next (in bfloat16 the logits of the 32 layers
of the 8B sizes are 6e-2 off the ones in 64 bits, those of 6 layers 2.5e-2), so the deep models are cut to a number of
their equal layers at which two correct implementations can still be told from a wrong one; the Vabanex design is
taken with its dense layers, because two correct roundings choose different experts for some tokens.
"""
import gc
import hashlib
import json
import math
from pathlib import Path

import torch

import batchspec_b200
from batchspec_b200.config import config_from_json_dict
from batchspec_b200.engine import Engine, StepEntry

PAGE = 16
PRESETS = Path(batchspec_b200.__file__).parent / "config" / "presets"
DEVICE = "cuda:0"
LAYERS = {"llama-3.2-1b": 16, "llama-3.2-3b": 8, "llama-3-8b": 4, "llama-3.1-8b": 4, "vabanex-w2048": 4, "lupusun-w2048": 8,
          "tokolorn-w2048": 4}


def listed():
    return [
        # one user typing at the smallest shipped Llama, short context: launches and latency
        dict(name="decode-1b-x1", kind="decode", model="llama-3.2-1b", dtype="bfloat16", layers=16, requests=1, lo=37, hi=37),
        # the headline: a small interactive batch at 8B sizes with 2,048-token prompts
        dict(name="decode-8b-x8", kind="decode", model="llama-3-8b", dtype="bfloat16", layers=6, requests=8, lo=2048, hi=2048),
        # a loaded server: many requests of very different lengths
        dict(name="decode-3b-x61-ragged", kind="decode", model="llama-3.2-3b", dtype="bfloat16", layers=8, requests=61, lo=64, hi=3000),
        # time to first token of one 2,048-token prompt at 8B sizes
        dict(name="prompt-8b-2048", kind="prompt", model="llama-3-8b", dtype="bfloat16", layers=4, requests=1, lo=2048, hi=2048, rows="last"),
        # continuous batching: prompts in portions beside decoding requests, one long prompt among short ones
        dict(name="serve-8b-portions", kind="serve", model="llama-3.1-8b", dtype="bfloat16", layers=4, requests=5, lo=100, hi=7001, portion=2048, new=3),
        # the 32-bit path, as used to check a model: a few short prompts, and decoding
        dict(name="prompt-1b-fp32", kind="prompt", model="llama-3.2-1b", dtype="float32", layers=16, requests=3, lo=61, hi=700, rows="last"),
        dict(name="decode-1b-fp32-x4", kind="decode", model="llama-3.2-1b", dtype="float32", layers=16, requests=4, lo=33, hi=500),
        # latent attention: scoring one text, and a loaded server's decode step
        dict(name="score-vabanex-2048", kind="prompt", model="vabanex-w2048", dtype="bfloat16", layers=4, requests=1, lo=2048, hi=2048, rows="all"),
        dict(name="decode-vabanex-x64", kind="decode", model="vabanex-w2048", dtype="bfloat16", layers=4, requests=64, lo=300, hi=4096),
        # gated delta rule beside chunked attention: several ragged prompts at once
        dict(name="prompt-lupusun-x3", kind="prompt", model="lupusun-w2048", dtype="bfloat16", layers=8, requests=3, lo=333, hi=2048, rows="last"),
        # lightning attention and the selective scan beside window attention: one prompt, and a medium decode batch
        dict(name="prompt-tokolorn-2048", kind="prompt", model="tokolorn-w2048", dtype="bfloat16", layers=4, requests=1, lo=2048, hi=2048, rows="last"),
        dict(name="decode-tokolorn-x24", kind="decode", model="tokolorn-w2048", dtype="bfloat16", layers=4, requests=24, lo=50, hi=2500),
    ]


def draw(rng):
    """One more case of these ranges.  Upper ends keep a case below the largest listed one."""
    def between(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "serve"])
    c = dict(kind=kind)
    if kind == "decode":
        c["model"], most, longest = rng.choice([("llama-3.2-1b", 64, 3000), ("llama-3.2-3b", 64, 2500), ("llama-3-8b", 8, 2048),
                                                ("vabanex-w2048", 64, 4096), ("lupusun-w2048", 64, 3000),
                                                ("tokolorn-w2048", 64, 3000)])
        c["dtype"] = "float32" if c["model"] == "llama-3.2-1b" and rng.random() < 0.4 else "bfloat16"
        c["layers"] = LAYERS[c["model"]]
        c["requests"] = between(1, most if c["dtype"] == "bfloat16" else 8)
        c["lo"] = between(16, 400)
        c["hi"] = c["lo"] if c["requests"] == 1 else between(c["lo"], longest if c["dtype"] == "bfloat16" else 700)
    elif kind == "prompt":
        c["model"], longest = rng.choice([("llama-3-8b", 2048), ("llama-3.2-3b", 3000), ("llama-3.2-1b", 4000),
                                          ("vabanex-w2048", 2500), ("lupusun-w2048", 3000), ("tokolorn-w2048", 3000)])
        c["dtype"] = "float32" if c["model"] == "llama-3.2-1b" and rng.random() < 0.5 else "bfloat16"
        c["layers"] = LAYERS[c["model"]]
        c["requests"] = rng.choice([1, 1, 2, 3, 4])
        c["lo"] = between(17, 400)
        c["hi"] = between(c["lo"], longest if c["dtype"] == "bfloat16" else 700)
        if c["requests"] == 1:
            c["lo"] = c["hi"]
        c["rows"] = "all" if c["model"] == "vabanex-w2048" else "last"
    else:
        c["model"] = rng.choice(["llama-3.1-8b", "llama-3.2-3b", "llama-3.2-1b"])
        c["dtype"] = "bfloat16"
        c["layers"] = LAYERS[c["model"]]
        c["requests"] = rng.randint(2, 6)
        c["lo"] = between(20, 300)
        c["hi"] = between(1000, 4000)
        c["portion"] = rng.choice([512, 1024, 2048])
        c["new"] = rng.randint(1, 4)
    return c


# ------------------------------------------------------------------------------------------------- what a case means
def config_of(case):
    """The preset's keys, with the case's number of layers."""
    cfg = json.loads((PRESETS / f"{case['model']}.json").read_text())
    if "hidden_size" in cfg:
        cfg["num_hidden_layers"] = case["layers"]
    elif cfg["architecture"] == "Vabanex":
        cfg["layers"] = [cfg["layers"][0]] * case["layers"]
    return cfg


def vocab_of(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def lengths(case):
    n, lo, hi = case["requests"], case["lo"], case["hi"]
    return [int(round(lo * (hi / lo) ** (i / (n - 1)))) if n > 1 else hi for i in range(n)]


def tokens_of(case, seed):
    """Per request its prompt and the tokens that it decodes."""
    vocab, more = vocab_of(config_of(case)), case.get("new", 1)
    gen = torch.Generator().manual_seed(seed)
    return [torch.randint(vocab, (n + more,), generator=gen).tolist() for n in lengths(case)]


def serve_plan(case):
    """Steps of a continuous-batching run: per step a list of (request, first token, count)."""
    lens, new = lengths(case), case["new"]
    done, steps = [0] * len(lens), []
    while any(d < n + new for d, n in zip(done, lens)):
        step = []
        for r, n in enumerate(lens):
            if done[r] < n + new:
                count = min(case["portion"], n - done[r]) if done[r] < n else 1
                step.append((r, done[r], count))
                done[r] += count
        steps.append(step)
    return steps


# ------------------------------------------------------------------------------------------------- the measured path
def prepare(case, seed):
    gc.collect()                 # an earlier state's engine refers to itself through its captured steps
    eng = Engine(dtype=case["dtype"], device=DEVICE)
    eng.load_model(config=config_from_json_dict(config_of(case)), random_seed=seed, draw_on_device=True)
    lens, toks = lengths(case), tokens_of(case, seed)
    eng.setup_caches(max_batch_size=len(lens), max_seq_length=-(-(max(lens) + 512) // PAGE) * PAGE, page_size=PAGE,
                     prefill_chunk_size=512)
    eng.setup_sampling_params(temperature=0.0)
    state = dict(case=case, eng=eng, toks=toks, lens=lens)
    if case["kind"] == "decode":
        # the step is captured on requests that leave again, as a server does before its first real ones: repeating a
        # position only rewrites its cache entry, but would advance a recurrent state
        state["graph"] = eng.decode_graph(len(lens))
        for r in range(len(lens)):
            eng.admit(r)
        _decode(state)
        for r in range(len(lens)):
            eng.release(r)
        batch, room = [], 0
        for r, n in enumerate(lens):
            eng.admit(r)
            batch.append(StepEntry(r, toks[r][:n]))
            room += n
            if room >= 8192 or r == len(lens) - 1:
                eng.step(batch)
                batch, room = [], 0
    return state


@torch.inference_mode()
def _decode(state):
    eng, n = state["eng"], len(state["lens"])
    ids = list(range(n))
    for r in ids:
        eng.cache.reserve(r, 1)
    state["graph"].run(ids, [t[-1] for t in state["toks"]], [0.0] * n, [-1] * n, [0.0] * n, ids, [0] * n)
    return state["graph"].logits[:n]


def run(state):
    case, eng, toks = state["case"], state["eng"], state["toks"]
    if case["kind"] == "decode":
        return _decode(state)
    if case["kind"] == "prompt":
        entries = []
        for r, n in enumerate(state["lens"]):
            eng.admit(r)
            entries.append(StepEntry(r, toks[r][:n], want=range(n) if case["rows"] == "all" else (n - 1,)))
        logits = eng.step(entries)
        for r in range(len(entries)):
            eng.release(r)
        return logits
    out = []
    for step in serve_plan(case):
        entries = []
        for r, first, count in step:
            if first == 0:
                eng.admit(r)
            ends = first + count
            entries.append(StepEntry(r, toks[r][first:ends], want=(count - 1,) if ends >= state["lens"][r] else ()))
        out.append(eng.step(entries))
        for r, first, count in step:
            if first + count == len(toks[r]):
                eng.release(r)
    return out


# ------------------------------------------------------------------------------------------------- what it cannot do without
def _layers(case):
    """Per layer run: (weights, cache values per token, multiply-adds per (query, key) pair, keys a query sees at most,
    state values per request)."""
    cfg = config_of(case)
    if "hidden_size" in cfg:
        d, ff, q = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_attention_heads"] * cfg["head_dim"]
        kv = cfg["num_key_value_heads"] * cfg["head_dim"]
        w = d * (2 * q + 2 * kv) + 3 * d * ff
        return [(w, 2 * kv, 2 * q, None, 0)] * cfg["num_hidden_layers"]
    d, out = cfg["width"], []
    for i in _order(cfg):
        layer = cfg["layers"][i]
        m, f = layer["mixer"], layer["mlp"]
        w = 3 * d * f["ff"]
        cache, pair, seen, held = 0, 0, None, 0
        if layer["type"] == "latent_attention":
            h, qk = m["heads"], m["dim"] + m["rot_dim"]
            a = d * m["q_rank"] + m["q_rank"] * h * qk + d * (m["kv_rank"] + m["rot_dim"]) + h * (m["dim"] + m["vdim"]) * m["kv_rank"] \
                + d * h + d * h * m["vdim"]
            cache, pair = m["kv_rank"] + m["rot_dim"], h * (qk + m["vdim"])
        elif layer["type"] in ("delta", "lightning"):
            h, g = m["heads"], m.get("kv_heads", m["heads"])
            a = d * (2 * g * m["dim"] + 3 * h * m["vdim"])
            held = h * m["dim"] * m["vdim"]
        else:
            p = m.get("left", m)
            q, kv = p["heads"] * p["dim"], p["kv_heads"] * p["dim"]
            a = d * (2 * q + 2 * kv)
            cache, pair, seen = 2 * kv, 2 * q, p["mask"]["size"]
            if "right" in m:
                s = m["right"]
                a += d * 3 * s["inner"] + s["inner"] * (2 * s["dt_rank"] + 2 * s["state"]) + d * q
                held = s["inner"] * s["state"]
        out.append((w + a, cache, pair, seen, held))
    return out


def _order(cfg):
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return list(range(n))
    return list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def work(case):
    cfg, size = config_of(case), 4 if case["dtype"] == "float32" else 2
    d, vocab = cfg.get("hidden_size") or cfg["width"], vocab_of(cfg)
    lens = lengths(case)
    if case["kind"] == "decode":
        steps = [[(r, n, 1, 1) for r, n in enumerate(lens)]]
    elif case["kind"] == "prompt":
        steps = [[(r, 0, n, n if case["rows"] == "all" else 1) for r, n in enumerate(lens)]]
    else:
        steps = [[(r, first, count, int(first + count >= lens[r])) for r, first, count in step] for step in serve_plan(case)]
    total, flops = 0.0, 0.0
    for step in steps:
        rows, n = sum(s[3] for s in step), sum(s[2] for s in step)
        total += (vocab * d * size if rows else 0) + rows * vocab * 4 + n * d * size
        flops += 2.0 * rows * vocab * d
        for weights, cache, pair, seen, held in _layers(case):
            total += weights * size
            flops += 2.0 * weights * n
            for _, first, count, _ in step:
                ends = first + count
                total += min(ends, seen or ends) * cache * size + 2 * held * 4
                flops += 4.0 * held * count
                flops += 2.0 * pair * count * (min(seen, first + count / 2) if seen else first + (count + 1) / 2)
    return dict(bytes=total, flops=flops)


def tolerance(case):
    """Measured: one prompt whole against the same with its last token decoded differs by 0.008 (Vabanex), 0.017 (8B
    sizes, 4 layers), 0.022 (1B sizes) in bfloat16, at most 0.1 at one place, and each is as far from the 64-bit
    values; in 32 bits the logits are 9e-6 off those."""
    return dict(rel=3e-5, max=3e-4) if case["dtype"] == "float32" else dict(rel=0.03, max=0.4)


# ------------------------------------------------------------------------------------------------- the same in 64 bits
class _Weights:
    """The seeded random tensors by checkpoint name: N(0, 0.02) drawn in 32 bits on the device by a generator whose
    seed is a hash of (seed, name), matrices rounded to the run's type; scales are 1 + N(0, 0.01)."""

    def __init__(self, case, seed):
        self.seed, self.dtype = seed, getattr(torch, case["dtype"])

    def draw(self, name, shape):
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(int.from_bytes(hashlib.sha256(f"{self.seed}:{name}".encode()).digest()[:8], "little") & ((1 << 63) - 1))
        return torch.randn(shape, generator=gen, dtype=torch.float32, device=DEVICE)

    def matrix(self, name, *shape):
        return self.draw(name, shape).mul_(0.02).to(self.dtype).double()

    def vector(self, name, *shape):
        return self.draw(name, shape).mul_(0.02).double()

    def ones(self, name, *shape):
        return self.draw(name, shape).mul_(0.01).add_(1.0).double()


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.nn.functional.softplus(x, threshold=60)


def _yarn(base, dims, scaling):
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=DEVICE) / dims)
    if not scaling:
        return f, 1.0

    def place(turns):
        return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(place(scaling["fast"])), 0), min(math.ceil(place(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, device=DEVICE, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / scaling["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0


def _llama_frequencies(cfg):
    dims, s = cfg["head_dim"], cfg["rope_scaling"]
    f = cfg["rope_theta"] ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=DEVICE) / dims)
    if s:
        turns = s["original_max_position_embeddings"] * f / (2 * math.pi)
        smooth = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
        f = f * ((1 - smooth) / s["factor"] + smooth)
    return f


def _rotate(x, f, mag=1.0, pairs=False):
    """x [T, heads, dim] from position 0 on: (j, j + dims/2) turn together, or (2j, 2j + 1) with ``pairs``."""
    a = torch.arange(x.shape[0], dtype=torch.float64, device=DEVICE)[:, None] * f
    c, s = (a.cos() * mag)[:, None], (a.sin() * mag)[:, None]
    h = f.numel()
    if pairs:
        u, v = x[..., :2 * h:2], x[..., 1:2 * h:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., 2 * h:]], -1)
    u, v = x[..., :h], x[..., h:2 * h]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * h:]], -1)


def _attend(q, k, v, scale, window=None, chunk=None, sink=None, cap=None):
    """q [T, H, D], k, v [T, G, D]: causal, over the last ``window`` keys or the keys of the own ``chunk``."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device=DEVICE)
    see = i[None] <= i[:, None]
    if window:
        see &= i[:, None] - i[None] < window
    if chunk:
        see &= i[:, None] // chunk == i[None] // chunk
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=DEVICE)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill_(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :T] @ v[:, h * G // H]
    return out.reshape(T, -1)


def _each(spans, fn):
    """fn over the rows of every request."""
    return torch.cat([fn(a, b) for a, b in spans])


def _conv(x, w, bias=None):
    """Causal, per channel; the last tap multiplies the token's own row."""
    taps = w.shape[1]
    y = sum(torch.nn.functional.pad(x, (0, 0, j, 0))[:x.shape[0]] * w[:, taps - 1 - j] for j in range(taps))
    return y if bias is None else y + bias


def _exact_llama(cfg, W, x, spans):
    d, ff, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    H, G, eps, f = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"], _llama_frequencies(cfg)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W.ones(p + "input_layernorm.weight", d)
        q, k, v = (h @ W.matrix(p + f"self_attn.{n}_proj.weight", m * hd, d).T for n, m in (("q", H), ("k", G), ("v", G)))
        o = _each(spans, lambda a, b: _attend(_rotate(q[a:b].view(-1, H, hd), f), _rotate(k[a:b].view(-1, G, hd), f),
                                              v[a:b].view(-1, G, hd), hd ** -0.5))
        x = x + o @ W.matrix(p + "self_attn.o_proj.weight", d, H * hd).T
        h = _rms(x, eps) * W.ones(p + "post_attention_layernorm.weight", d)
        g = _silu(h @ W.matrix(p + "mlp.gate_proj.weight", ff, d).T) * (h @ W.matrix(p + "mlp.up_proj.weight", ff, d).T)
        x = x + g @ W.matrix(p + "mlp.down_proj.weight", d, ff).T
    return _rms(x, eps) * W.ones("model.norm.weight", d)


def _exact_vabanex(cfg, W, x, spans):
    d, eps = cfg["width"], cfg["norm"]["eps"]

    def norm(x, name):
        c = x - x.mean(-1, keepdim=True)
        return _rms(c, eps) * W.ones(name, d) + W.vector(name + ".b", d)
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        H, D, R, V, C = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        freq, mag = _yarn(m["rot"]["base"], R, m["rot"]["scaling"])
        h = norm(x, f"l{i}.norm1")
        cq = _rms(h @ W.matrix(p + "dq", m["q_rank"], d).T, eps) * W.ones(p + "dq.norm", m["q_rank"])
        q = (cq @ W.matrix(p + "uq", H * (D + R), m["q_rank"]).T).view(-1, H, D + R)
        down = h @ W.matrix(p + "dkv", C + R, d).T
        c = _rms(down[:, :C], eps) * W.ones(p + "dkv.norm", C)
        k = (c @ W.matrix(p + "uk", H * D, C).T).view(-1, H, D)
        v = (c @ W.matrix(p + "uv", H * V, C).T).view(-1, H, V)

        def mix(a, b):
            qr = torch.cat([q[a:b, :, :D], _rotate(q[a:b, :, D:], freq, mag, pairs=True)], -1)
            kr = _rotate(down[a:b, None, C:], freq, mag, pairs=True).expand(-1, H, -1)
            return _attend(qr, torch.cat([k[a:b], kr], -1), v[a:b], m["scale"])
        o = _each(spans, mix).view(-1, H, V) * torch.sigmoid(h @ W.matrix(p + "g", H, d).T)[:, :, None]
        x = x + o.flatten(1) @ W.matrix(p + "o", d, H * V).T
        h, p = norm(x, f"l{i}.norm2"), f"l{i}.mlp."
        g = (h @ W.matrix(p + "gate", f["ff"], d).T).clamp(max=f["limit"])
        u = (h @ W.matrix(p + "up", f["ff"], d).T).clamp(-f["limit"], f["limit"])
        x = x + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ W.matrix(p + "down", d, f["ff"]).T
    return norm(x, "final.norm")


def _exact_lupusun(cfg, W, x, spans):
    d, eps, mult = cfg["width"], cfg["norm"]["eps"], cfg["residual_mult"]
    x0 = x = _rms(x, eps) * W.ones("embed.norm", d)
    loop, before = cfg["loop"], -1
    for i in _order(cfg):
        if i == loop["start"] and before >= i:
            x = x + x0
        before = i
        layer, p = cfg["layers"][i], f"l{i}.mix."
        m, ff = layer["mixer"], layer["mlp"]["ff"]
        H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        h = _rms(x, eps) * W.ones(f"l{i}.norm1", d)
        if layer["type"] == "attention":
            q, k, v = (h @ W.matrix(p + n, c, d).T + W.vector(p + n + ".b", c) for n, c in (("q", H * D), ("k", G * D), ("v", G * V)))
            f, mag = _yarn(m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"])
            sink = W.vector(p + "sink", H)
            y = _each(spans, lambda a, b: _attend(_rms(_rotate(q[a:b].view(-1, H, D), f, mag), eps),
                                                  _rms(_rotate(k[a:b].view(-1, G, D), f, mag), eps), v[a:b].view(-1, G, V),
                                                  m["scale"], chunk=m["mask"]["size"], sink=sink))
        else:
            def taps(n, c):
                rows, conv = h @ W.matrix(p + n, c, d).T, W.matrix(p + n + ".conv", c, m["conv"])
                return _silu(_each(spans, lambda a, b: _conv(rows[a:b], conv)))
            q, k, v = taps("q", G * D).view(-1, G, D), taps("k", G * D).view(-1, G, D), taps("v", H * V).view(-1, H, V)
            q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, k = (q * D ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
            beta = torch.sigmoid(h @ W.matrix(p + "b", H, d).T)
            g = torch.exp(-torch.exp(W.vector(p + "A_log", H)) * _softplus(h @ W.matrix(p + "a", H, d).T + W.vector(p + "dt_bias", H)))
            o = torch.empty(x.shape[0], H, V, dtype=torch.float64, device=DEVICE)
            for a, b in spans:
                S = torch.zeros(H, D, V, dtype=torch.float64, device=DEVICE)
                for t in range(a, b):
                    S = S * g[t, :, None, None]
                    u = beta[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
                    S = S + k[t, :, :, None] * u[:, None]
                    o[t] = (q[t, :, None] @ S)[:, 0]
            y = (_rms(o, eps) * W.ones(p + "norm", V) * _silu(h @ W.matrix(p + "g", H * V, d).T).view(-1, H, V)).flatten(1)
        x = x + mult * (y @ W.matrix(p + "o", d, H * V).T)
        h, p = _rms(x, eps) * W.ones(f"l{i}.norm2", d), f"l{i}.mlp."
        g = torch.relu(h @ W.matrix(p + "gate", ff, d).T) * (h @ W.matrix(p + "up", ff, d).T)
        x = x + mult * (g @ W.matrix(p + "down", d, ff).T)
    return _rms(x, eps) * W.ones("final.norm", d)


def _exact_tokolorn(cfg, W, x, spans, tokens):
    d, eps, bg = cfg["width"], cfg["norm"]["eps"], cfg["embedding"]["bigram"]
    prev = torch.roll(tokens, 1)
    row = (prev * bg["mul_prev"] + tokens * bg["mul_cur"]) % bg["buckets"]
    for a, _ in spans:
        row[a] = bg["buckets"]
    x = x + W.matrix("bigram", bg["buckets"] + 1, d)[row]
    for i in _order(cfg):
        layer, p = cfg["layers"][i], f"l{i}.mix."
        m, ff = layer["mixer"], layer["mlp"]["ff"]
        h = _rms(x, eps) * W.ones(f"l{i}.norm1")
        if layer["type"] == "lightning":
            H, D, V = m["heads"], m["dim"], m["vdim"]
            q, k, v = (_silu(h @ W.matrix(p + n, H * c, d).T).view(-1, H, c) for n, c in (("q", D), ("k", D), ("v", V)))
            decay = torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE)[:, None, None]
            o = torch.empty(x.shape[0], H, V, dtype=torch.float64, device=DEVICE)
            for a, b in spans:
                S = torch.zeros(H, D, V, dtype=torch.float64, device=DEVICE)
                for t in range(a, b):
                    S = S * decay + k[t, :, :, None] * v[t, :, None]
                    o[t] = (q[t, :, None] @ S)[:, 0]
            y = _rms(o.flatten(1), eps) * W.ones(p + "norm", H * V) * torch.sigmoid(h @ W.matrix(p + "g", H * V, d).T)
            y = y @ W.matrix(p + "o", d, H * V).T
        elif layer["type"] == "attention":
            H, G, D = m["heads"], m["kv_heads"], m["dim"]
            q, k = (h @ W.matrix(p + n, c * D, d).T for n, c in (("q", H), ("k", G)))
            zero = torch.zeros(H, dtype=torch.float64, device=DEVICE)
            y = _each(spans, lambda a, b: _attend(q[a:b].view(-1, H, D), k[a:b].view(-1, G, D), k[a:b].view(-1, G, D), m["scale"],
                                                  chunk=m["mask"]["size"], sink=zero)) @ W.matrix(p + "o", d, H * D).T
        else:
            left, s, lp, rp = m["left"], m["right"], p + "left.", p + "right."
            H, G, D, I, N, R = left["heads"], left["kv_heads"], left["dim"], s["inner"], s["state"], s["dt_rank"]
            f, _ = _yarn(left["rot"]["base"], left["rot"]["dims"], None)
            q, k, v = (h @ W.matrix(lp + n, c * D, d).T for n, c in (("q", H), ("k", G), ("v", G)))
            o = _each(spans, lambda a, b: _attend(_rotate(q[a:b].view(-1, H, D), f, pairs=True),
                                                  _rotate(k[a:b].view(-1, G, D), f, pairs=True), v[a:b].view(-1, G, D), left["scale"],
                                                  window=left["mask"]["size"], cap=left["softcap"]))
            y = m["left_scale"] * ((o * torch.sigmoid(h @ W.matrix(lp + "g", H * D, d).T)) @ W.matrix(lp + "o", d, H * D).T)
            xz = h @ W.matrix(rp + "in", 2 * I, d).T
            conv, bias = W.matrix(rp + "conv", I, s["conv"]), W.vector(rp + "conv.b", I)
            xc = _silu(_each(spans, lambda a, b: _conv(xz[a:b, :I], conv, bias)))
            low = xc @ W.matrix(rp + "x", R + 2 * N, I).T
            dt = _softplus(low[:, :R] @ W.matrix(rp + "dt", I, R).T + W.vector(rp + "dt.b", I))
            A, skip = -torch.exp(W.matrix(rp + "A_log", I, N)), W.ones(rp + "D", I)
            o = torch.empty_like(xc)
            for a, b in spans:
                S = torch.zeros(I, N, dtype=torch.float64, device=DEVICE)
                for t in range(a, b):
                    S = torch.exp(dt[t, :, None] * A) * S + (dt[t] * xc[t])[:, None] * low[t, None, R:R + N]
                    o[t] = S @ low[t, R + N:] + skip * xc[t]
            y = y + m["right_scale"] * ((o * _silu(xz[:, I:])) @ W.matrix(rp + "o", d, I).T)
        x = x + y * W.ones(f"l{i}.ls1", d)
        h, p = _rms(x, eps) * W.ones(f"l{i}.norm2"), f"l{i}.mlp."
        g = torch.nn.functional.gelu(h @ W.matrix(p + "gate", ff, d).T, approximate="tanh") * (h @ W.matrix(p + "up", ff, d).T)
        x = x + (g @ W.matrix(p + "down", d, ff).T) * W.ones(f"l{i}.ls2", d)
    return _rms(x, eps) * W.ones("final.norm") * cfg["logit_scale"]


@torch.inference_mode()
def exact(case, seed):
    """Whole sequences in 64 bits; the logits of the rows that ``run`` returns, in its layout."""
    cfg, lens, toks, W = config_of(case), lengths(case), tokens_of(case, seed), _Weights(case, seed)
    if case["kind"] == "prompt":
        toks = [t[:n] for t, n in zip(toks, lens)]
    starts = [0]
    for t in toks:
        starts.append(starts[-1] + len(t))
    spans = list(zip(starts, starts[1:]))
    ids = torch.tensor([i for t in toks for i in t], device=DEVICE)
    llama, vocab = "hidden_size" in cfg, vocab_of(cfg)
    d = cfg["hidden_size"] if llama else cfg["width"]
    table = W.draw("model.embed_tokens.weight" if llama else "embed", (vocab, d)).mul_(0.02).to(W.dtype)
    x = table[ids].double()
    if llama:
        x = _exact_llama(cfg, W, x, spans)
    else:
        kind = cfg["architecture"]
        x = _exact_tokolorn(cfg, W, x, spans, ids) if kind == "Tokolorn" else {"Vabanex": _exact_vabanex, "Lupusun": _exact_lupusun}[kind](cfg, W, x, spans)
    head = table.double() if llama and cfg["tie_word_embeddings"] else W.matrix("lm_head.weight" if llama else "head", vocab, d)
    cap = cfg.get("logit_softcap")

    def logits(rows):
        z = x[rows] @ head.T
        return cap * torch.tanh(z / cap) if cap else z
    if case["kind"] == "decode":
        return logits([b - 1 for _, b in spans])
    if case["kind"] == "prompt":
        return logits(slice(None) if case["rows"] == "all" else [b - 1 for _, b in spans])
    return [logits([starts[r] + first + count - 1 for r, first, count in step if first + count >= lens[r]]) for step in serve_plan(case)]
