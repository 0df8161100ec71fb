"""What the framework's speed is measured on: layers as a program builds them from the registered parts (a mixer, a feed-forward,
an output head with its sampler, each with weights, cache and a step's batch), and whole models replayed through the engine.

A case is a dict of plain values.  ``kind`` says which layer:

  replay     a whole Qwen3 model through ``Engine.step``: unequal prompts in one step, then given tokens one by one
  attention  grouped-query attention with per-head norms and rotary positions
  latent     attention over a cached latent (one row per position for all heads)
  delta      the gated delta rule, one decay per head or per key channel
  mamba2     the Mamba-2 mixer
  lightning  linear attention with a fixed decay per head
  ffn        the SwiGLU feed-forward
  experts    silu-gated experts under a softmax router, beside a shared expert or alone
  head       final norm, head product and one draw per row

``n_seq`` sequences bring between ``short`` and ``long`` tokens each (spread evenly in an irregular order); a layer that decodes
has ``long`` = 0: every sequence brings one token after between ``held_short`` and ``held`` positions (or after a state that is
not zero).  Steps of few tokens are captured once and replayed, as the engine does with them; steps of many tokens are launched.
The sizes are those of the Qwen3 shapes and of the layers of width 2,048 and 4,096 that ``bench.py`` measures, and of the
tests' small models."""
import hashlib
import math
import random

import torch

F64 = torch.float64
CAPTURED_UP_TO = 1024       # tokens of a step that a program replays from a graph (the engine: single tokens, short prompts)
EPS = 1e-6


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest model of the configurations, in the true 32-bit engine: 4 prompts of 1 to 40 tokens and 12 tokens each;
        # what counts is latency, launches and the host
        dict(name="replay_small_f32", kind="replay", dtype="f32", layers=3, hidden=96, heads=6, kv_heads=2, head_dim=32, inter=200, vocab=384,
             n_seq=4, short=1, long=40, decode=12),
        # a batch of 8 requests to four layers of the 4B shape with its vocabulary: short unequal prompts, then 16 tokens each
        dict(name="replay_4b_bf16", kind="replay", dtype="bf16", layers=4, hidden=2560, heads=32, kv_heads=8, head_dim=128, inter=9728,
             vocab=151936, n_seq=8, short=20, long=250, decode=16),
        # attention of a prompt step, the benchmark's 2,048 tokens as three unequal prompts (4B shape)
        dict(name="attention_prompt", kind="attention", dtype="bf16", hidden=2560, heads=32, kv_heads=8, head_dim=128, n_seq=3, short=301,
             long=1200, held_short=0, held=0),
        # attention of a decode step at batch 64, unequal lengths up to the benchmark's context of 8,192 (8B shape)
        dict(name="attention_decode_64", kind="attention", dtype="bf16", hidden=4096, heads=32, kv_heads=8, head_dim=128, n_seq=64, short=0,
             long=0, held_short=2048, held=8191),
        # feed-forward of a prompt of 1,000 tokens in the 32B shape: the largest products
        dict(name="ffn_32b_bf16", kind="ffn", dtype="bf16", hidden=5120, inter=25600, tokens=1000),
        # the same layer of the 4B shape in the 32-bit engine (the check run), a prompt of 500 tokens
        dict(name="ffn_4b_f32", kind="ffn", dtype="f32", hidden=2560, inter=9728, tokens=500),
        # 64 sequences' logits and draws (8B shape, the usual sampling options)
        dict(name="head_64", kind="head", dtype="bf16", hidden=4096, vocab=151936, rows=64, top_k=20, top_p=0.95),
        # a mixture of sixteen experts, two per token, beside a shared one: a prompt of 777 tokens
        dict(name="experts_prompt", kind="experts", dtype="bf16", hidden=2048, inter=1024, experts=16, top=2, shared=1024, tokens=777),
        # linear attention with the delta rule over two unequal prompts
        dict(name="delta_prompt", kind="delta", dtype="bf16", hidden=2048, heads=16, qk_heads=16, dim=128, decay="head", n_seq=2, short=700,
             long=1348, fresh=True),
        # Mamba-2 over one prompt of 2,048 tokens
        dict(name="mamba2_prompt", kind="mamba2", dtype="bf16", hidden=2048, heads=64, vdim=64, state=128, groups=8, n_seq=1, short=2048,
             long=2048, fresh=True),
        # latent attention of a decode step, 16 sequences of up to 4,096 positions
        dict(name="latent_decode_16", kind="latent", dtype="bf16", hidden=2048, heads=16, dim=64, rot=64, vdim=128, rank=512, n_seq=16,
             short=0, long=0, held_short=1000, held=4000),
        # linear attention with a state per sequence, a decode step of 32 sequences
        dict(name="lightning_decode_32", kind="lightning", dtype="bf16", hidden=2048, heads=16, dim=128, vdim=128, n_seq=32, short=1, long=1,
             fresh=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the kinds, sizes over the ranges that the configurations and ``bench.py``'s layers span."""
    kind = rng.choice(["replay", "attention", "attention", "latent", "delta", "delta", "mamba2", "lightning", "ffn", "ffn", "experts", "head"])
    c = dict(kind=kind, dtype="f32" if rng.random() < 0.3 else "bf16")
    wide = c["dtype"] == "bf16"
    if kind == "replay":
        hd = rng.choice([32, 64, 128])
        kv = rng.choice([1, 2, 4])
        c.update(layers=rng.randint(1, 4), hidden=8 * _log(rng, 8, 256 if wide else 128), heads=kv * rng.choice([1, 2, 4]), kv_heads=kv, head_dim=hd,
                 inter=8 * _log(rng, 16, 512 if wide else 128), vocab=_log(rng, 256, 32000), n_seq=_log(rng, 1, 16), short=1,
                 long=_log(rng, 2, 300), decode=rng.randint(1, 16))
        return c
    decoding = rng.random() < 0.5
    if kind in ("attention", "latent"):
        # a prompt, a prompt's next piece after what the cache holds, or single tokens
        if decoding:
            n_seq, held = _log(rng, 1, 64 if wide else 16), _log(rng, 16, 8000 if wide else 2000)
            c.update(n_seq=n_seq, short=0, long=0, held_short=_log(rng, 1, held), held=held)
        else:
            n_seq, long = rng.randint(1, 4), _log(rng, 8, 1200 if wide else 300)
            held = 0 if rng.random() < 0.6 else _log(rng, 10, 1500)
            c.update(n_seq=n_seq, short=_log(rng, 1, long), long=long, held_short=held // 3, held=held)
        if kind == "attention":
            hd = rng.choice([64, 128, 128])
            heads, kv = rng.choice([(16, 8), (32, 8), (40, 8), (24, 4), (8, 2)])
            c.update(hidden=rng.choice([1024, 2048, 2560, 4096] if wide else [512, 1024]), heads=heads, kv_heads=kv, head_dim=hd)
        else:
            c.update(hidden=rng.choice([1024, 2048, 4096] if wide else [512, 1024]), heads=rng.choice([8, 16, 32] if wide else [8]),
                     dim=rng.choice([32, 64, 128]), rot=rng.choice([32, 64]), vdim=rng.choice([64, 128]), rank=rng.choice([256, 512]))
        return c
    if kind in ("delta", "mamba2", "lightning"):
        if decoding:
            c.update(n_seq=_log(rng, 1, 64), short=1, long=1, fresh=False)
        else:
            long = _log(rng, 16, 2048 if wide else 700)
            c.update(n_seq=rng.randint(1, 3), short=_log(rng, 1, long), long=long, fresh=rng.random() < 0.6)
        width = rng.choice([1024, 2048] if wide else [512, 1024])
        c["hidden"] = width
        if kind == "delta":
            dim = rng.choice([64, 128, 128])
            heads = width // dim
            c.update(heads=heads, qk_heads=heads // rng.choice([1, 2]), dim=dim, decay=rng.choice(["head", "channel"]))
        elif kind == "mamba2":
            vdim = rng.choice([32, 64])
            c.update(heads=2 * width // vdim, vdim=vdim, state=rng.choice([64, 128]), groups=rng.choice([1, 4, 8]))
        else:
            dim = rng.choice([64, 128])
            c.update(heads=width // dim, dim=dim, vdim=dim)
        return c
    if kind == "ffn":
        c.update(hidden=8 * _log(rng, 64, 512 if wide else 256), inter=8 * _log(rng, 128, 1600 if wide else 800), tokens=_log(rng, 1, 3000 if wide else 600))
    elif kind == "experts":
        experts = rng.choice([8, 16, 32])
        c.update(hidden=rng.choice([1024, 2048]), inter=8 * _log(rng, 32, 160), experts=experts, top=rng.choice([1, 2, 4]),
                 shared=rng.choice([0, 512]), tokens=_log(rng, 1, 2500 if wide else 300))
    else:
        c.update(hidden=rng.choice([1024, 2048, 2560, 4096]), vocab=_log(rng, 1000, 151936), rows=_log(rng, 1, 64 if wide else 8),
                 top_k=rng.choice([0, 20, 50]), top_p=rng.choice([1.0, 0.95, 0.9]))
    return c


# ---------------------------------------------------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------------------------------------------------
def _normal(seed, name, shape, std=1.0, mean=0.0, dtype=torch.float32):
    """float32 values rounded to ``dtype``: what a checkpoint of that type holds."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=g)
    return t.to(dtype)


def _dtype(c):
    return torch.float32 if c["dtype"] == "f32" else torch.bfloat16


def _spread(n, lo, hi, step=0.6180339887498949):
    """n numbers from lo to hi: the largest, the smallest, and irregularly between."""
    out = [lo + int(round((hi - lo) * ((i * step) % 1.0))) for i in range(n)]
    out[0] = hi
    if n > 1:
        out[1] = lo
    return out


def _step(c):
    """(new tokens per sequence, positions held per sequence)."""
    if c["kind"] in ("attention", "latent"):
        held = _spread(c["n_seq"], c["held_short"], c["held"])
        new = [1] * c["n_seq"] if c["long"] == 0 else _spread(c["n_seq"], c["short"], c["long"], 0.7548776662466927)
        return new, held
    return _spread(c["n_seq"], c["short"], c["long"]), [0] * c["n_seq"]


def _weights(c, seed):
    """The layer's tensors under its parts' names.  Projections of unit inputs have about unit variance; norms, decays and step
    sizes are spread as trained ones are."""
    dt, h = _dtype(c), c.get("hidden")
    n = lambda name, shape, std, mean=0.0: _normal(seed, name, shape, std, mean, dt)
    lin = lambda name, out, inn, gain=1.0: n(name, (out, inn), gain / math.sqrt(inn))
    k = c["kind"]
    w = {}
    if k == "attention":
        H, G, d = c["heads"], c["kv_heads"], c["head_dim"]
        w = {"q_proj.weight": lin("q", H * d, h), "k_proj.weight": lin("k", G * d, h), "v_proj.weight": lin("v", G * d, h),
             "o_proj.weight": lin("o", h, H * d), "q_norm.weight": n("qn", (d,), 0.1, 1.0), "k_norm.weight": n("kn", (d,), 0.1, 1.0)}
    elif k == "latent":
        H, d, r, vd, rank = c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"]
        w = {"q": lin("q", H * (d + r), h), "dkv": lin("dkv", rank + r, h), "dkv.norm": n("dn", (rank,), 0.1, 1.0), "uk": lin("uk", H * d, rank),
             "uv": lin("uv", H * vd, rank), "o": lin("o", h, H * vd)}
    elif k == "delta":
        H, G, d = c["heads"], c["qk_heads"], c["dim"]
        w = {"q": lin("q", G * d, h), "k": lin("k", G * d, h), "v": lin("v", H * d, h), "b": lin("b", H, h), "A_log": n("A", (H,), 0.5),
             "norm": n("norm", (d,), 0.1, 1.0), "o": lin("o", h, H * d)}
        for x, rows in (("q", G * d), ("k", G * d), ("v", H * d)):
            w[x + ".conv"] = n(x + "c", (rows, 4), 0.5)
        if c["decay"] == "head":
            w.update({"a": lin("a", H, h), "dt_bias": n("dt", (H,), 1.0, -2.0), "g": lin("g", H * d, h)})
        else:
            r = max(8, d // 2)
            w.update({"a1": lin("a1", r, h), "a2": lin("a2", H * d, r), "dt_bias": n("dt", (H * d,), 1.0, -2.0), "g1": lin("g1", r, h),
                      "g2": lin("g2", H * d, r)})
    elif k == "mamba2":
        inner, gn = c["heads"] * c["vdim"], c["groups"] * c["state"]
        w = {"in": lin("in", 2 * inner + 2 * gn + c["heads"], h), "conv": n("conv", (inner + 2 * gn, 4), 0.4), "conv.b": n("cb", (inner + 2 * gn,), 0.1),
             "dt_bias": n("dt", (c["heads"],), 0.5, -1.0), "A_log": n("A", (c["heads"],), 0.5), "D": n("D", (c["heads"],), 0.2, 1.0),
             "norm": n("norm", (inner,), 0.1, 1.0), "o": lin("o", h, inner)}
    elif k == "lightning":
        qk, vd = c["heads"] * c["dim"], c["heads"] * c["vdim"]
        w = {"q": lin("q", qk, h), "k": lin("k", qk, h), "v": lin("v", vd, h), "g": lin("g", vd, h), "o": lin("o", h, vd),
             "norm": n("norm", (vd,), 0.1, 1.0)}
    elif k == "ffn":
        w = {"gate_proj.weight": lin("gate", c["inter"], h), "up_proj.weight": lin("up", c["inter"], h), "down_proj.weight": lin("down", h, c["inter"])}
    elif k == "experts":
        for e in range(c["experts"]):
            w.update({f"e{e}.gate": lin(f"g{e}", c["inter"], h), f"e{e}.up": lin(f"u{e}", c["inter"], h), f"e{e}.down": lin(f"d{e}", h, c["inter"])})
        w["router"] = lin("router", c["experts"], h)
        if c["shared"]:
            w.update({"shared.gate": lin("sg", c["shared"], h), "shared.up": lin("su", c["shared"], h), "shared.down": lin("sd", h, c["shared"])})
    elif k == "head":
        w = {"model.norm.weight": n("norm", (h,), 0.1, 1.0), "lm_head.weight": lin("head", c["vocab"], h, 2.0)}
    elif k == "replay":
        H, G, d = c["heads"], c["kv_heads"], c["head_dim"]
        w["model.embed_tokens.weight"] = n("embed", (c["vocab"], h), 1.0 / math.sqrt(h))
        w["model.norm.weight"] = n("final", (h,), 0.1, 1.0)
        for i in range(c["layers"]):
            p = f"model.layers.{i}."
            for name, rows, cols in (("self_attn.q_proj", H * d, h), ("self_attn.k_proj", G * d, h), ("self_attn.v_proj", G * d, h),
                                     ("self_attn.o_proj", h, H * d), ("mlp.gate_proj", c["inter"], h), ("mlp.up_proj", c["inter"], h),
                                     ("mlp.down_proj", h, c["inter"])):
                w[p + name + ".weight"] = lin(f"{i}{name}", rows, cols)
            for name, size in (("self_attn.q_norm", d), ("self_attn.k_norm", d), ("input_layernorm", h), ("post_attention_layernorm", h)):
                w[p + name + ".weight"] = n(f"{i}{name}", (size,), 0.1, 1.0)
    return w


def _x(c, seed, rows):
    """Rows as a norm leaves them."""
    return _normal(seed, "x", (rows, c["hidden"]), 1.0, 0.0, _dtype(c))


def _held(c, seed, i, n):
    """What the cache holds of sequence i: keys and values [kv_heads, n, d], or the latent's rows [1, n, rank + rot]."""
    dt = _dtype(c)
    if c["kind"] == "latent":
        return _normal(seed, f"c{i}", (1, n, c["rank"] + c["rot"]), 1.0, 0.0, dt), None
    shape = (c["kv_heads"], n, c["head_dim"])
    return _normal(seed, f"k{i}", shape, 1.0, 0.0, dt), _normal(seed, f"v{i}", shape, 1.0, 0.0, dt)


def _state(c, seed):
    """(the convolution's last inputs [n_seq, taps - 1, channels] or None, the state [n_seq, ...]), zero for sequences that begin."""
    n = c["n_seq"]
    if c["kind"] == "delta":
        conv, s = (n, 3, (2 * c["qk_heads"] + c["heads"]) * c["dim"]), (n, c["heads"], c["dim"], c["dim"])
    elif c["kind"] == "mamba2":
        conv, s = (n, 3, c["heads"] * c["vdim"] + 2 * c["groups"] * c["state"]), (n, c["heads"], c["vdim"], c["state"])
    else:
        conv, s = None, (n, c["heads"], c["dim"], c["vdim"])
    if c["fresh"]:
        return (torch.zeros(conv, device="cuda") if conv else None), torch.zeros(s, device="cuda")
    return (_normal(seed, "tail", conv) if conv else None), _normal(seed, "S", s, 0.3)


def _decays(c):
    return [1.0 - 2.0 ** (-2.0 - 6.0 * i / max(1, c["heads"] - 1)) for i in range(c["heads"])]


def _tokens(c, seed):
    """(prompts, the tokens that follow) of a replay."""
    r = random.Random(seed * 7919 + 11)
    lens = _spread(c["n_seq"], c["short"], c["long"])
    return [[r.randrange(c["vocab"]) for _ in range(n)] for n in lens], [[r.randrange(c["vocab"]) for _ in range(c["decode"])] for _ in lens]


# ---------------------------------------------------------------------------------------------------------------------
# the framework's side
# ---------------------------------------------------------------------------------------------------------------------
def _mixer(c, ctx):
    from toyinfer_b200.parts.base import PartSpec, build_part
    k = c["kind"]
    if k == "attention":
        p = dict(n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["head_dim"], qk_norm_eps=EPS, position="rope")
        return build_part("mixer", PartSpec("gqa_attention", p), ctx, "")
    if k == "latent":
        p = dict(n_heads=c["heads"], dim=c["dim"], rot_dim=c["rot"], vdim=c["vdim"], kv_rank=c["rank"], scale=(c["dim"] + c["rot"]) ** -0.5,
                 eps=EPS, position="rope", sinks=False)
        return build_part("mixer", PartSpec("latent_attention", p), ctx, "")
    if k == "delta":
        p = dict(n_heads=c["heads"], n_qk_heads=c["qk_heads"], dim=c["dim"], vdim=c["dim"], conv=4, eps=EPS)
        return build_part("mixer", PartSpec("head_delta" if c["decay"] == "head" else "channel_delta", p), ctx, "")
    if k == "mamba2":
        p = dict(n_heads=c["heads"], vdim=c["vdim"], state=c["state"], groups=c["groups"], conv=4, norm_groups=c["groups"], eps=EPS)
        return build_part("mixer", PartSpec("mamba2", p), ctx, "")
    p = dict(n_heads=c["heads"], dim=c["dim"], vdim=c["vdim"], decay=_decays(c), eps=EPS)
    return build_part("mixer", PartSpec("lightning", p), ctx, "")


def _fill(c, seed, cache, mem, held):
    """Puts what the sequences hold already into the layer's memory."""
    if hasattr(mem, "state"):
        tail, S = _state(c, seed)
        n = c["n_seq"]
        rows = mem.state[:n].view(n, -1)
        at = 0
        if tail is not None:
            at = tail[0].numel()
            rows[:, :at] = tail.reshape(n, -1)
        rows[:, at:] = S.reshape(n, -1)
        return
    for i, n in enumerate(held):
        if n == 0:
            continue
        page = mem.page_size
        pages = -(-n // page)
        at = mem.page_table[i, :pages].long()
        for rows, store in zip(_held(c, seed, i, n), (mem.k_pages, mem.v_pages)):
            if rows is not None:
                heads, _, d = rows.shape
                full = torch.zeros((heads, pages * page, d), dtype=rows.dtype, device=rows.device)
                full[:, :n] = rows
                store[at] = full.view(heads, pages, page, d).permute(1, 0, 2, 3).contiguous()


def _layer(c, seed):
    """A mixer with its weights, memory and batch."""
    from toyinfer_b200.cache import CacheManager
    from toyinfer_b200.engine.batch import BatchBuffers, fill_batch
    from toyinfer_b200.parts.base import BuildContext, PartSpec, build_part
    dt, dev = _dtype(c), torch.device("cuda")
    new, held = _step(c)
    longest = max(a + b for a, b in zip(new, held))
    ctx = BuildContext(dtype=dt, device=dev, hidden_size=c["hidden"])
    if c["kind"] in ("attention", "latent"):
        dim = c["head_dim"] if c["kind"] == "attention" else c["rot"]
        ctx.positions["rope"] = build_part("position", PartSpec("rotary_half", {"dim": dim, "theta": 1e6, "max_positions": longest}), ctx, "")
    mixer = _mixer(c, ctx)
    mixer.check_kernels(dt)
    mixer.bind(_weights(c, seed))
    need = sum(-(-(a + b) // 64) * 64 for a, b in zip(new, held))
    cache = CacheManager([mixer.memory_request()], need, c["n_seq"], longest, dt, dev)
    mem = cache.views(1)[0]
    slots = [cache.allocate_slot() for _ in new]
    for s, n in zip(slots, held):
        if n:
            cache.reserve(s, n // 64 * 64)
    for s, a, b in zip(slots, new, held):       # the pages that this step writes come last, side by side
        cache.reserve(s, a + b)
    cache.flush()
    if all(n == 1 for n in new) and (any(held) or hasattr(mem, "state")):
        mode = "extend"
    else:
        mode = "mixed" if any(held) or not c.get("fresh", True) else "start"
    buf = BatchBuffers(len(new), sum(new), dev)
    starts = [b if hasattr(mem, "k_pages") else (0 if c["fresh"] else 100) for b in held]
    batch = fill_batch(buf, mode, slots, starts, [[0] * n for n in new], cache.scratch_slot, longest)
    x = _x(c, seed, sum(new))
    if hasattr(mem, "state"):
        after = [mem.state[:c["n_seq"]]]
    else:                                        # the pages that hold the step's keys and values
        first = min(int(cache.kv_groups[0].table_host[s, b // 64]) for s, b in zip(slots, held))
        after = [t[first:] for t in (mem.k_pages, mem.v_pages) if t is not None]
    return dict(forward=lambda: mixer.forward(x, batch, mem, {}), after=after, tokens=sum(new), keep=(mixer, cache, buf, batch, x),
                fill=lambda: _fill(c, seed, cache, mem, held))


def _plain_part(c, seed):
    """A feed-forward, or the head with its sampler."""
    from toyinfer_b200.parts.base import BuildContext, PartSpec, build_part
    dt = _dtype(c)
    ctx = BuildContext(dtype=dt, device=torch.device("cuda"), hidden_size=c["hidden"])
    if c["kind"] == "head":
        from toyinfer_b200.sampling import Sampler, SamplingParams
        norm = PartSpec("rmsnorm", {"size": c["hidden"], "eps": EPS})
        part = build_part("head", PartSpec("linear", {"vocab_size": c["vocab"], "norm": norm}), ctx, "")
        part.bind(_weights(c, seed))
        sampler = Sampler(SamplingParams(temperature=0.7, top_k=c["top_k"], top_p=c["top_p"], seed=seed), "cuda")
        h, delta = _x(c, seed, c["rows"]), _normal(seed, "delta", (c["rows"], c["hidden"]), 1.0, 0.0, dt)
        rows = torch.arange(c["rows"], dtype=torch.int32, device="cuda")
        keys, steps = list(range(c["rows"])), [5] * c["rows"]

        def forward():
            logits = part.forward(h, delta, rows)
            return logits, sampler.sample(logits, keys, steps)

        return dict(forward=forward, after=[], tokens=CAPTURED_UP_TO + 1, keep=part, fill=lambda: None)      # (the sampler uploads: launched)
    if c["kind"] == "ffn":
        part = build_part("feed_forward", PartSpec("swiglu", {"intermediate_size": c["inter"]}), ctx, "")
    else:
        part = build_part("feed_forward", PartSpec("softmax_moe", dict(n_experts=c["experts"], top=c["top"], intermediate_size=c["inter"],
                                                                       correction=False, shared_size=c["shared"])), ctx, "")
    part.check_kernels(dt)
    part.bind(_weights(c, seed))
    x = _x(c, seed, c["tokens"])
    return dict(forward=lambda: part.forward(x, None), after=[], tokens=c["tokens"], keep=(part, x), fill=lambda: None)


def _replay(c, seed):
    from toyinfer_b200.config.registry import architecture_of
    from toyinfer_b200.engine import Engine
    from toyinfer_b200.parts.model import DecoderModel
    import toyinfer_b200.models  # noqa: F401  (registers the architectures)
    cfg = {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": c["layers"], "hidden_size": c["hidden"], "num_attention_heads": c["heads"],
           "num_key_value_heads": c["kv_heads"], "head_dim": c["head_dim"], "intermediate_size": c["inter"], "vocab_size": c["vocab"],
           "rope_theta": 1e6, "rms_norm_eps": EPS, "max_position_embeddings": 1024, "tie_word_embeddings": True}
    arch = architecture_of(cfg)
    model = DecoderModel(arch.describe(arch.config_cls.from_dict(cfg)), _dtype(c), "cuda")
    model.bind(_weights(c, seed))
    engine = Engine(model, max_tokens=c["n_seq"] * 384, max_batch=c["n_seq"], max_seq_len=384)
    prompts, after = _tokens(c, seed)
    rows = torch.empty((c["decode"] + 1, c["n_seq"], c["vocab"]), dtype=torch.float32, device="cuda")
    return dict(engine=engine, prompts=prompts, after=after, rows=rows)


def prepare(case, seed):
    if case["kind"] == "replay":
        s = _replay(case, seed)
        for _ in range(2):           # an engine that has served requests of these shapes
            run(s)
        return s
    s = _plain_part(case, seed) if case["kind"] in ("ffn", "experts", "head") else _layer(case, seed)
    s["graph"] = None
    if s["tokens"] <= CAPTURED_UP_TO:
        s["forward"]()               # kernels' one-time set-up stays outside the capture
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = s["forward"]()
    s["fill"]()
    return s


def run(state):
    if "engine" in state:
        engine, rows = state["engine"], state["rows"]
        slots = [engine.new_sequence() for _ in state["prompts"]]
        rows[0].copy_(engine.step(list(zip(slots, state["prompts"]))))
        for t in range(rows.shape[0] - 1):
            rows[t + 1].copy_(engine.step([(s, [a[t]]) for s, a in zip(slots, state["after"])]))
        for s in slots:
            engine.end_sequence(s)
        return rows
    if state["graph"] is None:
        out = state["forward"]()
    else:
        state["graph"].replay()
        out = state["out"]
    return [out] + state["after"]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    c, e = case, 4 if case["dtype"] == "f32" else 2
    h, k = c.get("hidden"), c["kind"]
    if k == "replay":
        H, G, d = c["heads"], c["kv_heads"], c["head_dim"]
        per_layer = h * (2 * H + 2 * G) * d + 3 * h * c["inter"]
        lens = _spread(c["n_seq"], c["short"], c["long"])
        tokens = sum(lens) + c["n_seq"] * c["decode"]
        steps = c["decode"] + 1
        pairs = sum((n + c["decode"]) * (n + c["decode"] + 1) // 2 for n in lens)
        kv = sum(sum(range(n, n + c["decode"])) for n in lens) * 2 * G * d
        flops = 2 * tokens * per_layer * c["layers"] + 2 * steps * c["n_seq"] * h * c["vocab"] + 4 * pairs * H * d * c["layers"]
        return {"bytes": e * (steps * (per_layer * c["layers"] + h * c["vocab"]) + c["layers"] * kv) + 4 * steps * c["n_seq"] * c["vocab"], "flops": flops}
    if k == "ffn":
        return {"bytes": e * (3 * h * c["inter"] + 2 * c["tokens"] * h), "flops": 6 * c["tokens"] * h * c["inter"]}
    if k == "experts":
        used = min(c["experts"], c["tokens"] * c["top"])
        return {"bytes": e * (3 * h * (c["inter"] * used + c["shared"]) + h * c["experts"] + 2 * c["tokens"] * h),
                "flops": 2 * c["tokens"] * h * (3 * c["inter"] * c["top"] + 3 * c["shared"] + c["experts"])}
    if k == "head":
        return {"bytes": e * (h * c["vocab"] + 2 * c["rows"] * h) + 4 * c["rows"] * c["vocab"], "flops": 2 * c["rows"] * h * c["vocab"]}
    new, held = _step(c)
    M = sum(new)
    pairs = sum(n * p + n * (n + 1) // 2 for n, p in zip(new, held))
    if k == "attention":
        H, G, d = c["heads"], c["kv_heads"], c["head_dim"]
        weights = h * (2 * H + 2 * G) * d
        return {"bytes": e * (weights + 2 * M * h + 2 * G * d * (sum(held) + M)), "flops": 2 * M * weights + 4 * pairs * H * d}
    if k == "latent":
        H, row = c["heads"], c["rank"] + c["rot"]
        weights = h * (H * (c["dim"] + c["rot"]) + row + H * c["vdim"]) + c["rank"] * H * (c["dim"] + c["vdim"])
        # scores and sums either over keys and values per head, or over the latent's rows
        attend = min(2 * pairs * H * (c["dim"] + c["rot"] + c["vdim"]) + 2 * (M + sum(held)) * c["rank"] * H * (c["dim"] + c["vdim"]),
                     2 * pairs * H * (row + c["rank"]) + 2 * M * c["rank"] * H * (c["dim"] + c["vdim"]))
        return {"bytes": e * (weights + 2 * M * h + row * (sum(held) + M)),
                "flops": 2 * M * (weights - c["rank"] * H * (c["dim"] + c["vdim"])) + attend}
    if k == "delta":
        H, G, d = c["heads"], c["qk_heads"], c["dim"]
        gates = h * (H + H * d) if c["decay"] == "head" else (h + H * d) * 2 * max(8, d // 2)
        weights = h * (2 * G * d + 2 * H * d + H) + gates
        state, step = H * d * d, 7 * H * d * d
    elif k == "mamba2":
        inner, gn = c["heads"] * c["vdim"], c["groups"] * c["state"]
        weights = h * (3 * inner + 2 * gn + c["heads"])
        state, step = inner * c["state"], 5 * inner * c["state"]
    else:
        H = c["heads"]
        weights = h * H * (2 * c["dim"] + 3 * c["vdim"])
        state, step = H * c["dim"] * c["vdim"], 5 * H * c["dim"] * c["vdim"]
    return {"bytes": e * (weights + 2 * M * h) + 4 * 2 * c["n_seq"] * state, "flops": M * (2 * weights + step)}


def tolerance(case):
    """About four times the error against ``exact``: 2e-7 to 7e-7 in the 32-bit engine; in bfloat16, whose every result is rounded
    to 2^-9, 0.0035 to 0.0045 for a layer and 0.012 for the logits after four of them."""
    if case["dtype"] == "f32":
        return {"rel": 4e-6, "max": 1e-4, "differ": 0.01}
    if case["kind"] == "replay":
        return {"rel": 0.03, "max": 0.4, "differ": 0.01}
    return {"rel": 0.016, "max": 0.25, "differ": 0.01}


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _silu(x):
    return x / (1.0 + torch.exp(-x))


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _turn(x, pos):
    """x [T, heads, d], the pairs (i, i + d / 2) turned by position * 1e6^(-2 i / d)."""
    half = x.shape[-1] // 2
    f = 1e6 ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / x.shape[-1])
    a = pos[:, None].to(F64) * f[None, :]
    cos, sin = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], dim=-1)


def _attend(q, k, v, start, scale):
    """q [T, H, d] at positions start.., k [G, P, d] and v [G, P, dv] at positions 0.. -> [T, H * dv]."""
    T, H = q.shape[:2]
    G, P = k.shape[:2]
    out = torch.empty((T, H, v.shape[2]), dtype=F64, device=q.device)
    for t0 in range(0, T, 512):
        n = min(512, T - t0)
        seen = torch.arange(P, device=q.device)[None, :] <= (start + t0 + torch.arange(n, device=q.device))[:, None]
        for g in range(G):
            heads = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("thd,pd->htp", q[t0:t0 + n, heads], k[g]) * scale
            s = s.masked_fill(~seen[None], float("-inf"))
            out[t0:t0 + n, heads] = torch.einsum("htp,pv->thv", torch.softmax(s, dim=-1), v[g])
    return out.reshape(T, -1)


def _exact_attention(c, w, x, seed):
    new, held = _step(c)
    H, G, d = c["heads"], c["kv_heads"], c["head_dim"]
    out, at = [], 0
    for i, (n, p) in enumerate(zip(new, held)):
        z = x[at:at + n]
        at += n
        pos = p + torch.arange(n, device="cuda")
        q = _turn(_rms((z @ w["q_proj.weight"].T).view(n, H, d), w["q_norm.weight"]), pos)
        k = _turn(_rms((z @ w["k_proj.weight"].T).view(n, G, d), w["k_norm.weight"]), pos).transpose(0, 1)
        v = (z @ w["v_proj.weight"].T).view(n, G, d).transpose(0, 1)
        if p:
            kh, vh = _held(c, seed, i, p)
            k, v = torch.cat([kh.to(F64), k], dim=1), torch.cat([vh.to(F64), v], dim=1)
        out.append(_attend(q, k, v, p, d ** -0.5) @ w["o_proj.weight"].T)
    return [torch.cat(out), None, None]


def _exact_latent(c, w, x, seed):
    new, held = _step(c)
    H, d, r, vd, rank = c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"]
    out, at = [], 0
    for i, (n, p) in enumerate(zip(new, held)):
        z = x[at:at + n]
        at += n
        pos = p + torch.arange(n, device="cuda")
        q = (z @ w["q"].T).view(n, H, d + r)
        q = torch.cat([q[..., :d], _turn(q[..., d:], pos)], dim=-1)
        down = z @ w["dkv"].T
        rows = torch.cat([_rms(down[:, :rank], w["dkv.norm"]), _turn(down[:, None, rank:], pos)[:, 0]], dim=1)
        if p:
            rows = torch.cat([_held(c, seed, i, p)[0][0].to(F64), rows])
        lat, turned = rows[:, :rank], rows[:, rank:]
        key = torch.cat([(lat @ w["uk"].T).view(-1, H, d), turned[:, None, :].expand(-1, H, -1)], dim=-1).transpose(0, 1)
        val = (lat @ w["uv"].T).view(-1, H, vd).transpose(0, 1)
        out.append(_attend(q, key, val, p, (d + r) ** -0.5) @ w["o"].T)
    return [torch.cat(out), None]


def _conv(z, tail, taps, bias=None):
    """z [T, C] after the rows ``tail`` [taps - 1, C] -> (silu of the causal convolution, the last taps - 1 inputs)."""
    rows = torch.cat([tail, z])
    n = taps.shape[1]
    y = sum(rows[j:j + z.shape[0]] * taps[:, j] for j in range(n))
    return _silu(y if bias is None else y + bias), rows[-(n - 1):]


def _exact_recurrent(c, w, x, seed):
    new, _ = _step(c)
    tails, states = _state(c, seed)
    out, left = [], []
    at = 0
    k = c["kind"]
    for i, n in enumerate(new):
        z = x[at:at + n]
        at += n
        S = states[i].to(F64)
        tail = tails[i].to(F64) if tails is not None else None
        o = []
        if k == "delta":
            H, G, d = c["heads"], c["qk_heads"], c["dim"]
            proj = torch.cat([z @ w["q"].T, z @ w["k"].T, z @ w["v"].T], dim=1)
            u, tail = _conv(proj, tail, torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]))
            unit = lambda a: a / torch.sqrt((a * a).sum(dim=-1, keepdim=True) + 1e-6)
            q = (unit(u[:, :G * d].view(n, G, d)) * d ** -0.5).repeat_interleave(H // G, dim=1)
            kk = unit(u[:, G * d:2 * G * d].view(n, G, d)).repeat_interleave(H // G, dim=1)
            v = u[:, 2 * G * d:].view(n, H, d)
            beta = torch.sigmoid(z @ w["b"].T)
            if c["decay"] == "head":
                g = torch.exp(-torch.exp(w["A_log"]) * _softplus(z @ w["a"].T + w["dt_bias"]))[:, :, None].expand(n, H, d)
                gate = _silu(z @ w["g"].T)
            else:
                g = torch.exp(-torch.exp(w["A_log"])[:, None] * _softplus((z @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(n, H, d))
                gate = torch.sigmoid((z @ w["g1"].T) @ w["g2"].T)
            for t in range(n):
                S = g[t, :, :, None] * S
                e = beta[t, :, None] * (v[t] - torch.bmm(kk[t, :, None], S)[:, 0])
                S = torch.baddbmm(S, kk[t, :, :, None], e[:, None])
                o.append(torch.bmm(q[t, :, None], S)[:, 0])
            y = _rms(torch.stack(o), w["norm"]).reshape(n, H * d) * gate
        elif k == "mamba2":
            H, vd, N, G = c["heads"], c["vdim"], c["state"], c["groups"]
            inner, gn = H * vd, G * N
            proj = z @ w["in"].T
            u, tail = _conv(proj[:, inner:2 * inner + 2 * gn], tail, w["conv"], w["conv.b"])
            dt = _softplus(proj[:, 2 * inner + 2 * gn:] + w["dt_bias"])
            a = torch.exp(-torch.exp(w["A_log"]) * dt)
            v = u[:, :inner].view(n, H, vd)
            B = u[:, inner:inner + gn].view(n, G, N).repeat_interleave(H // G, dim=1)
            C = u[:, inner + gn:].view(n, G, N).repeat_interleave(H // G, dim=1)
            for t in range(n):
                S = torch.baddbmm(S * a[t, :, None, None], (dt[t, :, None] * v[t])[:, :, None], B[t, :, None])
                o.append(torch.bmm(S, C[t, :, :, None])[:, :, 0])
            y = (torch.stack(o) + w["D"][:, None] * v).reshape(n, inner) * _silu(proj[:, :inner])
            y = _rms(y.view(n, G, inner // G)).reshape(n, inner) * w["norm"]
        else:
            H, d, vd = c["heads"], c["dim"], c["vdim"]
            q, kk, v = (_silu(z @ w[m].T).view(n, H, -1) for m in "qkv")
            decay = torch.tensor(_decays(c), dtype=F64, device="cuda")[:, None, None]
            for t in range(n):
                S = torch.baddbmm(S * decay, kk[t, :, :, None], v[t, :, None])
                o.append(torch.bmm(q[t, :, None], S)[:, 0])
            y = _rms(torch.stack(o).reshape(n, H * vd), w["norm"]) * torch.sigmoid(z @ w["g"].T)
        out.append(y @ w["o"].T)
        left.append(S.reshape(-1) if tail is None else torch.cat([tail.reshape(-1), S.reshape(-1)]))
    after = torch.stack(left)
    return [torch.cat(out), after.view(states.shape) if tails is None else after]


def _exact_experts(c, w, x):
    z = x @ w["router"].T
    best, chosen = torch.topk(z, c["top"], dim=1)
    weight = torch.zeros_like(z).scatter_(1, chosen, torch.softmax(best, dim=1))
    part = lambda r, p: (_silu(r @ w[p + "gate"].T) * (r @ w[p + "up"].T)) @ w[p + "down"].T
    y = part(x, "shared.") if c["shared"] else torch.zeros_like(x)
    for e in range(c["experts"]):
        who = weight[:, e].nonzero()[:, 0]
        if who.numel():
            y[who] += weight[who, e, None] * part(x[who], f"e{e}.")
    return [y]


def _exact_replay(c, w, seed):
    H, G, d = c["heads"], c["kv_heads"], c["head_dim"]
    prompts, after = _tokens(c, seed)
    E = w["model.embed_tokens.weight"].to(F64)
    out = torch.empty((c["decode"] + 1, c["n_seq"], c["vocab"]), dtype=F64, device="cuda")
    for i, (p, a) in enumerate(zip(prompts, after)):
        ids = p + a
        n = len(ids)
        pos = torch.arange(n, device="cuda")
        x = E[torch.tensor(ids, device="cuda")]
        for layer in range(c["layers"]):
            t = lambda name: w[f"model.layers.{layer}.{name}.weight"].to(F64)
            z = _rms(x, t("input_layernorm"))
            q = _turn(_rms((z @ t("self_attn.q_proj").T).view(n, H, d), t("self_attn.q_norm")), pos)
            k = _turn(_rms((z @ t("self_attn.k_proj").T).view(n, G, d), t("self_attn.k_norm")), pos).transpose(0, 1)
            v = (z @ t("self_attn.v_proj").T).view(n, G, d).transpose(0, 1)
            x = x + _attend(q, k, v, 0, d ** -0.5) @ t("self_attn.o_proj").T
            z = _rms(x, t("post_attention_layernorm"))
            x = x + (_silu(z @ t("mlp.gate_proj").T) * (z @ t("mlp.up_proj").T)) @ t("mlp.down_proj").T
        out[:, i] = _rms(x[len(p) - 1:], w["model.norm.weight"].to(F64)) @ E.T
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "replay":
        return _exact_replay(c, _weights(c, seed), seed)
    w = {k: v.to(F64) for k, v in _weights(c, seed).items()}
    if c["kind"] == "head":
        h = _x(c, seed, c["rows"]).to(F64) + _normal(seed, "delta", (c["rows"], c["hidden"]), 1.0, 0.0, _dtype(c)).to(F64)
        return [[_rms(h, w["model.norm.weight"]) @ w["lm_head.weight"].T, None]]
    x = _x(c, seed, c["tokens"] if "tokens" in c else sum(_step(c)[0])).to(F64)
    if c["kind"] == "ffn":
        return [(_silu(x @ w["gate_proj.weight"].T) * (x @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T]
    if c["kind"] == "experts":
        return _exact_experts(c, w, x)
    if c["kind"] == "attention":
        return _exact_attention(c, w, x, seed)
    if c["kind"] == "latent":
        return _exact_latent(c, w, x, seed)
    return _exact_recurrent(c, w, x, seed)
