"""The work that a program has this library do, as cases that can be timed and compared.

Every case builds an ``Engine`` of a few layers at the layer sizes of the benchmark (the cost of a whole model is that of its
layers, times their number, and one head) and makes one pass through ``Engine.step``: a batch of prompts, or a decode step of
sequences that hold a prompt already.  Four designs stand for the library's paths:

  dense   Qwen3: grouped-query attention with normed and rotated heads, gated feed-forward; in bfloat16 and in true 32 bits
  latent  Bozavik: latent attention (rotated, and without positions behind a sink), routed experts beside a shared one
  delta   Sugizen: the gated delta rule, then attention by blocks with a gate a head; clamped gated feed-forward
  space   Tinuzen: windowed attention with a bias by distance, then attention with a sink beside a state-space mixer

``exact`` restates each design in 64 bits with plain torch.
"""
import math

import torch

import ultima_b200 as u

DEVICE = "cuda:0"
VOCAB = 32768
EPS = 1e-5
STEPS_FROM_START = 4             # decode of designs with state: that many steps of sequences that begin


# ---------------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------------
def _case(name, family, mode, batch, length, width, layers, dtype="bfloat16", ragged=False, dim=128):
    c = dict(family=family, mode=mode, batch=batch, length=length, ragged=ragged, width=width, dim=dim, layers=layers, dtype=dtype)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user's chat: a token a step, the weights stream through the chip for a single row
        _case("dense_decode_1", "dense", "decode", 1, 2048, 4096, 4),
        # the benchmark's decode: eight sequences, here at unequal lengths
        _case("dense_decode_8", "dense", "decode", 8, 2011, 4096, 4, ragged=True),
        # a full server: 64 sequences, cache and weights weigh alike
        _case("dense_decode_64", "dense", "decode", 64, 2048, 4096, 4, ragged=True),
        # a short question: few tokens, launches and latency count
        _case("dense_prompt_short", "dense", "prompt", 1, 45, 4096, 4),
        # requests that arrive together with unequal prompts
        _case("dense_prompts_ragged", "dense", "prompt", 6, 611, 4096, 4, ragged=True),
        # a document as a prompt, the benchmark's length
        _case("dense_prompt_2048", "dense", "prompt", 1, 2048, 4096, 4),
        # the true 32-bit path, with which bfloat16 results are judged: a prompt, and steps behind it
        _case("dense_f32_prompt", "dense", "prompt", 2, 389, 2048, 2, dtype="float32", ragged=True),
        _case("dense_f32_decode", "dense", "decode", 4, 389, 2048, 2, dtype="float32", ragged=True),
        # latent attention and routed experts: a prompt that reaches every expert, a step that reaches some
        _case("latent_prompt_2048", "latent", "prompt", 1, 2048, 2048, 2),
        _case("latent_decode_8", "latent", "decode", 8, 1500, 2048, 2, ragged=True),
        # recurrent designs reading a document
        _case("delta_prompt_2048", "delta", "prompt", 1, 2048, 2048, 2),
        _case("space_prompt_2048", "space", "prompt", 1, 2048, 2048, 2),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    family = rng.choice(["dense"] * 6 + ["f32"] * 2 + ["latent"] * 2 + ["delta", "space"])
    mode = rng.choice(["prompt", "decode"])
    if family == "f32":
        batch = spread(1, 8)
        return _case(None, "dense", mode, batch, spread(9, 780 // batch if mode == "prompt" else 600), rng.choice([1024, 2048]), 2,
                     dtype="float32", ragged=rng.random() < 0.5, dim=rng.choice([64, 128]))
    if family == "dense":
        width, dim, layers = rng.choice([2048, 4096]), rng.choice([64, 128, 128]), rng.randint(2, 4)
        if mode == "decode":
            return _case(None, "dense", mode, spread(1, 64), spread(60, 2048), width, layers, ragged=rng.random() < 0.5, dim=dim)
        batch = spread(1, 8)
        return _case(None, "dense", mode, batch, spread(12, 2048 // batch), width, layers, ragged=rng.random() < 0.5, dim=dim)
    if mode == "decode":
        return _case(None, family, mode, spread(1, 32), spread(40, 1800), 2048, 2, ragged=rng.random() < 0.5)
    batch = spread(1, 4)
    return _case(None, family, mode, batch, spread(30, 2048 // batch), 2048, 2, ragged=rng.random() < 0.5)


def _lengths(case):
    """Positions of each sequence: all alike, or from the longest down to about half of it."""
    n, b = case["length"], case["batch"]
    return [n - (n * i) // (2 * b) if case["ragged"] else n for i in range(b)]


def _from_start(case):
    return case["mode"] == "decode" and case["family"] in ("delta", "space")


def _sizes(case):
    w, d = case["width"], case["dim"]
    heads = w // d
    return dict(width=w, dim=d, heads=heads, kv_heads=max(1, heads // 4), ff=3 * w, layers=case["layers"])


# ---------------------------------------------------------------------------------------------------------------------
# configurations and weights
# ---------------------------------------------------------------------------------------------------------------------
def _config(case):
    z = _sizes(case)
    w, d, H, G, ff = z["width"], z["dim"], z["heads"], z["kv_heads"], z["ff"]
    family = case["family"]
    if family == "dense":
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=VOCAB, hidden_size=w, intermediate_size=ff,
                    num_hidden_layers=z["layers"], num_attention_heads=H, num_key_value_heads=G, head_dim=d, rms_norm_eps=EPS,
                    rope_theta=1000000.0, max_position_embeddings=8192, tie_word_embeddings=False, hidden_act="silu")
    base = {"vocab": VOCAB, "width": w, "norm": {"eps": EPS}}
    if family == "latent":
        rotated = {"heads": H, "dim": d, "rot_dim": 64, "vdim": d, "q_rank": w * 3 // 8, "kv_rank": 192, "scale": (d + 64) ** -0.5,
                   "rot": {"base": 500000.0, "dims": 64}}
        plain = {"heads": H, "dim": d, "vdim": d, "q_rank": w * 3 // 8, "kv_rank": 256, "scale": d ** -0.5}
        mlp = {"kind": "moe", "expert": {"ff": ff // 6, "limit": 7.0}, "shared": {"ff": ff // 3, "limit": 7.0},
               "router": {"experts": 32, "top": 4}}
        layers = [{"type": "latent_attention", "mixer": dict(plain), "mlp": dict(mlp)} if i % 2 else
                  {"type": "latent_attention_2", "mixer": dict(rotated), "mlp": dict(mlp)} for i in range(z["layers"])]
        return dict(base, architecture="Bozavik", embedding={"scale": 12.0}, residual_mult=0.3, layers=layers)
    if family == "delta":
        delta = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "conv": 4, "decay_rank": 64, "gate_rank": 64}
        att = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "rot": {"base": 500000.0, "dims": d // 2},
               "mask": {"size": 1024}}
        mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
        return dict(base, architecture="Sugizen", layers=[
            {"type": "attention", "mixer": dict(att), "mlp": dict(mlp)} if i % 2 else
            {"type": "channel_delta", "mixer": dict(delta), "mlp": dict(mlp)} for i in range(z["layers"])])
    att = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": 1024, "keep_first": 4}}
    left = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "rot": {"base": 10000.0, "dims": d}}
    right = {"heads": w // 64, "vdim": 64, "state": 128, "groups": 2, "conv": 4, "norm_groups": 2}
    mlp = {"kind": "dense", "ff": ff}
    return dict(base, architecture="Tinuzen", embedding={"scale": 16.0, "bigram": {"buckets": 16381, "mul_prev": 31, "mul_cur": 7}},
                loop={"start": 0, "stop": z["layers"], "times": 1}, layers=[
                    {"type": "parallel", "mixer": {"left": dict(left), "right": dict(right), "left_scale": 1.2, "right_scale": 0.9},
                     "mlp": dict(mlp)} if i % 2 else
                    {"type": "attention", "mixer": dict(att), "mlp": dict(mlp)} for i in range(z["layers"])])


def _weights(case, seed):
    """Stored name -> tensor on the GPU: matrices in the run's type, vectors in 32 bits."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(1000003 * int(seed) + 17)
    run = getattr(torch, case["dtype"])
    W = {}

    def mat(name, rows, cols, std=None):
        W[name] = torch.randn(rows, cols, generator=gen, device=DEVICE, dtype=torch.float32).mul_(std or cols ** -0.5).to(run)

    def vec(name, *shape, mean=0.0, std=0.05):
        W[name] = torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float32).mul_(std).add_(mean)

    z, cfg, family = _sizes(case), _config(case), case["family"]
    w, d, H, G, ff = z["width"], z["dim"], z["heads"], z["kv_heads"], z["ff"]
    if family == "dense":
        mat("model.embed_tokens.weight", VOCAB, w, 0.5)
        for i in range(z["layers"]):
            p = f"model.layers.{i}."
            vec(p + "input_layernorm.weight", w, mean=1.0)
            mat(p + "self_attn.q_proj.weight", H * d, w)
            mat(p + "self_attn.k_proj.weight", G * d, w)
            mat(p + "self_attn.v_proj.weight", G * d, w)
            mat(p + "self_attn.o_proj.weight", w, H * d)
            vec(p + "self_attn.q_norm.weight", d, mean=1.0)
            vec(p + "self_attn.k_norm.weight", d, mean=1.0)
            vec(p + "post_attention_layernorm.weight", w, mean=1.0)
            mat(p + "mlp.gate_proj.weight", ff, w)
            mat(p + "mlp.up_proj.weight", ff, w)
            mat(p + "mlp.down_proj.weight", w, ff)
        vec("model.norm.weight", w, mean=1.0)
        mat("lm_head.weight", VOCAB, w)
        return W

    def dense(p, inner):
        mat(p + "gate", inner, w)
        mat(p + "up", inner, w)
        mat(p + "down", w, inner)

    mat("embed", VOCAB, w, 0.05 if family != "delta" else 0.5)
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.", L["mixer"]
        if family == "latent":
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                vec(p + n, w, mean=1.0)
                vec(p + n + ".b", w)
            rot, rank = m.get("rot_dim", 0), m["kv_rank"]
            mat(p + "mix.dq", m["q_rank"], w)
            vec(p + "mix.dq.norm", m["q_rank"], mean=1.0)
            mat(p + "mix.uq", H * (d + rot), m["q_rank"])
            mat(p + "mix.dkv", rank + rot, w)
            vec(p + "mix.dkv.norm", rank, mean=1.0)
            mat(p + "mix.uk", H * d, rank)
            mat(p + "mix.uv", H * d, rank)
            mat(p + "mix.o", w, H * d)
            mat(p + "mix.g", H if rot else H * d, w)
            if not rot:
                vec(p + "mix.sink", H, std=1.0)
            mat(p + "mlp.router", 32, w, 0.3)
            for e in range(32):
                dense(f"{p}mlp.e{e}.", ff // 6)
            dense(p + "mlp.shared.", ff // 3)
            mat(p + "mlp.shared.sg", 1, w)
        elif L["type"] == "channel_delta":
            for n, rows in (("q", G * d), ("k", G * d), ("v", H * d)):
                mat(p + "mix." + n, rows, w)
                vec(p + "mix." + n + ".conv", rows, 4, std=0.3)
            mat(p + "mix.b", H, w)
            vec(p + "mix.A_log", H, std=0.5)
            vec(p + "mix.norm", d, mean=1.0)
            mat(p + "mix.a1", 64, w)
            mat(p + "mix.a2", H * d, 64)
            vec(p + "mix.dt_bias", H * d, mean=-2.0, std=1.0)       # decays of a few to a few dozen tokens
            mat(p + "mix.g1", 64, w)
            mat(p + "mix.g2", H * d, 64)
            mat(p + "mix.o", w, H * d)
        elif family == "delta":
            mat(p + "mix.q", H * d, w)
            mat(p + "mix.k", G * d, w)
            mat(p + "mix.v", G * d, w)
            mat(p + "mix.o", w, H * d)
            mat(p + "mix.g", H, w)
            vec(p + "mix.q.norm", d, mean=1.0)
            vec(p + "mix.k.norm", d, mean=1.0)
        elif L["type"] == "attention":
            mat(p + "mix.q", H * d, w)
            mat(p + "mix.k", G * d, w)
            mat(p + "mix.v", G * d, w)
            mat(p + "mix.o", w, H * d)
            vec(p + "mix.q.norm", H * d, mean=1.0)
            vec(p + "mix.k.norm", G * d, mean=1.0)
        else:
            r = m["right"]
            inner, conv = r["heads"] * r["vdim"], r["heads"] * r["vdim"] + 2 * r["groups"] * r["state"]
            mat(p + "mix.left.q", H * d, w)
            mat(p + "mix.left.k", G * d, w)
            mat(p + "mix.left.o", w, H * d)
            mat(p + "mix.left.g", H * d, w)
            mat(p + "mix.right.in", inner + conv + r["heads"], w)
            vec(p + "mix.right.conv", conv, 4, std=0.3)
            vec(p + "mix.right.conv.b", conv, std=0.1)
            vec(p + "mix.right.dt_bias", r["heads"], mean=-2.0, std=1.0)
            vec(p + "mix.right.A_log", r["heads"], std=0.5)
            vec(p + "mix.right.D", r["heads"], mean=1.0)
            vec(p + "mix.right.norm", inner, mean=1.0)
            mat(p + "mix.right.o", w, inner)
        if family != "latent":
            vec(p + "norm1", w, mean=1.0)
            dense(p + "mlp.", ff)
        if family == "delta":
            vec(p + "norm2", w, mean=1.0)
        if family == "space":
            for g in ("rg1", "rg2"):
                mat(p + g, w, w)
                vec(p + g + ".b", w, std=0.5)
    if family == "space":
        mat("bigram", 16382, w, 0.5)
        vec("loop.step", 1, w, std=0.1)
    vec("final.norm", w, mean=1.0)
    if family == "latent":
        vec("final.norm.b", w)
    mat("head", VOCAB, w)
    return W


def _tokens(case, seed):
    """Token ids: every sequence's prompt and, for decode, the tokens of the steps behind it."""
    gen = torch.Generator()
    gen.manual_seed(7919 * int(seed) + 3)
    extra = 0 if case["mode"] == "prompt" else 1
    if _from_start(case):
        return [torch.randint(0, VOCAB, (STEPS_FROM_START,), generator=gen).tolist() for _ in range(case["batch"])]
    return [torch.randint(0, VOCAB, (n + extra,), generator=gen).tolist() for n in _lengths(case)]


def _wanted(n):
    """The places of a prompt whose logits are asked for: every 16th token and the last."""
    return sorted(set(range(15, n, 16)) | {n - 1})


# ---------------------------------------------------------------------------------------------------------------------
# a program's side
# ---------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    spec = u.model_spec_for(u.config_from_dict(_config(case)))
    reach = max(_lengths(case)) + 64
    pages = sum(-(-(n + 1) // 64) for n in _lengths(case))
    eng = u.Engine(spec, _weights(case, seed), dtype=case["dtype"], max_tokens=64 * (pages + 1), max_seqs=case["batch"],
                   max_context=reach, with_sampler=False, window_pass=2048)
    ids = _tokens(case, seed)
    state = dict(engine=eng, case=dict(case), ids=ids)
    if case["mode"] == "prompt":
        state["want"] = [_wanted(len(t)) for t in ids]
    elif not _from_start(case):
        state["slots"] = eng.open(case["batch"])
        eng.step(state["slots"], [t[:-1] for t in ids], [[] for _ in ids])
        state["last"] = [[t[-1]] for t in ids]
        state["lengths"] = _lengths(case)
    return state


def run(state):
    eng, case = state["engine"], state["case"]
    if case["mode"] == "prompt":
        slots = eng.open(case["batch"])
        logits = eng.step(slots, state["ids"], state["want"])
        eng.close(slots)
        return logits
    if _from_start(case):
        slots = eng.open(case["batch"])
        out = [eng.step(slots, [[t[i]] for t in state["ids"]]) for i in range(STEPS_FROM_START)]
        eng.close(slots)
        return out
    # a step behind the prompts, which stay for the next pass
    logits = eng.step(state["slots"], state["last"])
    for s, n in zip(state["slots"], state["lengths"]):
        eng.truncate(s, n)
    return logits


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    z, cfg, family = _sizes(case), _config(case), case["family"]
    w, d, H, G, ff = z["width"], z["dim"], z["heads"], z["kv_heads"], z["ff"]
    el = 4 if case["dtype"] == "float32" else 2
    lengths, B = _lengths(case), case["batch"]
    steps = STEPS_FROM_START if _from_start(case) else 1
    if case["mode"] == "prompt":
        T, rows = sum(lengths), sum(len(_wanted(n)) for n in lengths)
        seen = [(n, n * (n + 1) // 2) for n in lengths]             # (cached positions, query-key pairs)
    elif _from_start(case):
        T, rows, seen = B, B, [(STEPS_FROM_START // 2, STEPS_FROM_START // 2)] * B
    else:
        T, rows, seen = B, B, [(n + 1, n + 1) for n in lengths]
    params = flops = kv = 0.0
    for L in cfg.get("layers") or [None] * z["layers"]:
        active, other = 3 * w * ff, 0.0                              # feed-forward weights a token passes; recurrence
        mix = w * (H + 2 * G) * d + H * d * w
        row, pair = 2 * G * d, 4 * H * d
        read = active
        if family == "latent":
            rot = L["mixer"].get("rot_dim", 0)
            rank, q = L["mixer"]["kv_rank"], L["mixer"]["q_rank"]
            mix = w * q + q * H * (d + rot) + w * (rank + rot) + 2 * H * d * rank + H * d * w + w * (H if rot else H * d)
            row, pair = rank + rot, 2 * H * (2 * rank + rot)
            one = 3 * w * (ff // 6)
            active = 4 * one + 3 * w * (ff // 3) + 32 * w
            read = one * 32 * (1 - (1 - 4 / 32) ** T) + 3 * w * (ff // 3) + 32 * w
        elif L and L["type"] == "channel_delta":
            mix = w * (2 * G + H) * d + w * H + 128 * (w + H * d) + H * d * w
            row, pair, other = 0, 0, 8 * H * d * d
        elif family == "space":
            mix += 2 * w * w
            if L["type"] == "parallel":
                r = L["mixer"]["right"]
                inner = r["heads"] * r["vdim"]
                mix += w * (H - G) * d + w * (2 * inner + 2 * r["groups"] * r["state"] + r["heads"]) + inner * w
                row, other = G * d, 6 * inner * r["state"]
        params += mix + read
        flops += T * (2 * (mix + active) + other) + pair * sum(p for _, p in seen)
        kv += row * sum(n for n, _ in seen)
        if other and case["mode"] == "decode":
            kv += T * other / 4 * 2                                   # a step reads and writes the 32-bit state (two elements' worth each)
    params += VOCAB * w
    flops += 2.0 * rows * VOCAB * w
    return {"bytes": steps * (el * (params + kv + T * w) + 4.0 * rows * VOCAB), "flops": steps * flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 0.03, "max": 0.5} if case["family"] == "latent" else {"rel": 0.02, "max": 0.2}


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _layer_norm(x, w, b):
    c = x - x.mean(-1, keepdim=True)
    return c * torch.rsqrt((c * c).mean(-1, keepdim=True) + EPS) * w + b


def _turn(x, base, dims, neighbours=False):
    """x [T, heads, n]: pairs of the first ``dims`` columns turned by the position's angles."""
    T, half = x.shape[0], dims // 2
    f = torch.arange(half, dtype=x.dtype, device=x.device).mul(-2.0 / dims)
    a = torch.arange(T, dtype=x.dtype, device=x.device)[:, None] * torch.pow(torch.tensor(float(base), dtype=x.dtype, device=x.device), f)
    c, s = a.cos()[:, None], a.sin()[:, None]
    out = x.clone()
    one, two = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, half), slice(half, dims))
    p, q = x[..., one], x[..., two]
    out[..., one], out[..., two] = p * c - q * s, q * c + p * s
    return out


def _attend(q, k, v, scale, window=None, keep=0, block=None, slopes=None, sink=None):
    """q [T, H, .], k [T, G, .], v [T, G, .] -> [T, H, .], head by head of the keys."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device=q.device)[:, None]
    j = torch.arange(T, device=q.device)[None, :]
    seen = j <= i
    if window is not None:
        seen = seen & ((i - j < window) | (j < keep))
    if block is not None:
        seen = seen & (i // block == j // block)
    out = []
    for h in range(H):
        g = h // (H // G)
        s = q[:, h] @ k[:, g].T * scale
        if slopes is not None:
            s = s - slopes[h] * (i - j)
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        p = torch.softmax(s, -1)
        out.append(p[:, :T] @ v[:, g])
    return torch.stack(out, 1)


def _conv(x, taps):
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _clamped(h, g, up, down, limit=7.0):
    a, b = (h @ g.T).clamp(max=limit), (h @ up.T).clamp(-limit, limit)
    return (a * torch.sigmoid(1.702 * a) * (b + 1)) @ down.T


def _dense_layer(x, M, i, z):
    p, H, G, d = f"model.layers.{i}.", z["heads"], z["kv_heads"], z["dim"]
    h = _rms(x, M(p + "input_layernorm.weight"))
    a = p + "self_attn."
    q = _rms((h @ M(a + "q_proj.weight").T).view(-1, H, d), M(a + "q_norm.weight"))
    k = _rms((h @ M(a + "k_proj.weight").T).view(-1, G, d), M(a + "k_norm.weight"))
    v = (h @ M(a + "v_proj.weight").T).view(-1, G, d)
    o = _attend(_turn(q, 1e6, d), _turn(k, 1e6, d), v, d ** -0.5)
    x = x + o.reshape(-1, H * d) @ M(a + "o_proj.weight").T
    h = _rms(x, M(p + "post_attention_layernorm.weight"))
    m = p + "mlp."
    return x + (_silu(h @ M(m + "gate_proj.weight").T) * (h @ M(m + "up_proj.weight").T)) @ M(m + "down_proj.weight").T


def _latent_layer(x, M, i, L, z):
    p, m, H, d = f"l{i}.", L["mixer"], z["heads"], z["dim"]
    rank, rot = m["kv_rank"], m.get("rot_dim", 0)
    h = _layer_norm(x, M(p + "norm1"), M(p + "norm1.b"))
    q = (_rms(h @ M(p + "mix.dq").T, M(p + "mix.dq.norm")) @ M(p + "mix.uq").T).view(-1, H, d + rot)
    low = h @ M(p + "mix.dkv").T
    c = _rms(low[:, :rank], M(p + "mix.dkv.norm"))
    k, v = (c @ M(p + "mix.uk").T).view(-1, H, d), (c @ M(p + "mix.uv").T).view(-1, H, d)
    if rot:
        turned = _turn(low[:, None, rank:], m["rot"]["base"], rot)
        q = torch.cat([q[..., :d], _turn(q[..., d:], m["rot"]["base"], rot)], -1)
        k = torch.cat([k, turned.expand(-1, H, -1)], -1)
    o = _attend(q, k, v, m["scale"], sink=None if rot else M(p + "mix.sink"))
    g = torch.sigmoid(h @ M(p + "mix.g").T)
    o = o * g[:, :, None] if rot else o * g.view(-1, H, d)
    x = x + 0.3 * _layer_norm(o.reshape(-1, H * d) @ M(p + "mix.o").T, M(p + "norm1b"), M(p + "norm1b.b"))
    h = _layer_norm(x, M(p + "norm2"), M(p + "norm2.b"))
    e = p + "mlp."
    best = torch.topk(h @ M(e + "router").T, 4, dim=-1)
    wts = torch.softmax(best.values, -1)
    y = torch.sigmoid(h @ M(e + "shared.sg").T) * _clamped(h, M(e + "shared.gate"), M(e + "shared.up"), M(e + "shared.down"))
    for n in range(32):
        t, k = torch.nonzero(best.indices == n, as_tuple=True)
        if t.numel():
            one = _clamped(h[t], M(f"{e}e{n}.gate"), M(f"{e}e{n}.up"), M(f"{e}e{n}.down"))
            y.index_add_(0, t, wts[t, k][:, None] * one)
    return x + 0.3 * _layer_norm(y, M(p + "norm2b"), M(p + "norm2b.b"))


def _delta_layer(x, M, i, L, z):
    p, m, H, G, d = f"l{i}.", L["mixer"], z["heads"], z["kv_heads"], z["dim"]
    T = x.shape[0]
    if L["type"] == "channel_delta":
        q, k, v = (_silu(_conv(x @ M(p + "mix." + n).T, M(p + "mix." + n + ".conv"))).view(T, -1, d) for n in "qkv")
        q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
        beta = torch.sigmoid(x @ M(p + "mix.b").T)
        step = _softplus((x @ M(p + "mix.a1").T) @ M(p + "mix.a2").T + M(p + "mix.dt_bias")).view(T, H, d)
        decay = torch.exp(-torch.exp(M(p + "mix.A_log"))[None, :, None] * step)
        S, o = x.new_zeros(H, d, d), torch.empty_like(v)
        for t in range(T):
            S = decay[t][:, :, None] * S
            r = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = S + k[t][:, :, None] * r[:, None, :]
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = _rms(o, M(p + "mix.norm")) * torch.sigmoid((x @ M(p + "mix.g1").T) @ M(p + "mix.g2").T).view(T, H, d)
    else:
        rot = m["rot"]
        q = _turn(_rms((x @ M(p + "mix.q").T).view(T, H, d), M(p + "mix.q.norm")), rot["base"], rot["dims"])
        k = _turn(_rms((x @ M(p + "mix.k").T).view(T, G, d), M(p + "mix.k.norm")), rot["base"], rot["dims"])
        o = _attend(q, k, (x @ M(p + "mix.v").T).view(T, G, d), m["scale"], block=m["mask"]["size"])
        o = o * torch.sigmoid(x @ M(p + "mix.g").T)[:, :, None]
    x = x + _rms(o.reshape(T, H * d) @ M(p + "mix.o").T, M(p + "norm1"))
    return x + _rms(_clamped(x, M(p + "mlp.gate"), M(p + "mlp.up"), M(p + "mlp.down")), M(p + "norm2"))


def _space_layer(x, M, i, L, z):
    p, m, H, G, d = f"l{i}.", L["mixer"], z["heads"], z["kv_heads"], z["dim"]
    T = x.shape[0]
    h = _rms(x, M(p + "norm1"))
    if L["type"] == "attention":
        q = _rms(h @ M(p + "mix.q").T, M(p + "mix.q.norm")).view(T, H, d)
        k = _rms(h @ M(p + "mix.k").T, M(p + "mix.k.norm")).view(T, G, d)
        slopes = 2.0 ** (-8.0 * (torch.arange(H, dtype=x.dtype, device=x.device) + 1) / H)
        o = _attend(q, k, (h @ M(p + "mix.v").T).view(T, G, d), m["scale"], m["mask"]["size"], m["mask"]["keep_first"], slopes=slopes)
        y = o.reshape(T, H * d) @ M(p + "mix.o").T
    else:
        a, b = p + "mix.left.", p + "mix.right."
        q, k = (h @ M(a + "q").T).view(T, H, d), (h @ M(a + "k").T).view(T, G, d)
        rot = m["left"]["rot"]
        o = _attend(_turn(q, rot["base"], rot["dims"], True), _turn(k, rot["base"], rot["dims"], True), k, m["left"]["scale"],
                    sink=x.new_zeros(H))
        y = 1.2 * ((o.reshape(T, H * d) * torch.sigmoid(h @ M(a + "g").T)) @ M(a + "o").T)
        r = m["right"]
        HR, P, N, GR = r["heads"], r["vdim"], r["state"], r["groups"]
        inner = HR * P
        s = h @ M(b + "in").T
        gate, mid, dt = s[:, :inner], s[:, inner:2 * inner + 2 * GR * N], s[:, 2 * inner + 2 * GR * N:]
        mid = _silu(_conv(mid, M(b + "conv")) + M(b + "conv.b"))
        v = mid[:, :inner].reshape(T, HR, P)
        key = mid[:, inner:inner + GR * N].reshape(T, GR, N).repeat_interleave(HR // GR, 1)
        out = mid[:, inner + GR * N:].reshape(T, GR, N).repeat_interleave(HR // GR, 1)
        dt = _softplus(dt + M(b + "dt_bias"))
        keepf = torch.exp(-torch.exp(M(b + "A_log")) * dt)
        S, o = x.new_zeros(HR, N, P), torch.empty_like(v)
        for t in range(T):
            S = keepf[t][:, None, None] * S + (dt[t][:, None] * key[t])[:, :, None] * v[t][:, None, :]
            o[t] = torch.bmm(out[t][:, None], S)[:, 0]
        o = (o + M(b + "D")[:, None] * v).reshape(T, inner) * _silu(gate)
        o = o.view(T, r["norm_groups"], -1)
        o = (o * torch.rsqrt((o * o).mean(-1, keepdim=True) + EPS)).reshape(T, inner) * M(b + "norm")
        y = y + 0.9 * (o @ M(b + "o").T)
    f = (torch.relu(h @ M(p + "mlp.gate").T) * (h @ M(p + "mlp.up").T)) @ M(p + "mlp.down").T
    return x + torch.sigmoid(h @ M(p + "rg1").T + M(p + "rg1.b")) * y + torch.sigmoid(h @ M(p + "rg2").T + M(p + "rg2.b")) * f


def exact(case, seed):
    W, z, cfg, family = _weights(case, seed), _sizes(case), _config(case), case["family"]

    def M(name):
        return W[name].double()

    with torch.no_grad():
        streams = []
        for ids in _tokens(case, seed):
            t = torch.tensor(ids, device=DEVICE)
            x = W["model.embed_tokens.weight" if family == "dense" else "embed"][t].double()
            if family == "latent":
                x = x * 12.0
            if family == "space":
                b = cfg["embedding"]["bigram"]
                rows = torch.full_like(t, b["buckets"])
                rows[1:] = (t[:-1] * b["mul_prev"] + t[1:] * b["mul_cur"]) % b["buckets"]
                x = x * cfg["embedding"]["scale"] + W["bigram"][rows].double() + M("loop.step")[0]
            streams.append(x)
        for i in range(z["layers"]):
            held = {}

            def H(name):                     # a layer's weights are widened once for all sequences
                if name not in held:
                    held[name] = M(name)
                return held[name]
            for s, x in enumerate(streams):
                if family == "dense":
                    streams[s] = _dense_layer(x, H, i, z)
                else:
                    step = {"latent": _latent_layer, "delta": _delta_layer, "space": _space_layer}[family]
                    streams[s] = step(x, H, i, cfg["layers"][i], z)
        head = M("lm_head.weight" if family == "dense" else "head")

        def logits(x):
            if family == "latent":
                h = _layer_norm(x, M("final.norm"), M("final.norm.b"))
            else:
                h = _rms(x, M("model.norm.weight" if family == "dense" else "final.norm"))
            return h @ head.T
        if case["mode"] == "prompt":
            return logits(torch.cat([x[torch.tensor(_wanted(x.shape[0]), device=DEVICE)] for x in streams]))
        if _from_start(case):
            return [logits(torch.stack([x[i] for x in streams])) for i in range(STEPS_FROM_START)]
        return logits(torch.stack([x[-1] for x in streams]))
