"""The work that is timed: steps of models with random weights through the engine's public entry points.

What a program that serves a model does is one of four kinds of pass, all through ``Engine.step``:

  prompt    new sequences bring their prompts (of unequal lengths) in one step; the logits of the last ``want`` tokens
            of each are asked for: 1 to go on generating, more to score a continuation.
  decode    sequences with a filled cache get one token each per step, the token already on the device, for ``steps``
            steps; then the cache is taken back to where it was (``Engine.cache.truncate``), so that every pass does the
            same.  The logits are kept and the most likely token is sampled, as a generation loop does; the tokens fed are
            given, so that one different choice does not lead to another text.
  request   both: new sequences, their prompts, then ``steps`` decode steps with given tokens, the sequences closed again.
            For the designs with a state per sequence, which cannot be taken back.
  sampled   a request in 32 bits whose tokens are sampled with temperature, top-k and top-p and fed back on the device.

Model sizes are those of bench.py: the LLaMA-MoE-3.5B shape ("moe"), the dense Llama ("llama") and the small Llama with
experts ("moe_small") that it sets beside other designs, and the sizes s and m of two of these ("salepel", "zufadra").
``layers``: how many of them there are.  Weights are random, N(0, 0.02), a function of (seed, tensor name, index).

``exact`` restates the models in 64 bits with plain torch, and the rule for the weights, which the package documents
(``weights/counter_random.py``).
"""
import math
import random

import numpy as np
import torch

import transformer_b200 as tb
from transformer_b200.sampling import Sampler

VOCAB = 32000
STD = 0.02
SAMPLE = {"temperature": 0.8, "top_k": 40, "top_p": 0.9}


# ---- the cases -----------------------------------------------------------------------------------------------------
def _case(name, kind, model, layers, batch, low, high, *, size="", dtype="bfloat16", steps=0, want=1):
    """Prompts of ``batch`` sequences, lengths uniform in [low, high]."""
    c = {"kind": kind, "model": model, "size": size, "layers": layers, "dtype": dtype, "batch": batch, "low": low,
         "high": high, "steps": steps, "want": want}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one user, a small model, a short context: what a step costs when there is next to nothing to do
        _case("llama_decode_1", "decode", "llama", 8, 1, 201, 201, size="s", steps=4),
        # one user of the full model: the first of the benchmark's three points
        _case("moe_decode_1", "decode", "moe", 32, 1, 1088, 1088, steps=4),
        # the benchmark's own setting: eight sequences of unequal lengths
        _case("moe_decode_8", "decode", "moe", 32, 8, 128, 2048, steps=8),
        # a busy server: every expert is in use, the cache is as large as the weights
        _case("moe_decode_64", "decode", "moe", 8, 64, 128, 2048, steps=8),
        # a short question to the full model
        _case("moe_prompt_short", "prompt", "moe", 32, 1, 131, 131),
        # the benchmark's prompt; the last 64 tokens are scored
        _case("moe_prompt_2048", "prompt", "moe", 32, 1, 2048, 2048, want=64),
        # several users' prompts at once, more tokens than one piece of a step holds
        _case("moe_prompts_ragged", "prompt", "moe", 8, 11, 128, 2048, want=8),
        # grouped-query attention over long contexts: the cache is larger than the weights
        _case("llama_decode_16", "decode", "llama", 8, 16, 512, 8000, size="m", steps=6),
        # the 32-bit path, with sampling
        _case("moe_small_sampled_float32", "sampled", "moe_small", 8, 3, 16, 200, size="s", dtype="float32", steps=12),
        # latent attention and matrix memory: the second half of a long text of odd length is scored
        _case("salepel_score", "prompt", "salepel", 4, 1, 2039, 2039, size="m", want=1000),
        # delta rule and windowed attention: two long prompts of unequal lengths
        _case("zufadra_prompts", "prompt", "zufadra", 8, 2, 900, 2100, size="m", want=8),
        # the same design serving eight short requests
        _case("zufadra_requests", "request", "zufadra", 8, 8, 20, 120, size="m", steps=8),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "prompt", "request", "sampled"])
    if kind == "decode":
        model, size, layers = rng.choice([("llama", "s", 8), ("llama", "m", 8), ("moe", "", rng.randint(4, 12))])
        low = _log_int(rng, 16, 1024)
        high = _log_int(rng, low, 2048 if model == "moe" else 6000)
        return _case(None, kind, model, layers, _log_int(rng, 1, 64), low, high, size=size, steps=rng.randint(2, 6))
    if kind == "sampled":
        low = _log_int(rng, 4, 100)
        return _case(None, kind, rng.choice(["llama", "moe_small"]), 8, rng.randint(1, 6), low, _log_int(rng, low, 200),
                     size="s", dtype="float32", steps=rng.randint(4, 12))
    if kind == "request":
        low = _log_int(rng, 4, 100)
        return _case(None, kind, "zufadra", 8, _log_int(rng, 1, 12), low,
                     _log_int(rng, low, 300), size=rng.choice("sm"), steps=rng.randint(2, 8))
    model, size, layers = rng.choice([("llama", rng.choice("sm"), 8), ("moe", "", rng.randint(4, 12)),
                                      ("salepel", rng.choice("sm"), 4), ("zufadra", rng.choice("sm"), 8)])
    batch = _log_int(rng, 1, 6)
    low = _log_int(rng, 16, 2000 if batch == 1 else 600)
    return _case(None, kind, model, layers, batch, low, _log_int(rng, low, 2048), size=size,
                 want=rng.randint(200, 600) if model == "salepel" else rng.randint(1, 8))


def _config(c):
    """config.json keys of the case's model, with the sizes that bench.py gives them."""
    L, big = c["layers"], c["size"] == "m"
    if c["model"] in ("moe", "llama", "moe_small"):
        d, nh, nkvh, di, E, k, ctx, theta = {
            "moe": (4096, 32, 32, 688, 16, 4, 4096, 10000.0),
            "llama": (2048, 16, 4, 5632, 0, 0, 8192, 10000.0) if big else (1024, 8, 2, 2816, 0, 0, 8192, 10000.0),
            "moe_small": (1024, 4, 1, 512, 8, 2, 8192, 10000.0),
        }[c["model"]]
        cfg = {"model_type": "llama", "num_hidden_layers": L, "hidden_size": d, "num_attention_heads": nh,
               "num_key_value_heads": nkvh, "head_dim": 128, "intermediate_size": di, "max_position_embeddings": ctx,
               "vocab_size": VOCAB, "rms_norm_eps": 1e-5, "rope_theta": theta, "tie_word_embeddings": False}
        return dict(cfg, num_local_experts=E, num_experts_per_tok=k) if E else cfg
    if c["model"] == "salepel":
        d, H, dim, rot, vdim, rank, q_rank, window, mh, mdim, mvdim, E, ident, top, ff = \
            (2048, 16, 128, 64, 128, 512, 768, 2048, 8, 128, 256, 16, 2, 4, 704) if big else \
            (1024, 8, 64, 32, 64, 256, 384, 1024, 4, 128, 256, 8, 1, 2, 512)
        att = {"heads": H, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank, "q_rank": q_rank,
               "mask": {"size": window}, "rot": {"base": 10000.0, "dims": rot}, "scale": (dim + rot) ** -0.5}
        mem = {"heads": mh, "dim": mdim, "vdim": mvdim, "gate_cap": 15.0}
        mlp = {"kind": "moe", "router": {"experts": E, "identity": ident, "top": top}, "expert": {"ff": ff, "limit": 7.0}}
        layers = []
        for i in range(L):     # of four: a latent of its own, the matrix memory, two that read the first one's latent
            own = att if i % 4 == 0 else dict(att, kv_from=i - i % 4)
            layers.append({"type": "mlstm", "mixer": mem, "mlp": mlp} if i % 4 == 1 else
                          {"type": "latent_attention", "mixer": own, "mlp": mlp})
        return {"architecture": "Salepel", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0},
                "max_context": 8192, "layers": layers}
    d, H, G, dim, window, rank, ff = (2048, 16, 4, 128, 2048, 128, 5632) if big else (1024, 8, 2, 128, 1024, 64, 2816)
    att = {"heads": H, "kv_heads": G, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 30.0,
           "mask": {"size": window, "keep_first": 4},
           "rot": {"base": 500000.0, "dims": dim // 2,
                   "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    mem = {"heads": H, "kv_heads": H, "dim": dim, "vdim": dim, "conv": 4, "decay_rank": rank, "gate_rank": rank}
    layers = [{"type": "channel_delta" if i % 2 == 0 else "attention", "mixer": mem if i % 2 == 0 else att,
               "mlp": {"kind": "dense", "ff": ff}} for i in range(L)]
    return {"architecture": "Zufadra", "vocab": VOCAB, "width": d, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
            "logit_scale": 0.5, "embedding": {"scale": 8.0, "bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
            "max_context": 8192, "layers": layers}


def _lengths(c):
    """The prompts' lengths: part of the case, the same for every seed."""
    rng = random.Random(f"{c['batch']} {c['low']} {c['high']}")
    return [rng.randint(c["low"], c["high"]) for _ in range(c["batch"])]


def _inputs(c, seed):
    """(prompts, fed [steps][batch], uniform numbers [steps][batch]): uniform-random token ids."""
    rng = np.random.RandomState(1000003 * (seed % 2000) + 17)
    prompts = [rng.randint(0, VOCAB, n).tolist() for n in _lengths(c)]
    fed = rng.randint(0, VOCAB, (c["steps"], c["batch"])).tolist()
    u = (rng.randint(0, 1 << 24, (max(1, c["steps"]), c["batch"])) / float(1 << 24)).tolist()
    return prompts, fed, u


# ---- a pass --------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """The engine with its weights, the prompts as token lists, the decode steps' tokens on the device and, to decode, the
    sequences in its cache.  One pass over other tokens of the same shape has been made: the engine has served before."""
    c, lens = case, _lengths(case)
    room = sum((n + c["steps"] + 2 + 63) // 64 * 64 for n in lens)
    engine = tb.random_model(_config(c), seed=seed, dtype=c["dtype"], std=STD, max_tokens=room, max_slots=c["batch"] + 1)
    state = {"case": c, "engine": engine, "sampler": Sampler(engine.device), "args": tb.SampleArgs(
        **SAMPLE) if c["kind"] == "sampled" else tb.SampleArgs(), "one_each": [[0]] * c["batch"]}
    for s in (seed + 1, seed):
        prompts, fed, u = _inputs(c, s)
        state.update(prompts=prompts, u=u, fed=torch.tensor(fed, dtype=torch.int32, device=engine.device),
                     want=[list(range(max(0, n - c["want"]), n)) for n in lens])
        if c["kind"] == "decode":
            state["slots"] = [engine.open() for _ in prompts]
            engine.step(state["slots"], prompts)
        if s != seed:
            run(state)
            for slot in state.get("slots", ()):
                engine.close(slot)
    return state


def _decode(state, slots, logits, ids, first):
    c, engine, sampler = state["case"], state["engine"], state["sampler"]
    for i in range(first, first + c["steps"]):
        lg = engine.step(slots, state["one_each"], device_tokens=state["fed"][i - first])
        logits[i].copy_(lg)
        ids[i].copy_(sampler.sample(lg, state["args"])[0])


def run(state):
    c, engine, sampler = state["case"], state["engine"], state["sampler"]
    B, dev = c["batch"], engine.device
    if c["kind"] == "decode":
        logits = torch.empty((c["steps"], B, VOCAB), dtype=torch.float32, device=dev)
        ids = torch.empty((c["steps"], B), dtype=torch.int32, device=dev)
        before = [engine.cache.length(s) for s in state["slots"]]
        _decode(state, state["slots"], logits, ids, 0)
        for s, n in zip(state["slots"], before):
            engine.cache.truncate(s, n)
        return {"logits": logits, "ids": ids}
    slots = [engine.open() for _ in range(B)]
    try:
        if c["kind"] == "prompt":
            return {"logits": engine.step(slots, state["prompts"], want=state["want"])}
        logits = torch.empty((c["steps"] + 1, B, VOCAB), dtype=torch.float32, device=dev)
        ids = torch.empty((c["steps"] + 1, B), dtype=torch.int32, device=dev)
        lg = engine.step(slots, state["prompts"])
        logits[0].copy_(lg)
        if c["kind"] == "request":
            ids[0].copy_(sampler.sample(lg, state["args"])[0])
            _decode(state, slots, logits, ids, 1)
            return {"logits": logits, "ids": ids}
        for i in range(c["steps"]):
            ids[i].copy_(sampler.sample(lg, state["args"], state["u"][i])[0])
            lg = engine.step(slots, state["one_each"], device_tokens=ids[i])
            logits[i + 1].copy_(lg)
        return {"logits": logits, "ids": ids[:c["steps"]]}
    finally:
        for s in slots:
            engine.close(s)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _layer_costs(cfg):
    """Per layer: parameters every token meets, parameters of one expert, experts, experts per token, multiply-adds per
    (query, key) pair, values cached per token, window, state values per sequence, multiply-adds of the state per token."""
    out = []
    if "hidden_size" in cfg:
        d, nh, nkvh, dh, di = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                                "intermediate_size"))
        E, k = cfg.get("num_local_experts", 0), cfg.get("num_experts_per_tok", 0)
        fixed = d * (nh + 2 * nkvh) * dh + nh * dh * d + (E * d if E else 3 * d * di)
        return [(fixed, 3 * d * di if E else 0, E, k, 2 * nh * dh, 2 * nkvh * dh, None, 0, 0)] * cfg["num_hidden_layers"]
    d = cfg["width"]
    for layer in cfg["layers"]:
        m, f = layer["mixer"], layer["mlp"]
        H, dim, dv = m["heads"], m["dim"], m["vdim"]
        pair = cached = state = ops = 0
        window = m["mask"]["size"] if "mask" in m else None
        if layer["type"] == "latent_attention":
            r, qr, rd = m["kv_rank"], m["q_rank"], m["rot_dim"]
            fixed = qr * d + H * (dim + rd) * qr + H * (dim + dv) * r + d * H * dv + (0 if "kv_from" in m else (r + rd) * d)
            # each key costs a head the smaller of its own sizes and the latent's
            pair, cached = H * (dim + rd + dv), r + rd
        elif layer["type"] == "mlstm":
            fixed = 2 * H * dim * d + 3 * H * dv * d + 2 * H * d
            state, ops = H * dim * (dv + 1), 2 * H * dim * dv
        elif layer["type"] == "attention":
            G = m["kv_heads"]
            fixed = d * (H * dim + G * (dim + dv) + 2 * H * dv)
            pair, cached = H * (dim + dv), G * (dim + dv)
        else:
            G, ra, rg = m["kv_heads"], m["decay_rank"], m["gate_rank"]
            fixed = d * (2 * G * dim + 2 * H * dv + ra + rg + H) + H * dim * ra + H * dv * rg
            state, ops = H * dim * dv, 3 * H * dim * dv
        if f["kind"] == "moe":
            R = f["router"]
            out.append((fixed + (R["experts"] + R["identity"]) * d, 3 * d * f["expert"]["ff"], R["experts"],
                        R["top"] * R["experts"] / (R["experts"] + R["identity"]), pair, cached, window, state, ops))
        else:
            out.append((fixed + 3 * d * f["ff"], 0, 0, 0, pair, cached, window, state, ops))
    return out


def _step_work(cfg, elem, lens, before, rows):
    """(bytes, flops) of one step: lens[b] new tokens behind before[b] cached ones, ``rows`` logits rows."""
    n, B = sum(lens), len(lens)
    d = cfg.get("hidden_size", cfg.get("width"))
    traffic = VOCAB * d * elem + n * d * elem + 4 * rows * VOCAB
    macs = rows * VOCAB * d
    for fixed, expert, E, k, pair, cached, window, state, ops in _layer_costs(cfg):
        used = E * (1 - (1 - k / E) ** n) if E else 0
        traffic += elem * (fixed + used * expert) + 4 * state * B * (2 if any(before) else 1)
        macs += n * (fixed + k * expert + ops)
        for new, old in zip(lens, before):
            w = window or old + new
            traffic += elem * cached * (min(old, w) + new)
            macs += pair * sum(min(p + 1, w) for p in range(old, old + new))
    return traffic, 2 * macs


def work(case):
    c, lens = case, _lengths(case)
    cfg, elem = _config(c), 2 if c["dtype"] == "bfloat16" else 4
    total = [0, 0]

    def add(new, before, rows):
        b, f = _step_work(cfg, elem, new, before, rows)
        total[0] += b
        total[1] += f
    if c["kind"] != "decode":
        add(lens, [0] * len(lens), sum(min(n, c["want"]) for n in lens))
    for i in range(c["steps"]):
        add([1] * len(lens), [n + i for n in lens], len(lens))
    return {"bytes": total[0], "flops": total[1]}


def tolerance(case):
    """About four times the distance from ``exact`` that was measured.  bfloat16 activations alone leave 0.7 to 2.1 % of the
    logits after 8 layers (llama, zufadra).  Where experts are chosen, a token whose last chosen and first left-out expert
    are as good as equal may go to the other one, and its row is then another: 2 to 5 % over all rows for "moe" (whose rows
    without such a token are off by 0.8 to 1.5 %), 7 to 16 % for "salepel" (0.5 to 1.1 %), whose blocks norm what the
    experts return.  In 32 bits 1 to 2.2e-6.  ``differ``: two tokens as good as equally likely."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "differ": 0.05}
    return {"rel": {"llama": 0.05, "zufadra": 0.08, "moe": 0.2, "salepel": 0.5}[case["model"]], "differ": 0.3}


# ---- the same in 64 bits, with plain torch ---------------------------------------------------------------------------
_G, _M64 = 0x9E3779B97F4A7C15, (1 << 64) - 1


def _signed(z):
    z &= _M64
    return z - (1 << 64) if z >> 63 else z


def _shift(z, n):
    return (z >> n) & ((1 << (64 - n)) - 1)     # a logical shift of int64


def _mix(z, m0, m1):
    z = (z ^ _shift(z, 30)) * m0
    z = (z ^ _shift(z, 27)) * m1
    return z ^ _shift(z, 31)


class _Weights:
    """Tensors of the random model by file name, float64 on the GPU."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = int(seed), torch.bfloat16 if dtype == "bfloat16" else torch.float32

    def __call__(self, name, *shape, norm=False):
        """``norm``: a tensor that is kept in 32 bits whatever the model's type."""
        h = 0xCBF29CE484222325
        for byte in name.encode():
            h = ((h ^ byte) * 0x100000001B3) & _M64
        z = (self.seed * _G + h) & _M64
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M64
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M64
        base, m0, m1 = _signed(z ^ (z >> 31)), _signed(0xBF58476D1CE4E5B9), _signed(0x94D049BB133111EB)
        scale = torch.tensor(float(np.float32(STD / math.sqrt(8.0 * ((1 << 32) - 1) / 12.0))), device="cuda")
        n = math.prod(shape)
        out = torch.empty(n, dtype=torch.float64, device="cuda")
        for lo in range(0, n, 1 << 25):
            i2 = torch.arange(lo, min(n, lo + (1 << 25)), dtype=torch.int64, device="cuda") * 2
            total = torch.zeros_like(i2)
            for j in (0, 1):
                h = _mix((i2 + j) * _signed(_G) + base, m0, m1)
                for f in range(4):
                    total += _shift(h, 16 * f) & 0xFFFF if f else h & 0xFFFF
            v = (total - 4 * 65535).float() * scale
            out[lo:lo + v.numel()] = v if norm else v.to(self.dtype)
        return out.view(*shape)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _turn(x, pos, freqs, half):
    """x [n, heads, >= 2 len(freqs)]: pairs (2i, 2i + 1), or (i, i + len(freqs)) if ``half``, turn by pos * freqs[i]."""
    f = torch.tensor(freqs, dtype=torch.float64, device="cuda")
    ang = pos.double()[:, None, None] * f
    r = f.numel()
    a, b = (slice(0, r), slice(r, 2 * r)) if half else (slice(0, 2 * r, 2), slice(1, 2 * r, 2))
    y = x.clone()
    y[..., a] = x[..., a] * ang.cos() - x[..., b] * ang.sin()
    y[..., b] = x[..., b] * ang.cos() + x[..., a] * ang.sin()
    return y


def _attend(q, k, v, scale, window=None, keep=0, cap=None):
    """q [n, H, dk], k [n, G, dk], v [n, G, dv] -> [n, H, dv], causal."""
    n, H = q.shape[:2]
    rep = H // k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device="cuda")
    i, j = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None, :]
    see = j <= i
    if window is not None:
        see &= (i - j < window) | (j < keep)
    step = max(1, min(H, (1 << 28) // (n * n)))
    for h0 in range(0, H, step):
        heads = torch.arange(h0, min(H, h0 + step), device="cuda")
        s = torch.matmul(q[:, heads].transpose(0, 1), k[:, heads // rep].permute(1, 2, 0)) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s.masked_fill_(~see, float("-inf"))
        out[:, heads] = torch.matmul(torch.softmax(s, dim=-1), v[:, heads // rep].transpose(0, 1)).transpose(0, 1)
    return out


def _experts(x, choice, weight, E, gate_up_down, glu):
    """sum_j weight[:, j] * expert_{choice[:, j]}(x); a choice from E on hands x through."""
    out = torch.zeros_like(x)
    for e in range(E):
        tok, j = torch.nonzero(choice == e, as_tuple=True)
        if tok.numel():
            g, u, dn = gate_up_down(e)
            out.index_add_(0, tok, weight[tok, j][:, None] * (glu(x[tok] @ g.T, x[tok] @ u.T) @ dn.T))
    return out + (weight * (choice >= E)).sum(dim=1, keepdim=True) * x


def _exact_llama(cfg, W, seqs):
    d, nh, nkvh, dh, di = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim",
                                            "intermediate_size"))
    E, k, eps = cfg.get("num_local_experts", 0), cfg.get("num_experts_per_tok", 0), cfg["rms_norm_eps"]
    freqs = [cfg["rope_theta"] ** (-2.0 * i / dh) for i in range(dh // 2)]
    x = torch.cat([W("token_embd.weight", VOCAB, d)[s] for s in seqs])
    lens = [s.numel() for s in seqs]
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    silu = torch.nn.functional.silu
    for i in range(cfg["num_hidden_layers"]):
        p = f"blk.{i}."
        z = _rms(x, eps) @ W(p + "attn_qkv.weight", (nh + 2 * nkvh) * dh, d).T
        q, kk, v = (t.reshape(len(x), -1, dh) for t in z.split([nh * dh, nkvh * dh, nkvh * dh], dim=1))
        q, kk = _turn(q, pos, freqs, False), _turn(kk, pos, freqs, False)
        o = torch.cat([_attend(*t, dh ** -0.5) for t in zip(q.split(lens), kk.split(lens), v.split(lens))])
        del z, q, kk, v
        x = x + o.reshape(len(x), -1) @ W(p + "attn_output.weight", d, nh * dh).T
        h = _rms(x, eps)
        if E:
            lg = h @ W(p + "ffn_gate_inp.weight", E, d).T
            top = torch.topk(lg, k, dim=-1)
            gu, dn = W(p + "ffn_gate_up_exps.weight", E, 2 * di, d), W(p + "ffn_down_exps.weight", E, d, di)
            x = x + _experts(h, top.indices, torch.softmax(top.values, dim=-1), E,
                             lambda e: (gu[e, :di], gu[e, di:], dn[e]), lambda g, u: silu(g) * u)
            del gu, dn
        else:
            gu = h @ W(p + "ffn_gate_up.weight", 2 * di, d).T
            x = x + (silu(gu[:, :di]) * gu[:, di:]) @ W(p + "ffn_down.weight", d, di).T
    return _rms(x, eps), W("output.weight", VOCAB, d), 1.0


def _exact_salepel(cfg, W, seqs):
    d, eps = cfg["width"], cfg["norm"]["eps"]
    x = torch.cat([W("embed", VOCAB, d)[s] for s in seqs]) * cfg["embedding"]["scale"]
    lens = [s.numel() for s in seqs]
    n, pos = len(x), torch.cat([torch.arange(m, device="cuda") for m in lens])
    latents = {}
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        h = _rms(x, eps)
        if layer["type"] == "latent_attention":
            r, rd, qr = m["kv_rank"], m["rot_dim"], m["q_rank"]
            freqs = [m["rot"]["base"] ** (-2.0 * j / rd) for j in range(rd // 2)]
            src = m.get("kv_from", i)
            if src == i:
                kv = h @ W(p + "dkv", r + rd, d).T
                latents[i] = _rms(kv[:, :r], eps), _turn(kv[:, None, r:], pos, freqs, True)
            c, kr = latents[src]
            q = (_rms(h @ W(p + "dq", qr, d).T, eps) @ W(p + "uq", H * (dk + rd), qr).T).view(n, H, dk + rd)
            q = torch.cat([q[..., :dk], _turn(q[..., dk:], pos, freqs, True)], dim=-1)
            kk = torch.cat([(c @ W(p + "uk", H * dk, r).T).view(n, H, dk), kr.expand(n, H, rd)], dim=-1)
            v = (c @ W(p + "uv", H * dv, r).T).view(n, H, dv)
            o = torch.cat([_attend(*t, m["scale"], m["mask"]["size"])
                           for t in zip(q.split(lens), kk.split(lens), v.split(lens))])
            y = o.reshape(n, -1)
        else:
            q, kk = ((h @ W(p + t, H * dk, d).T).view(n, H, dk) for t in "qk")
            v, cap = (h @ W(p + "v", H * dv, d).T).view(n, H, dv), m["gate_cap"]
            ig, fg = (cap * torch.tanh((h @ W(p + t, H, d).T + W(p + t + ".b", H, norm=True)) / cap) for t in "if")
            fg = torch.nn.functional.logsigmoid(fg)
            outs = []
            for qs, ks, vs, ii, ff in zip(*(t.split(lens) for t in (q * dk ** -0.5, kk, v, ig, fg))):
                F = ff.cumsum(0).T                                                    # [H, n]
                D = F[:, :, None] - F[:, None, :] + ii.T[:, None, :]
                D.masked_fill_(~torch.ones(D.shape[1:], dtype=torch.bool, device="cuda").tril(), float("-inf"))
                top = torch.maximum(D.amax(dim=-1), F)
                C = torch.exp(D - top[:, :, None]) * torch.matmul(qs.transpose(0, 1), ks.permute(1, 2, 0))
                den = torch.maximum(C.sum(-1).abs(), torch.exp(-top)) + 1e-6
                outs.append((torch.matmul(C, vs.transpose(0, 1)) / den[:, :, None]).transpose(0, 1))
            y = _rms(torch.cat(outs), eps).reshape(n, H * dv) * torch.sigmoid(h @ W(p + "g", H * dv, d).T)
        x = x + _rms(y @ W(p + "o", d, H * dv).T, eps)
        f, p = layer["mlp"], f"l{i}.mlp."
        E, R, ff = f["router"]["experts"], f["router"]["experts"] + f["router"]["identity"], f["expert"]["ff"]
        h = _rms(x, eps)
        s = torch.softmax(h @ W(p + "router", R, d).T, dim=-1)
        choice = torch.topk(s + W(p + "correction", R, norm=True), f["router"]["top"], dim=-1).indices
        limit = f["expert"]["limit"]

        def glu(g, u):
            g = g.clamp(max=limit)
            return g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1.0)
        y = _experts(h, choice, torch.gather(s, 1, choice), E,
                     lambda e: (W(p + f"e{e}.gate", ff, d), W(p + f"e{e}.up", ff, d), W(p + f"e{e}.down", d, ff)), glu)
        x = x + _rms(y, eps)
    return _rms(x, eps), W("head", VOCAB, d), 1.0


def _scaled_freqs(rot):
    out, sc = [], rot["scaling"]
    for i in range(rot["dims"] // 2):
        f = rot["base"] ** (-2.0 * i / rot["dims"])
        wave = 2.0 * math.pi / f
        if wave > sc["original"] / sc["low"]:
            f /= sc["factor"]
        elif wave >= sc["original"] / sc["high"]:
            s = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
            f = (1.0 - s) * f / sc["factor"] + s * f
        out.append(f)
    return out


def _exact_zufadra(cfg, W, seqs):
    d, eps, mult, emb = cfg["width"], cfg["norm"]["eps"], cfg["residual_mult"], cfg["embedding"]
    big, table, pairs = emb["bigram"], W("embed", VOCAB, d), W("bigram", emb["bigram"]["buckets"] + 1, d)
    xs = []
    for s in seqs:
        at = torch.full_like(s, big["buckets"])
        at[1:] = (s[:-1] * big["mul_prev"] + s[1:] * big["mul_cur"]) % big["buckets"]
        xs.append(table[s] * emb["scale"] + pairs[at])
    x, lens = torch.cat(xs), [s.numel() for s in seqs]
    n, pos = len(x), torch.cat([torch.arange(m, device="cuda") for m in lens])
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}.mix."
        H, G, dim, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        if layer["type"] == "attention":
            freqs = _scaled_freqs(m["rot"])
            q = _turn(_rms(x @ W(p + "q", H * dim, d).T, eps).view(n, H, dim), pos, freqs, False)
            k = _turn(_rms(x @ W(p + "k", G * dim, d).T, eps).view(n, G, dim), pos, freqs, False)
            v = (x @ W(p + "v", G * dv, d).T).view(n, G, dv)
            o = torch.cat([_attend(*t, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], m["softcap"])
                           for t in zip(q.split(lens), k.split(lens), v.split(lens))])
            y = o.reshape(n, H * dv) * torch.sigmoid(x @ W(p + "g", H * dv, d).T)
        else:
            T, most, B = m["conv"], max(lens), len(lens)

            def padded(t):
                return torch.nn.utils.rnn.pad_sequence(list(t.split(lens)), batch_first=True)     # [B, most, ...]

            def conv(name, rows):
                z, taps = padded(x @ W(p + name, rows, d).T), W(p + name + ".conv", rows, T, norm=True)
                z = torch.nn.functional.pad(z, (0, 0, T - 1, 0))
                return torch.nn.functional.silu(sum(z[:, j:j + most] * taps[:, j] for j in range(T)))

            def unit(t):
                return t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
            q = unit(conv("q", G * dim).view(B, most, G, dim)) * dim ** -0.5
            k = unit(conv("k", G * dim).view(B, most, G, dim))
            q, k = (t.repeat_interleave(H // G, dim=2) for t in (q, k))
            v = conv("v", H * dv).view(B, most, H, dv)
            beta = padded(torch.sigmoid(x @ W(p + "b", H, d).T))
            a = (x @ W(p + "a1", m["decay_rank"], d).T) @ W(p + "a2", H * dim, m["decay_rank"]).T
            a = a + W(p + "dt_bias", H * dim, norm=True)
            rate = torch.exp(W(p + "A_log", H, norm=True))
            g = padded(torch.exp(-rate[:, None] * torch.nn.functional.softplus(a.view(n, H, dim))))
            S = torch.zeros(B, H, dim, dv, dtype=torch.float64, device="cuda")
            o = torch.empty(B, most, H, dv, dtype=torch.float64, device="cuda")
            for t in range(most):
                S *= g[:, t, :, :, None]
                u = beta[:, t, :, None] * (v[:, t] - torch.matmul(k[:, t, :, None], S)[:, :, 0])
                S += k[:, t, :, :, None] * u[:, :, None]
                o[:, t] = torch.matmul(q[:, t, :, None], S)[:, :, 0]
            o = torch.cat([o[b, :m_] for b, m_ in enumerate(lens)])
            gate = torch.sigmoid((x @ W(p + "g1", m["gate_rank"], d).T) @ W(p + "g2", H * dv, m["gate_rank"]).T)
            y = _rms(o, eps).reshape(n, H * dv) * gate
        x = x + mult * _rms(y @ W(p + "o", d, H * dv).T, eps)
        p, ff = f"l{i}.mlp.", layer["mlp"]["ff"]
        g, u = (x @ W(p + t, ff, d).T + W(p + t + ".b", ff, norm=True) for t in ("gate", "up"))
        y = (torch.nn.functional.silu(g) * u) @ W(p + "down", d, ff).T + W(p + "down.b", d, norm=True)
        x = x + mult * _rms(y, eps)
    return _rms(x, eps), W("head", VOCAB, d), cfg["logit_scale"]


def _exact_logits(c, seed, seqs, rows):
    """Logits of the given rows of each sequence, [sum of rows, VOCAB]."""
    fn = {"salepel": _exact_salepel, "zufadra": _exact_zufadra}.get(c["model"], _exact_llama)
    x, head, scale = fn(_config(c), _Weights(seed, c["dtype"]), [torch.tensor(s, device="cuda") for s in seqs])
    at = 0
    picked = []
    for s, r in zip(seqs, rows):
        picked.append(x[torch.tensor(r, device="cuda") + at])
        at += len(s)
    return torch.cat(picked) @ head.T * scale


def _draw_token(logits, u):
    """One token from a row of logits under SAMPLE: the top_k largest, softmax, the shortest prefix of mass top_p,
    then the first kept id, in ascending order, whose running mass exceeds u times the kept mass."""
    z = logits / SAMPLE["temperature"]
    order = torch.sort(z, descending=True, stable=True).indices[:SAMPLE["top_k"]]
    p = torch.softmax(z[order], dim=0)
    n = int((p.cumsum(0) < SAMPLE["top_p"]).sum()) + 1
    kept, at = order[:n].sort()
    mass = p[:n][at].cumsum(0)
    return int(kept[min(int((mass <= u * mass[-1]).sum()), n - 1)])


def exact(case, seed):
    c = case
    prompts, fed, u = _inputs(c, seed)
    if c["kind"] == "prompt":
        rows = [list(range(max(0, len(p) - c["want"]), len(p))) for p in prompts]
        return {"logits": _exact_logits(c, seed, prompts, rows)}
    seqs, ids = [list(p) for p in prompts], []
    if c["kind"] == "sampled":
        for i in range(c["steps"]):
            lg = _exact_logits(c, seed, seqs, [[len(s) - 1] for s in seqs])
            ids.append([_draw_token(lg[b], u[i][b]) for b in range(len(seqs))])
            for s, t in zip(seqs, ids[-1]):
                s.append(t)
    else:
        for step in fed:
            for s, t in zip(seqs, step):
                s.append(t)
    first = 0 if c["kind"] == "decode" else 1
    rows = [list(range(len(p) - (1 if first else 0), len(s))) for p, s in zip(prompts, seqs)]
    lg = _exact_logits(c, seed, seqs, rows).view(len(seqs), -1, VOCAB).transpose(0, 1)
    # the most likely tokens of the other kinds have no value of their own: two logits may be as good as equal
    return {"logits": lg, "ids": torch.tensor(ids, dtype=torch.int32) if c["kind"] == "sampled" else None}
