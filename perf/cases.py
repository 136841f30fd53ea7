"""What is timed of this package: rows steps of its engines, called as a serving program calls them - ``step`` with token ids, lanes and positions from
the host, the next tokens read back - for the DeepSeek-V4.1-Flash architecture ("flash") and the four layered decoders, in both directions of the path:
prompts in portions (prefill) and one row per sequence (decode).

A case names the model, its width, its layers, and the step: ``rows`` rows against ``ctx`` cached positions.  Prefill: the rows of ``prompts`` sequences
together; decode: one row for each of ``rows`` sequences, whose contexts differ.  Per-layer shapes are those of the package's benchmark; the number of
layers is cut (as its reduced configurations do) so that a state fits the card several times over, and so that random weights, which amplify rounding from
layer to layer, leave logits that two correct implementations agree on.
"""
from __future__ import annotations

import dataclasses
import math

import torch
import torch.nn.functional as F

from sparkflash_b200.config import reduced_config
from sparkflash_b200.models.deepseek_v41 import engine as flash_engine
from sparkflash_b200.models.deepseek_v41 import prepare as flash_weights
from sparkflash_b200.models.layered import LayeredEngine
from sparkflash_b200.utils import layered_bench

FLASH_EXPERTS = 64            # resident experts of a flash layer (six per row)
PORTION = 4096                # rows per step of the context's prefill, and the largest portion of a prompt
# layers of a case: one of every kind that the design has, eight where rounding allows it
LAYERS = {"flash": 6, "fanodra": 8, "gudutar": 4, "lifulorn": 4, "dironex": 4}
WIDTHS = ("w1024", "w2048", "w4096")


def _case(model, width, step, rows, ctx, prompts=1):
    return {"model": model, "width": width, "layers": LAYERS[model], "step": step, "rows": rows, "ctx": ctx, "prompts": prompts}


def listed():
    named = lambda name, *a, **k: {"name": name, **_case(*a, **k)}
    return [
        named("flash-decode-1", "flash", "", "decode", 1, 2048),                                # one user's next token after a 2,048-token prompt
        named("flash-decode-16", "flash", "", "decode", 16, 1500),                              # sixteen users, contexts of mixed lengths
        named("flash-decode-1-long", "flash", "", "decode", 1, 30000),                          # one user deep in a long document
        named("flash-prefill-4096", "flash", "", "prefill", 4096, 0),                           # the portion that long prompts are cut into
        named("flash-prefill-777", "flash", "", "prefill", 777, 333),                           # a chat's next turn: a ragged portion behind a short context
        named("fanodra-w1024-decode-1", "fanodra", "w1024", "decode", 1, 500),                  # the smallest step: launches and latency
        named("fanodra-w2048-prefill-4096", "fanodra", "w2048", "prefill", 4096, 0),            # first portion of a long prompt
        named("gudutar-w2048-decode-64", "gudutar", "w2048", "decode", 64, 1100),               # a full server: 64 sequences
        named("gudutar-w4096-prefill-1999", "gudutar", "w4096", "prefill", 1999, 0, prompts=3),  # three prompts of odd lengths in one step
        named("lifulorn-w2048-decode-16", "lifulorn", "w2048", "decode", 16, 4000),             # sixteen sequences, nearly every expert in use
        named("lifulorn-w4096-prefill-4096", "lifulorn", "w4096", "prefill", 4096, 0, prompts=4),  # four prompts together
        named("dironex-w2048-prefill-3000", "dironex", "w2048", "prefill", 3000, 5000),         # a later portion: attention over what is cached
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["flash", "flash", "fanodra", "gudutar", "lifulorn", "dironex"])
    width = "" if model == "flash" else rng.choice(WIDTHS)
    if rng.random() < 0.5:
        rows = spread(1, 16 if model == "flash" else 64)
        return _case(model, width, "decode", rows, spread(100, 8000 if rows <= 16 else 2000))
    rows = spread(100, 4000)
    return _case(model, width, "prefill", rows, 0 if rng.random() < 0.5 else spread(60, 4000), 1 if model == "flash" else rng.randint(1, 4))


# ---- the program that calls the engine -----------------------------------------------------------------------------------
def _config(case):
    if case["model"] == "flash":
        return reduced_config(FLASH_EXPERTS, case["layers"])
    cfg = layered_bench.CONFIGS[case["model"]][0](case["width"])
    unlooped = {"loop": None} if hasattr(cfg, "loop") else {"loop_start": 0, "loop_stop": 0, "loop_times": 0} if hasattr(cfg, "loop_times") else {}
    return dataclasses.replace(cfg, layers=cfg.layers[:case["layers"]], **unlooped)


def _lengths(case):
    """(cached positions, rows of the step) of every sequence."""
    rows, ctx = case["rows"], case["ctx"]
    if case["step"] == "decode":
        return [(ctx - 37 * i % max(1, ctx // 4), 1) for i in range(rows)]
    n, left, out = case["prompts"], rows, []
    for i in range(n):                                # portions of unequal length
        m = left if i == n - 1 else rows // n + (13 * (i + 1)) % 29 - 14
        out.append((ctx, m))
        left -= m
    return out


def _tokens(case, seed):
    """Every sequence's tokens: what is cached, then the step's rows."""
    g = torch.Generator().manual_seed(seed)
    vocab = _config(case).vocab_size
    return [torch.randint(0, vocab, (c + m,), generator=g).tolist() for c, m in _lengths(case)]


def prepare(case, seed):
    """An engine with its weights, whose caches hold every sequence's context, and the step's rows; one such step has run, as in a server that has
    warmed up."""
    cfg, lengths, seqs = _config(case), _lengths(case), _tokens(case, seed)
    rows = max(max(c for c, _ in lengths), case["rows"])
    size = dict(max_lanes=len(lengths), max_context=max(c + m for c, m in lengths) + 64, max_rows=max(128, min(PORTION, rows)))
    if case["model"] == "flash":
        weights = flash_weights.prepare_synthetic(cfg, seed=seed)
        eng = flash_engine.Engine(weights, arm="tc", synthetic_scales=True, **size)
    else:
        _, cls, tensors = layered_bench.CONFIGS[case["model"]]
        eng = LayeredEngine(cls(cfg, tensors(cfg, seed, "cuda"), max_context=size["max_context"]), **size)
    for lane, (c, _) in enumerate(lengths):
        for a in range(0, c, size["max_rows"]):
            b = min(a + size["max_rows"], c)
            eng.step(seqs[lane][a:b], [lane] * (b - a), list(range(a, b)), head=False, sync=False)
    step = {"engine": eng, "flash": case["model"] == "flash", "tokens": [], "lanes": [], "positions": [], "head": True}
    ends = []
    for lane, (c, m) in enumerate(lengths):
        step["tokens"] += seqs[lane][c:]
        step["lanes"] += [lane] * m
        step["positions"] += range(c, c + m)
        ends.append(len(step["tokens"]) - 1)
    if case["step"] == "prefill":
        step["head"] = "last" if len(ends) == 1 else ends
    run(step)
    eng.check_status()
    return step


def run(state):
    """The step, its tokens read back.  Returns the logits of the sampled rows, the caches and the recurrent states (flash: codes of the windows, of the
    compressed entries and of the index keys).  The tokens themselves are left out: random weights have near ties.  The same step again writes the
    same places of the caches."""
    eng, n = state["engine"], len(state["tokens"])
    eng.step(state["tokens"], state["lanes"], state["positions"], head=state["head"])
    if state["flash"]:
        codes = {k: list(getattr(eng.kv, k).values()) for k in ("win_q", "ckv_q", "ik_q")}
        return {"logits": eng.logits[n - 1:n] if state["head"] == "last" else eng.logits[:n], **codes}
    return {"logits": eng.logits, "k": eng.kv.k, "v": eng.kv.v, "states": list(eng.state.tensors.values())}


# ---- what a step cannot do without ---------------------------------------------------------------------------------------
def _seen(lengths, window=None):
    """(keys read, query-key pairs) of attention over the last ``window`` positions."""
    keys, pairs = 0, 0
    for c, m in lengths:
        w = window or c + m
        keys += min(c, w - 1) + m
        pairs += sum(min(c + i + 1, w) for i in range(m))
    return keys, pairs


def work(case):
    """Weights that the rows use, cached keys and states they see, and logits, once each; the products of all of them."""
    return _flash_work(case) if case["model"] == "flash" else _layered_work(case)


def _used(experts, top, rows):
    return experts * (1 - (1 - top / experts) ** rows)


def _flash_work(case):
    c, lengths, n = _config(case), _lengths(case), case["rows"]
    d, H, hd, q, mi = c.hidden_size, c.n_heads, c.head_dim, c.q_lora_rank, c.moe_inter
    heads = 1 if case["step"] == "prefill" else n
    dense = d * (q + hd) + H * hd * q + H * hd * c.o_lora_rank + d * c.o_groups * c.o_lora_rank + 3 * d * mi
    nbytes, flops = 2.0 * c.vocab_size * d + 4.0 * heads * c.vocab_size, 2.0 * heads * c.vocab_size * d
    wkeys, wpairs = _seen(lengths, c.window)
    for l in range(c.n_layers):
        mix = 2 * (2 + c.hc_mult) * c.hc_mult * c.hc_mult * d
        nbytes += dense * 33 / 32 + 4.0 * mix + 2.0 * c.n_routed_experts * d + 3 * d * mi * (17 / 32) * _used(c.n_routed_experts, c.top_k, n)
        flops += 2.0 * n * (dense + mix + c.n_routed_experts * d + 3 * d * mi * c.top_k)
        nbytes += wkeys * hd * 33 / 32
        pairs = wpairs
        if c.ratio(l):
            r = c.ratio(l)
            pairs += sum(min(c.index_topk, (a + i + 1) // r) for a, m in lengths for i in range(m))
            nbytes += sum(min(c.index_topk * m, (a + m) // r) for a, m in lengths) * hd * 9 / 16
        if c.is_index_source(l):
            entries, scored = _seen(lengths)
            nbytes += c.index_n_heads * c.index_head_dim * q * 33 / 32 + entries / c.ratio(l) * c.index_head_dim * 17 / 32
            flops += 2.0 * n * c.index_n_heads * c.index_head_dim * q + 2.0 * scored / c.ratio(l) * c.index_n_heads * c.index_head_dim
        flops += 4.0 * pairs * H * hd
    return {"bytes": nbytes, "flops": flops}


def _layered_work(case):
    cfg, lengths, n = _config(case), _lengths(case), case["rows"]
    heads = n if case["step"] == "decode" else case["prompts"]
    head_rows = cfg.vocab * cfg.width
    nbytes, flops = 4.0 * heads * cfg.vocab + 2.0 * head_rows, 2.0 * heads * head_rows
    for name, shape in cfg.shapes().items():
        size = math.prod(shape)
        if name in ("embed", "head") or name.startswith("side.embed"):
            continue
        L = cfg.layers[int(name[1:name.index(".")])] if name[0] == "l" and name[1].isdigit() else None
        r = (getattr(L, "mlp", None) or {}).get("router") if L is not None else None
        part = name.split(".")[2] if r and ".mlp.e" in name else ""
        if part[1:].isdigit():                        # a routed expert
            nbytes += 2.0 * size * _used(r["experts"], r["top"], n) / r["experts"]
            flops += 2.0 * n * size * r["top"] / r["experts"]
        else:
            nbytes += 2.0 * size
            flops += 2.0 * n * size if len(shape) > 1 and shape[-1] > 8 else 0.0
    for L in cfg.layers:
        m = L.mixer["left"] if L.type == "parallel" else L.mixer
        if "kv_heads" in m and L.type != "delta":
            keys, pairs = _seen(lengths, m["mask"]["size"] if "mask" in m else None)
            nbytes += 2.0 * keys * m["kv_heads"] * (m["dim"] + m["vdim"])
            flops += 2.0 * pairs * m["heads"] * (m["dim"] + m["vdim"])
        elif "kv_rank" in m:
            keys, pairs = _seen(lengths, m["mask"]["size"] if "mask" in m else None)
            nbytes += 2.0 * keys * (m["kv_rank"] + m["rot_dim"])
            flops += 2.0 * pairs * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        else:
            N = m.get("state", m.get("dim"))
            if N:
                nbytes += 8.0 * len(lengths) * m["heads"] * N * m["vdim"]
                flops += 4.0 * n * m["heads"] * N * m["vdim"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Measured on random weights.  Flash: activations in FP8 and a choice of experts that lies close make portions of other lengths, which sum in another
    order, differ by 0.04 and more at six layers, so the bounds are the largest that can be stated.  The others in bf16: portions of other lengths
    differ by up to 0.006 (Fanodra, Lifulorn, Dironex) and 0.012 (Gudutar), and single rows whose choice of experts lies close by more."""
    if case["model"] == "flash":
        return {"rel": 0.03, "max": 0.9, "differ": 0.01}
    return {"rel": 0.03 if case["model"] != "fanodra" else 0.025, "max": 0.9}


# ---- the layered decoders in 64 bits, from their equations ---------------------------------------------------------------
def exact(case, seed):
    """Logits of the sampled rows.  None for flash (a product of activations rounded to FP8 and of a choice between experts that lie close is another
    function after any other rounding: 0.2 to 0.6 between the package's own exact and tensor-core arms), and where the sequences are too long."""
    lengths = _lengths(case)
    if case["model"] == "flash" or sum(c + m for c, m in lengths) * int(case["width"][1:]) > 3e8:
        return None
    cfg = _config(case)
    w = {k: v.double() for k, v in layered_bench.CONFIGS[case["model"]][2](cfg, seed, "cuda").items()}
    forward = {"fanodra": _fanodra, "gudutar": _gudutar, "lifulorn": _lifulorn, "dironex": _dironex}[case["model"]]
    seqs = _tokens(case, seed)
    T = max(len(s) for s in seqs)
    out = []
    group = max(1, 40000 // T)                        # sequences at a time, filled up at the end (causal: what is behind does not matter)
    for a in range(0, len(seqs), group):
        some = seqs[a:a + group]
        ids = torch.tensor([s + [0] * (T - len(s)) for s in some], device="cuda")
        ends = torch.tensor([len(s) - 1 for s in some], device="cuda")
        h, table = forward(w, cfg, ids)
        out.append(h[torch.arange(len(some), device="cuda"), ends] @ table.t())
    return {"logits": torch.cat(out)}


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _ln(x, w, name, eps):
    return F.layer_norm(x, x.shape[-1:], w[name], w[name + ".b"], eps)


def _conv(x, w):
    """Causal depthwise convolution of x [B, T, C] with w [C, taps]; the last tap is the row itself."""
    taps, T = w.shape[1], x.shape[1]
    x = F.pad(x, (0, 0, taps - 1, 0))
    return sum(w[:, j] * x[:, j:j + T] for j in range(taps))


def _gelu(x):
    return F.gelu(x, approximate="tanh")


def _attend(q, k, v, scale, window=None, bias=None, cap=0.0, sink=None):
    """q [B, T, H, d], k and v [B, T, G, .]: softmax over the visible keys, a block of rows of one head group at a time."""
    B, T, H, _ = q.shape
    rep = H // k.shape[2]
    out = q.new_zeros(B, T, H, v.shape[-1])
    j = torch.arange(T, device=q.device)
    for b in range(B):
        for r0 in range(0, T, 1024):
            i = j[r0:r0 + 1024]
            lo, hi = max(0, r0 - window + 1) if window else 0, min(T, r0 + 1024)
            back = i[:, None] - j[None, lo:hi]
            hidden = (back < 0) | (back >= window) if window else back < 0
            for h in range(H):
                s = q[b, r0:r0 + 1024, h] @ k[b, lo:hi, h // rep].t() * scale
                if cap:
                    s = cap * torch.tanh(s / cap)
                if bias is not None:
                    s = s - bias(h, back.clamp(min=0).double())
                s = s.masked_fill(hidden, float("-inf"))
                if sink is not None:
                    s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
                p = torch.softmax(s, -1)[:, :hi - lo]
                out[b, r0:r0 + 1024, h] = p @ v[b, lo:hi, h // rep]
    return out.flatten(2)


def _frequencies(rot):
    base, dims, sc = rot["base"], rot["dims"], rot.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if sc is None:
        return f, 1.0
    if "fast" in sc:                                  # YaRN: divided along a ramp, cosine and sine scaled
        where = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(where(sc["fast"])), 0), min(math.ceil(where(sc["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(len(f))]
        return [x / sc["factor"] * r + x * (1 - r) for x, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1
    out = []
    for x in f:                                       # by how many wavelengths the original context holds
        s = min(max((sc["original"] * x / (2 * math.pi) - sc["low"]) / (sc["high"] - sc["low"]), 0.0), 1.0)
        out.append((1 - s) * x / sc["factor"] + s * x)
    return out, 1.0


def _turn(x, rot, pairs=False):
    """x [B, T, H, dim]: element i of the first ``dims`` turns with i + dims / 2, or with its neighbour (``pairs``)."""
    f, gain = _frequencies(rot)
    a = torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None] * torch.tensor(f, dtype=torch.float64, device=x.device)
    c, s = (gain * a.cos())[:, None], (gain * a.sin())[:, None]
    dims = rot["dims"]
    if pairs:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        turned = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        turned = torch.cat([u * c - v * s, v * c + u * s], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _fanodra(w, cfg, ids):
    eps = cfg.eps

    def recurrence(p, h):
        y = _gelu(h @ w[p + "y"].t() + w[p + "y.b"])
        u = _conv(h @ w[p + "x"].t() + w[p + "x.b"], w[p + "conv"]) + w[p + "conv.b"]
        parts = w[p + "ra"].shape[0]
        gate = lambda n: torch.sigmoid(torch.einsum("btkj,kij->btki", u.unflatten(-1, (parts, -1)), w[p + n]).flatten(2) + w[p + n + ".b"].flatten())
        la = -8 * gate("ra") * F.softplus(w[p + "lam"], threshold=50.0)
        x, a, S, out = torch.sqrt(-torch.expm1(2 * la)) * gate("ri") * u, la.exp(), 0.0, torch.empty_like(u)
        for t in range(u.shape[1]):
            S = a[:, t] * S + x[:, t]
            out[:, t] = S
        return (out * y) @ w[p + "o"].t()

    def attention(p, m, h):
        H, G, dim = m["heads"], m["kv_heads"], m["dim"]
        q = (_rms(h @ w[p + "q"].t() + w[p + "q.b"], eps) * w[p + "q.norm"]).unflatten(-1, (H, dim))
        k = (_rms(h @ w[p + "k"].t() + w[p + "k.b"], eps) * w[p + "k.norm"]).unflatten(-1, (G, dim))
        v = (h @ w[p + "v"].t() + w[p + "v.b"]).unflatten(-1, (G, m["vdim"]))
        far = lambda a, back: w[p + "r1"][a] * torch.log1p(w[p + "r2"][a] * back)
        return _attend(q, k, v, m["scale"], bias=far) @ w[p + "o"].t() + w[p + "o.b"]
    x = w["embed"][ids]
    for i, L in enumerate(cfg.layers):
        p = f"l{i}."
        h = _ln(x, w, p + "norm1", eps)
        h = h + _conv(h, w[p + "canon1"])
        if L.type == "parallel":
            left = _rms(attention(p + "mix.left.", L.mixer["left"], h), eps) * w[p + "mix.left.out"]
            y = 0.5 * (left + _rms(recurrence(p + "mix.right.", h), eps) * w[p + "mix.right.out"])
        else:
            y = recurrence(p + "mix.", h)
        x = x + _ln(y, w, p + "norm1b", eps)
        h = _ln(x, w, p + "norm2", eps)
        x = x + _ln((F.silu(h @ w[p + "mlp.gate"].t()) * (h @ w[p + "mlp.up"].t())) @ w[p + "mlp.down"].t(), w, p + "norm2b", eps)
    return _ln(x, w, "final.norm", eps), w["embed"]


def _decayed(q, k, v, a):
    """S = a S + k v^T, out = S^T q; q, k [B, T, H, N], v [B, T, H, P], a [B, T, H]."""
    S, out = q.new_zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3]), torch.empty_like(v)
    for t in range(q.shape[1]):
        S = S * a[:, t, :, None, None] + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = torch.einsum("bhnp,bhn->bhp", S, q[:, t])
    return out


def _gudutar(w, cfg, ids):
    eps = cfg.eps

    def mamba2(p, m, h):
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        z, xbc, dt = torch.split(h @ w[p + "in"].t(), [H * P, H * P + 2 * G * N, H], dim=-1)
        x, B, C = torch.split(F.silu(_conv(xbc, w[p + "conv"]) + w[p + "conv.b"]), [H * P, G * N, G * N], dim=-1)
        dt = F.softplus(dt + w[p + "dt_bias"], threshold=50.0)
        x = x.unflatten(-1, (H, P))
        wide = lambda t: t.unflatten(-1, (G, N)).repeat_interleave(H // G, 2)
        y = _decayed(wide(C), wide(B) * dt[..., None], x, torch.exp(-torch.exp(w[p + "A_log"]) * dt)) + w[p + "D"][:, None] * x
        y = (y.flatten(2) * F.silu(z)).unflatten(-1, (m["norm_groups"], -1))
        return (_rms(y, eps).flatten(2) * w[p + "norm"]) @ w[p + "o"].t()

    def retention(p, m, h):
        H, N, P = m["heads"], m["dim"], m["vdim"]
        q = _turn((h @ w[p + "q"].t()).unflatten(-1, (H, N)), m["rot"])
        k = _turn((h @ w[p + "k"].t()).unflatten(-1, (H, N)), m["rot"]) * N ** -0.5
        v = (h @ w[p + "v"].t()).unflatten(-1, (H, P))
        a = torch.tensor(m["decay"], dtype=torch.float64, device=h.device).expand(*h.shape[:2], H)
        return (_rms(_decayed(q, k, v, a), eps).flatten(2) * F.silu(h @ w[p + "g"].t())) @ w[p + "o"].t()

    def latent(p, m, h):
        H, dim, rd, r = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        q = (h @ w[p + "q"].t()).unflatten(-1, (H, dim + rd))
        q = torch.cat([q[..., :dim], _turn(q[..., dim:], m["rot"], pairs=True)], -1)
        down = h @ w[p + "dkv"].t()
        c, shared = _rms(down[..., :r], eps) * w[p + "dkv.norm"], _turn(down[:, :, None, r:], m["rot"], pairs=True)
        k = torch.cat([(c @ w[p + "uk"].t()).unflatten(-1, (H, dim)), shared.expand(-1, -1, H, -1)], -1)
        v = (c @ w[p + "uv"].t()).unflatten(-1, (H, m["vdim"]))
        return _attend(q, k, v, m["scale"], m["mask"]["size"]) @ w[p + "o"].t()
    x = w["embed"][ids] * cfg.embed_scale
    for i, L in enumerate(cfg.layers):
        p = f"l{i}."
        x = x + _ln({"mamba2": mamba2, "retention": retention, "latent_attention": latent}[L.type](p + "mix.", L.mixer, x), w, p + "norm1", eps)
        x = x + _ln((_gelu(x @ w[p + "mlp.gate"].t()) * (x @ w[p + "mlp.up"].t())) @ w[p + "mlp.down"].t(), w, p + "norm2", eps)
    return _ln(x, w, "final.norm", eps), w["head"]


def _experts(h, ids, wts, expert):
    """Weighted sum of the chosen experts; ids and wts [rows, top]."""
    y = torch.zeros_like(h)
    for e in ids.unique().tolist():
        rows, k = (ids == e).nonzero(as_tuple=True)
        y.index_add_(0, rows, wts[rows, k, None] * expert(e, h[rows]))
    return y


def _lifulorn(w, cfg, ids):
    eps, mult, first = cfg.eps, cfg.residual_mult, []

    def delta(p, m, h):
        H, N, P = m["heads"], m["dim"], m["vdim"]
        short = lambda n: F.silu(_conv(h @ w[p + n].t(), w[p + n + ".conv"])).unflatten(-1, (H, -1))
        unit = lambda x: x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        q, k, v = unit(short("q")) * N ** -0.5, unit(short("k")), short("v")
        beta = torch.sigmoid(h @ w[p + "b"].t())
        a = torch.exp(-torch.exp(w[p + "A_log"]) * F.softplus(h @ w[p + "a"].t() + w[p + "dt_bias"], threshold=50.0))
        S, out = h.new_zeros(h.shape[0], H, N, P), torch.empty_like(v)
        for t in range(h.shape[1]):
            S = S * a[:, t, :, None, None]
            u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhnp,bhn->bhp", S, k[:, t]))
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            out[:, t] = torch.einsum("bhnp,bhn->bhp", S, q[:, t])
        out = _rms(out, eps) * w[p + "norm"] * F.silu(h @ w[p + "g"].t()).unflatten(-1, (H, P))
        return out.flatten(2) @ w[p + "o"].t()

    def attention(p, m, h):
        H, G = m["heads"], m["kv_heads"]
        part = lambda n, heads: (h @ w[p + n].t() + w[p + n + ".b"]).unflatten(-1, (heads, -1))
        q, k, v = _turn(part("q", H), m["rot"]), _turn(part("k", G), m["rot"]), part("v", G)
        if first:
            v = (1 - w[p + "vmix"]) * v + w[p + "vmix"] * first[0]
        else:
            first.append(v)
        return _attend(q, k, v, m["scale"], m["mask"]["size"], cap=m.get("softcap") or 0.0, sink=w[p + "sink"]) @ w[p + "o"].t()

    def glu(p, h, limit):
        g, u = (h @ w[p + "gate"].t()).clamp(max=limit), (h @ w[p + "up"].t()).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[p + "down"].t()

    def mixture(p, m, h):
        best = (h @ w[p + "router"].t()).topk(m["router"]["top"], -1)
        y = _experts(h, best.indices, torch.softmax(best.values, -1), lambda e, x: glu(f"{p}e{e}.", x, m["expert"]["limit"]))
        return y + torch.sigmoid(h @ w[p + "shared.sg"].t()) * glu(p + "shared.", h, m["shared"]["limit"])
    x = w["embed"][ids]
    for i, L in enumerate(cfg.layers):
        p = f"l{i}."
        h = _rms(x, eps) * w[p + "norm1"]
        x = x + mult * (delta if L.type == "delta" else attention)(p + "mix.", L.mixer, h) * w[p + "ls1"]
        h = _rms(x, eps) * w[p + "norm2"]
        x = x + mult * mixture(p + "mlp.", L.mlp, h.flatten(0, 1)).view_as(h) * w[p + "ls2"]
        side = w["side.embed"][ids][..., i * cfg.side_dim:(i + 1) * cfg.side_dim]
        x = x + mult * _rms((_gelu(x @ w[p + "side.gate"].t()) * side) @ w[p + "side.proj"].t(), eps) * w[p + "side.norm"]
    return _rms(x, eps) * w["final.norm"], w["head"]


def _dironex(w, cfg, ids):
    eps = cfg.eps

    def attention(p, m, h):
        H, G, dim = m["heads"], m["kv_heads"], m["dim"]
        q = _rms((h @ w[p + "q"].t()).unflatten(-1, (H, dim)), eps) * w[p + "q.norm"]
        k = _rms((h @ w[p + "k"].t()).unflatten(-1, (G, dim)), eps) * w[p + "k.norm"]
        return _attend(q, k, (h @ w[p + "v"].t()).unflatten(-1, (G, m["vdim"])), m["scale"], m["mask"]["size"]) @ w[p + "o"].t()

    def latent(p, m, h):
        H, dim, rd, r = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        q = ((_rms(h @ w[p + "dq"].t(), eps) * w[p + "dq.norm"]) @ w[p + "uq"].t()).unflatten(-1, (H, dim + rd))
        q = torch.cat([q[..., :dim], _turn(q[..., dim:], m["rot"])], -1)
        down = h @ w[p + "dkv"].t()
        c, shared = _rms(down[..., :r], eps) * w[p + "dkv.norm"], _turn(down[:, :, None, r:], m["rot"])
        k = torch.cat([(c @ w[p + "uk"].t()).unflatten(-1, (H, dim)), shared.expand(-1, -1, H, -1)], -1)
        o = _attend(q, k, (c @ w[p + "uv"].t()).unflatten(-1, (H, m["vdim"])), m["scale"])
        return (o * torch.sigmoid(h @ w[p + "g"].t())) @ w[p + "o"].t()

    def xielu(z, a, b):
        return torch.where(z > 0, F.softplus(a) * z * z, (0.5 + F.softplus(b)) * (torch.expm1(z.clamp(max=0)) - z)) + z / 2

    def mixture(p, r, h):
        z = torch.sigmoid(h @ w[p + "router"].t())
        g = r.get("groups") or {"count": 1, "keep": 1}
        choice = (z + w[p + "correction"]).unflatten(-1, (g["count"], -1))
        kept = choice.topk(min(2, choice.shape[-1]), -1).values.sum(-1).topk(g["keep"], -1).indices
        shut = torch.ones(choice.shape[:2], dtype=torch.bool, device=h.device).scatter(1, kept, False)
        top = choice.masked_fill(shut[..., None], float("-inf")).flatten(1).topk(r["top"], -1).indices
        v = z.gather(1, top)
        return _experts(h, top, v / (v.sum(-1, keepdim=True) + 1e-20) * r["scale"],
                        lambda e, x: (x @ w[f"{p}e{e}.up"].t()).clamp(min=0).square() @ w[f"{p}e{e}.down"].t())
    X = [w["embed"][ids] * cfg.embed_scale] * cfg.streams
    for i, L in enumerate(cfg.layers):
        for k in (1, 2):
            p = f"l{i}."
            h = _rms(sum(a * x for a, x in zip(w[f"{p}hc{k}.in"], X)), eps) * w[f"{p}norm{k}"]
            h = h + _conv(h, w[f"{p}canon{k}"])
            if k == 1:
                y = (attention if L.type == "attention" else latent)(p + "mix.", L.mixer, h)
            elif L.mlp["kind"] == "dense":
                y = xielu(h @ w[p + "mlp.up"].t(), *w[p + "mlp.act"]) @ w[p + "mlp.down"].t()
            else:
                y = mixture(p + "mlp.", L.mlp["router"], h.flatten(0, 1)).view_as(h)
            mix, out = w[f"{p}hc{k}.mix"], w[f"{p}hc{k}.out"]
            X = [sum(mix[s, t] * X[s] for s in range(cfg.streams)) + cfg.residual_mult * out[t] * y for t in range(cfg.streams)]
    return _rms(sum(X), eps) * w["final.norm"], w["head"]
