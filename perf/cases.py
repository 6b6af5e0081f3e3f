"""Performance cases of the token loop: what is timed, on which inputs, and what the results have to be.

The models are the benchmark's own (`lumi_b200/synth.py`, `bench.py`): the 48-layer base model in fp32 and bf16, the byte-level
throughput sweep at a quarter of its depth (three sets of its states fit one card), the hybrid with attention, and the two designs that
list their layers at both benchmark widths.  Weights are random, drawn on the device from a fixed seed, and loaded once per
process, as a program that serves a model does; prompts and replies come from the case's seed.

`op` says which calls one pass makes:
  generate  reset, `generate` (greedy), then one step on its last token for the logits that follow
  serve     reset, `prefill` of the prompts, then `new` steps with sampling; the fed tokens are given, so that two implementations
            whose logits differ in the last bits stay on the same text
  step      `new` steps of sequences that go on from pass to pass (a server between two arrivals)
  prefill   reset, `prefill` (or `prefill_ragged` for prompts of different lengths), then one step on the first tokens of the replies,
            which reads every state and cache that the prompts left
  score     reset, `score`: log-probabilities at every position
  extend    reset of one slot, its tokens through `extend` in portions, the logits of each portion's last places
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

import lumi_b200
from lumi_b200 import synth, zozonex, zutazen

VOCAB = 32000


# ---------------------------------------------------------------------------------------------- models
def _zozonex_config(name):
    width, n, (heads, dk, dv), (ah, ag, ad), window, ff = {
        "w1024": (1024, 12, (16, 64, 128), (16, 4, 64), 1024, 4224),
        "w2048": (2048, 6, (16, 128, 128), (32, 8, 64), 1024, 8448)}[name]
    layers, shared = [], None
    for i in range(n):
        if (i + 1) % 6:
            layers.append(zozonex.delta(heads, dk, dv))
        else:
            layers.append(zozonex.attention(ah, ad, window, kv_heads=ag, ff=ff, kv_from=shared))
            shared = i if shared is None else None
    return zozonex.config(width, VOCAB, layers, max_seq_len=8192)


def _zutazen_config(name):
    width, n, (rh, rd), blocks, (lh, ld, lr, lv, rank), window, ff, experts = {
        "w1024": (1024, 12, (8, 128), 8, (16, 64, 32, 64, 256), 1024, 2816, (16, 2, 1408)),
        "w2048": (2048, 6, (16, 128), 16, (16, 128, 64, 128, 512), 1024, 5632, (32, 4, 1408))}[name]
    dense = zutazen.dense(ff)
    kinds = [zutazen.retention(rh, rd, rd, mlp=dense), zutazen.rglru(width, blocks, mlp=zutazen.moe(*experts)),
             zutazen.retention(rh, rd, rd, mlp=dense), zutazen.rglru(width, blocks, mlp=dense), zutazen.retention(rh, rd, rd, mlp=dense),
             zutazen.latent_attention(lh, ld, lr, lv, rank, window, mlp=dense)]
    return zutazen.config(width, VOCAB, [kinds[i % 6] for i in range(n)], max_seq_len=8192)


def _config(model):
    if model.startswith("base"):
        return synth.base_config(max_seq_len=4096)
    if model == "byte":
        return synth.base_config(n_layers=24, byte_level=True, max_seq_len=4096)
    if model == "hybrid":
        return synth.base_config(attention_interval=6, attn_mlp_dim=2816, attn_rope_base=10000.0, max_seq_len=4096)
    design, size = model.split("_")
    return (_zozonex_config if design == "zozonex" else _zutazen_config)(size)


def _specs(cfg):
    """(name, shape, distribution, scale, is a matrix) of every tensor."""
    if isinstance(cfg, synth.ModelConfig):
        return [("item." + n, shape, {"h_init": "normal", "ones": "near_one"}.get(kind, kind), scale, kind == "normal")
                for n, shape, kind, scale in synth.tensor_specs(cfg)]
    out = []
    for n, shape, kind in (zozonex if isinstance(cfg, zozonex.ZozonexConfig) else zutazen).tensor_specs(cfg):
        around_one = kind == "weight" or (kind == "norm" and isinstance(cfg, zutazen.ZutazenConfig))
        dist = "near_one" if around_one else kind if kind in ("a_log", "dt_bias", "lam") else "normal"
        scale = {"matrix": shape[-1] ** -0.5, "embed": 0.3, "conv": 0.6, "bias": 0.3, "norm": 0.2}.get(kind, 0.2)
        out.append((n, shape, dist, scale, True))
    return out


_RANGES = {"a_log": (-3.0, 2.0), "lam": (-6.0, 0.0)}


def _tensor(cfg, spec):
    """The values of one tensor (fp32, on the device): the same in every process."""
    name, shape, dist, scale, _ = spec
    g = torch.Generator(device="cuda")
    g.manual_seed(zlib.crc32(name.encode()))
    if dist == "normal":
        return torch.randn(shape, generator=g, device="cuda") * scale
    if dist == "near_one":
        return 1.0 + 0.1 * torch.randn(shape, generator=g, device="cuda")
    lo, hi = _RANGES.get(dist) or ((-4.0, -1.0) if isinstance(cfg, synth.ModelConfig) else (-4.0, 1.0))
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _is_bf16(model, spec):
    return model != "base_f32" and spec[4]


_models = {}


def _model(model):
    if model not in _models:
        cfg = _config(model)

        def tensors():
            for spec in _specs(cfg):
                t = _tensor(cfg, spec)
                if _is_bf16(model, spec):
                    yield spec[0], synth.BF16, t.bfloat16().view(torch.int16).cpu().numpy().view(np.uint16)
                else:
                    yield spec[0], synth.F32, t.cpu().numpy()

        _models[model] = lumi_b200.NmModel.from_tensors(cfg, tensors())
    return _models[model]


# ---------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one user at the fp32 checkpoint, as the reference's `generate` command runs it: latency of a token
        {"name": "generate_f32_1", "op": "generate", "model": "base_f32", "batch": 1, "prompt": 32, "new": 64},
        # a chat turn of one user, streamed token by token with sampling, on the model with attention
        {"name": "chat_hybrid_1", "op": "serve", "model": "hybrid", "batch": 1, "prompt": 203, "new": 48, "top_k": 50},
        # evaluation of an fp32 checkpoint: perplexity windows
        {"name": "score_f32_4", "op": "score", "model": "base_f32", "batch": 4, "prompt": 96},
        # a server with a moderate load between two arrivals
        {"name": "step_base_64", "op": "step", "model": "base_bf16", "batch": 64, "prompt": 16, "new": 16},
        # throughput decoding: as many sequences as a card is given
        {"name": "step_byte_2048", "op": "step", "model": "byte", "batch": 2048, "prompt": 8, "new": 2},
        # a batch of long prompts
        {"name": "prefill_base_32", "op": "prefill", "model": "base_bf16", "batch": 32, "prompt": 1024},
        # whole requests in a batch: prompts, then sampled replies
        {"name": "serve_hybrid_128", "op": "serve", "model": "hybrid", "batch": 128, "prompt": 256, "new": 32, "top_k": 50},
        # long prompts through the delta rule and windowed attention
        {"name": "prefill_zozonex_16", "op": "prefill", "model": "zozonex_w1024", "batch": 16, "prompt": 2048},
        # its decode steps, windows full
        {"name": "step_zozonex_64", "op": "step", "model": "zozonex_w1024", "batch": 64, "prompt": 1100, "new": 16},
        # prompts of different lengths through retention, recurrence, latent attention and experts
        {"name": "prefill_zutazen_48_ragged", "op": "prefill", "model": "zutazen_w1024", "batch": 48, "prompt": 512, "ragged": True},
        # the wide size's decode steps, windows full
        {"name": "step_zutazen_128", "op": "step", "model": "zutazen_w2048", "batch": 128, "prompt": 1100, "new": 16},
        # one sequence in portions: a follow-up question, then guessed tokens to be checked
        {"name": "extend_zutazen", "op": "extend", "model": "zutazen_w1024", "batch": 1, "prompt": 77, "portion": 23, "want": 5},
    ]


# op -> (model, largest batch, shortest and longest prompt, fewest and most new tokens)
_DRAWN = {
    "generate": [("base_f32", 6, 5, 100, 16, 64), ("base_bf16", 12, 5, 300, 16, 64)],
    "serve": [("hybrid", 160, 20, 600, 8, 48), ("zozonex_w2048", 64, 40, 700, 8, 32), ("zutazen_w1024", 64, 40, 700, 8, 32)],
    "score": [("base_f32", 8, 20, 120, 0, 0), ("hybrid", 24, 150, 1000, 0, 0)],
    "step": [("base_bf16", 256, 8, 40, 8, 16), ("byte", 2048, 4, 12, 2, 4), ("zozonex_w1024", 200, 1030, 1200, 8, 16),
             ("zutazen_w2048", 150, 1030, 1200, 8, 16)],
    "prefill": [("base_bf16", 64, 20, 1500, 0, 0), ("zozonex_w1024", 40, 50, 2500, 0, 0), ("zutazen_w1024", 64, 50, 1500, 0, 0)],
    "extend": [("zozonex_w1024", 1, 30, 900, 0, 0), ("zutazen_w1024", 1, 30, 900, 0, 0)],
}


def _span(rng, lo, hi):
    return lo if hi <= lo else min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        op = rng.choice(sorted(_DRAWN))
        model, batch, t0, t1, n0, n1 = rng.choice(_DRAWN[op])
        case = {"op": op, "model": model, "batch": _span(rng, 1, batch), "prompt": _span(rng, t0, t1)}
        if n1:
            case["new"] = _span(rng, n0, n1)
        if op == "serve":
            case["top_k"] = rng.choice([0, 50])
        if op == "prefill" and case["batch"] > 1 and rng.random() < 0.5:
            case["ragged"] = True
        if op == "extend":
            case["portion"] = _span(rng, 5, min(200, case["prompt"]))
            case["want"] = rng.randint(1, min(5, case["portion"]))
        if _cost(case) <= most:
            return case


# ---------------------------------------------------------------------------------------------- inputs and passes
def _texts(case, seed):
    """Prompts [batch, prompt], replies [batch, new] and the prompts' lengths."""
    g = np.random.Generator(np.random.Philox(key=[seed & 0xFFFFFFFFFFFFFFFF, 77]))
    V = _config(case["model"]).vocab_size
    B, T = case["batch"], case["prompt"]
    prompts = g.integers(3, V, size=(B, T), dtype=np.uint32)
    replies = g.integers(3, V, size=(B, max(1, case.get("new", 0))), dtype=np.uint32)
    lengths = np.full(B, T, dtype=np.int32)
    if case.get("ragged"):
        lengths = g.integers(max(1, T // 8), T + 1, size=B).astype(np.int32)
        lengths[g.integers(0, B)] = T
    return prompts, replies, lengths


def prepare(case, seed):
    prompts, replies, lengths = _texts(case, seed)
    sess = _model(case["model"]).init_states(case["batch"], case["prompt"] + case.get("new", 0) + 2)
    state = {"case": case, "sess": sess, "prompts": prompts, "replies": replies, "lengths": lengths, "sampling": None}
    if case.get("top_k"):
        state["sampling"] = lumi_b200.Sampling(0.8, case["top_k"], seed & 0xFFFFFFFF, 2, 1)
    if case["op"] == "step":
        sess.prefill(prompts, want_logits=False)
    return state


def _steps(state):
    """The replies' tokens one by one; the tokens chosen after each and the logits after the last."""
    sess, replies = state["sess"], state["replies"]
    chosen, logits = [], None
    for i in range(replies.shape[1]):
        logits, token = sess.forward_step(replies[:, i], state["sampling"], i, want_logits=i + 1 == replies.shape[1])
        chosen.append(token)
    return np.stack(chosen).astype(np.int64), logits


def _portions(case):
    T, p, w = case["prompt"], case["portion"], case["want"]
    return [(t, min(T, t + p), list(range(max(0, min(T, t + p) - t - w), min(T, t + p) - t))) for t in range(0, T, p)]


def run(state):
    case, sess, prompts = state["case"], state["sess"], state["prompts"]
    op = case["op"]
    if op == "step":
        tokens, logits = _steps(state)
        return {"tokens": tokens, "logits": logits}
    if op == "extend":
        sess.reset([0])
        return {"logits": np.concatenate([sess.extend(prompts[0, a:b], want) for a, b, want in _portions(case)])}
    sess.reset()
    if op == "generate":
        tokens = sess.generate(prompts, case["new"], ignore_eos=True)[0]
        logits, _ = sess.forward_step(tokens[:, -1])
        return {"tokens": tokens.astype(np.int64), "logits": logits}
    if op == "score":
        return {"logprobs": sess.score(prompts)}
    first = sess.prefill_ragged(prompts, state["lengths"]) if case.get("ragged") else sess.prefill(prompts)
    tokens, logits = _steps(state)
    return {"first": first, "tokens": tokens, "logits": logits}


# ---------------------------------------------------------------------------------------------- work
def _layer_counts(cfg):
    """Weights of the layers that a row multiplies with, weights that `rows` rows read, state bytes of a sequence (read and written by a
    step), recurrence flops of a token, cache bytes of a token, attention flops of a (query, key) pair, window."""
    if isinstance(cfg, synth.ModelConfig):
        D, n_attn = cfg.d_model, cfg.n_attn_layers()
        n_mamba = cfg.n_layers - n_attn
        w = n_mamba * D * (cfg.in_proj_out + cfg.d_inner) + n_attn * (2 * D * D + 2 * D * cfg.attn_kv_dim + 3 * D * cfg.mlp_dim)
        state = cfg.n_heads * (cfg.head_dim * cfg.d_state + cfg.head_dim + cfg.d_state + cfg.d_state // 2) * 4
        return {"active": w, "read": lambda rows: w, "state": n_mamba * state, "scan": n_mamba * 6 * cfg.d_inner * cfg.d_state,
                "cache": n_attn * 2 * cfg.attn_kv_dim, "pair": n_attn * 4 * D, "window": 1 << 30}
    D, act, fixed, experts, state, scan, cache, pair, window = cfg.d_model, 0, 0, [], 0, 0, 0, 0, 1 << 30
    for L in cfg.raw["layers"]:
        m, f = L["mixer"], L.get("mlp")
        gates = 2 if isinstance(cfg, zozonex.ZozonexConfig) else 3
        if L["type"] in ("delta", "retention"):
            H, dk, dv = m["heads"], m["dim"], m["vdim"]
            g = m.get("kv_heads", H)
            fixed += D * (2 * g * dk + 3 * H * dv + (2 * H if L["type"] == "delta" else 0))
            state += 4 * H * dk * dv
            scan += (8 if L["type"] == "delta" else 5) * H * dk * dv
        elif L["type"] == "rglru":
            C = m["width"]
            fixed += 3 * D * C + 2 * C * C // m["blocks"]
            state += 4 * C * (1 + m["conv"])
        elif L["type"] == "attention":
            H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            own = m.get("kv_from") is None
            fixed += D * (H * (dk + dv) + (G * (dk + dv) if own else 0))
            cache += G * (dk + dv) if own else 0
            pair += 2 * H * (dk + dv)
            window = m["mask"]["size"]
        else:
            H, d, r, dv, c = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            fixed += D * (H * (d + r) + c + r + 2 * H * dv) + c * H * (d + dv)
            cache += c + r
            pair += 2 * H * (d + r + dv)
            window = m["mask"]["size"]
        if f and f["kind"] == "dense":
            fixed += gates * D * f["ff"]
        elif f:
            E, top, w = f["router"]["experts"], f["router"]["top"], 3 * D * f["expert"]["ff"]
            fixed += E * D
            act += top * w
            experts.append((E, top, w))
    return {"active": fixed + act, "read": lambda rows: fixed + sum(w * min(E, E * (1 - (1 - top / E) ** rows)) for E, top, w in experts),
            "state": state, "scan": scan, "cache": cache, "pair": pair, "window": window}


def work(case):
    cfg = _config(case["model"])
    k, e = _layer_counts(cfg), 4 if case["model"] == "base_f32" else 2
    B, T, op, n = case["batch"], case["prompt"], case["op"], case.get("new", 0)
    head = cfg.vocab_size * cfg.d_model
    tokens = int(_texts(case, 0)[2].sum()) if case.get("ragged") else B * T
    pairs = lambda a, b: sum(min(t + 1, k["window"]) for t in range(a, b))  # noqa: E731

    def prompt(heads):
        """One reading of the weights, the rows of the embedding, states and cache written once."""
        return (e * (k["read"](tokens) + (head if heads else 0) + tokens * cfg.d_model) + B * k["state"] + e * tokens * k["cache"] + 4 * heads * cfg.vocab_size,
                2 * k["active"] * tokens + 2 * head * heads + tokens * k["scan"] + tokens / T * k["pair"] * pairs(0, T))

    def steps(first, count):
        """Each step reads the weights, states and caches, and writes the states."""
        seen = pairs(first, first + count)
        return (count * (e * (k["read"](B) + head) + 2 * B * k["state"]) + e * B * seen * k["cache"] + 4 * B * cfg.vocab_size,
                B * (count * (2 * k["active"] + 2 * head + k["scan"]) + seen * k["pair"]))

    if op == "step":
        parts = [steps(T, n)]
    elif op == "generate":
        parts = [prompt(B), steps(T, n)]
    elif op == "serve":
        parts = [prompt(B), steps(T, n)]
    elif op == "score":
        parts = [prompt(B * (T - 1))]
        parts[0] = (parts[0][0] - 4 * B * (T - 1) * cfg.vocab_size + 4 * B * (T - 1), parts[0][1])
    elif op == "extend":
        each = _portions(case)
        by, fl = prompt(sum(len(w) for _, _, w in each))
        parts = [(by + (len(each) - 1) * (e * (k["read"](case["portion"]) + head) + 2 * k["state"]), fl)]
    else:
        parts = [prompt(B), steps(T, 1)]
    return {"bytes": int(sum(p[0] for p in parts)), "flops": int(sum(p[1] for p in parts))}


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / 6e14) + 1e-3 * case.get("new", 0) / 4


def tolerance(case):
    """About four times the distance from 64 bits that was measured: fp32 weights 1.1e-6 (fp32 throughout); bf16 weights on the hybrid family
    2e-5 to 3e-5 (activations enter the products as two bf16 halves each); the listed designs 2e-4 to 1.4e-3 (bf16 caches and
    expanded keys and values, few rows).  Whole values are chosen tokens: near ties may fall either way."""
    rel = {"base_f32": 5e-6, "base_bf16": 1.2e-4, "byte": 1.2e-4, "hybrid": 1.2e-4}.get(case["model"], 5e-3)
    return {"rel": rel, "max": 10 * rel, "differ": 0.02}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
class _Wide:
    """Tensors by name in float64, rounded as the model holds them."""

    def __init__(self, model):
        self.model, self.cfg = model, _config(model)
        self.by_name = {s[0]: s for s in _specs(self.cfg)}

    def __getitem__(self, name):
        spec = self.by_name[name]
        t = _tensor(self.cfg, spec)
        return (t.bfloat16() if _is_bf16(self.model, spec) else t).double()


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn_pairs(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)


def _angles(T, dims, base):
    f = float(base) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    a = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * f
    return torch.cos(a), torch.sin(a)


def _causal_attention(q, k, v, scale, window, sink):
    """q [B, T, H, d], k [B, T, G, d], v [B, T, G, dv] -> [B, T, H * dv]"""
    B, T, H, _ = q.shape
    G = k.shape[2]
    i = torch.arange(T, device="cuda")
    ago = i[:, None] - i[None, :]
    hidden = (ago < 0) | (ago >= (window or T + 1))
    out = torch.empty(B, T, H, v.shape[3], dtype=torch.float64, device="cuda")
    for b in range(B):
        s = torch.einsum("tgjd,sgd->gjts", q[b].view(T, G, H // G, -1), k[b]).mul_(scale).masked_fill_(hidden, -math.inf)
        m = s.amax(-1, keepdim=True)
        if sink:
            m = m.clamp(min=0.0)
        s = s.sub_(m).exp_()
        den = s.sum(-1, keepdim=True) + (torch.exp(-m) if sink else 0.0)
        out[b] = torch.einsum("gjts,sgd->tgjd", s / den, v[b]).reshape(T, H, -1)
    return out.flatten(2)


def _mamba_layer(W, cfg, p, x):
    B, T, _ = x.shape
    H, P, N, G = cfg.n_heads, cfg.head_dim, cfg.d_state, cfg.n_groups
    proj = (_rms(x, 1e-5) * W[p + "norm.gamma"]) @ W[p + "in_proj.weight"].T
    xs, z, b, c, dt, lam, dda, theta = proj.split([cfg.d_inner, cfg.d_inner, cfg.bc_size, cfg.bc_size, H, H, H, H * N // 2], -1)
    silu = torch.nn.functional.silu
    sp = lambda v: torch.logaddexp(v, torch.zeros_like(v))  # noqa: E731
    xs = silu(xs).view(B, T, H, P)
    b = (_rms(b, 1e-5) * W[p + "b_norm.gamma"] + W[p + "b_bias"]).view(B, T, G, N).repeat_interleave(H // G, 2)
    c = (_rms(c, 1e-5) * W[p + "c_norm.gamma"] + W[p + "c_bias"]).view(B, T, G, N).repeat_interleave(H // G, 2)
    dt = sp(dt + W[p + "ssm.dt_bias"])
    decay = torch.cumsum((-sp(dda)).clamp(-1e6, -1e-4) * dt, 1)                       # [B, T, H]: log of the product up to t
    angle = torch.cumsum(dt[..., None] * torch.tanh(theta.view(B, T, H, N // 2)) * float(np.float32(np.pi)), 1)
    cos, sin = torch.cos(angle), torch.sin(angle)
    b, c = _turn_pairs(b, cos, sin), _turn_pairs(c, cos, sin)
    lam = torch.sigmoid(lam)
    # h_t = a_t h_(t-1) + a_t (1 - lam_t) u_(t-1) + lam_t u_t: u_s reaches h_t with the decay between them times lam_s (+ 1 - lam_(s+1) for s < t)
    later = torch.cat([1.0 - lam[:, 1:], torch.zeros_like(lam[:, :1])], 1)
    y = torch.empty(B, T, H, P, dtype=torch.float64, device="cuda")
    step = max(1, int(2 ** 28 / (H * T * T)))
    upper = torch.ones(T, T, dtype=torch.bool, device="cuda").triu_(1)
    for i in range(0, B, step):
        s = slice(i, i + step)
        d = decay[s].transpose(1, 2)                                                  # [b, H, T]
        mix = (d[..., :, None] - d[..., None, :]).masked_fill_(upper, -math.inf).exp_()
        weight = (lam[s] + later[s]).transpose(1, 2)[..., None, :].expand_as(mix).clone()
        weight.diagonal(dim1=-2, dim2=-1).copy_(lam[s].transpose(1, 2))
        mix.mul_(weight).mul_(c[s].transpose(1, 2) @ b[s].permute(0, 2, 3, 1))
        y[s] = (mix @ xs[s].transpose(1, 2)).transpose(1, 2)
    y += (torch.exp(decay) * torch.einsum("bthn,hn->bth", c, W[p + "ssm.h_init"]))[..., None]
    y += W[p + "ssm.d"][:, None] * xs
    return x + (y.flatten(2) * silu(z)) @ W[p + "out_proj.weight"].T


def _hybrid(W, cfg, tokens):
    x = W["item.embedding.weight"][tokens]
    T = tokens.shape[1]
    for i in range(cfg.n_layers):
        p = "item.blocks.%d." % i
        if not cfg.is_attention_layer(i):
            x = _mamba_layer(W, cfg, p, x)
            continue
        H, G, hd = cfg.attn_n_heads, cfg.attn_kv_heads, cfg.attn_head_dim
        h = _rms(x, 1e-5) * W[p + "attn_norm.gamma"]
        q, k, v = ((h @ W[p + n + "_proj.weight"].T).unflatten(-1, (-1, hd)) for n in "qkv")
        cos, sin = (a[:, None, :] for a in _angles(T, hd, cfg.attn_rope_base))
        x = x + _causal_attention(_turn_pairs(q, cos, sin), _turn_pairs(k, cos, sin), v, hd ** -0.5, 0, False) @ W[p + "attn_out_proj.weight"].T
        h = _rms(x, 1e-5) * W[p + "mlp_norm.gamma"]
        x = x + (torch.sigmoid(h @ W[p + "mlp_gate.weight"].T) * (h @ W[p + "mlp_up.weight"].T)) @ W[p + "mlp_down.weight"].T
    return x, lambda r: (_rms(r, 1e-5) * W["item.final_norm.gamma"]) @ W["item.embedding.weight"].T


def _conv(x, w):
    taps = w.shape[1]
    pad = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    return sum(pad[:, j:j + x.shape[1]] * w[:, j] for j in range(taps))


def _zozonex(W, cfg, tokens):
    eps, D, T = cfg.raw["norm"]["eps"], cfg.d_model, tokens.shape[1]
    silu = torch.nn.functional.silu
    cos, sin = _angles(T, D, 10000.0)
    x = W["embed"][tokens] * cfg.raw["embedding"]["scale"] + torch.stack([sin, cos], -1).flatten(-2)
    shared = {}
    for i, L in enumerate(cfg.raw["layers"]):
        p, m = "l%d." % i, L["mixer"]
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        proj = lambda n: x @ W[p + "mix." + n].T  # noqa: E731
        if L["type"] == "delta":
            q, k, v = (silu(_conv(proj(n), W[p + "mix." + n + ".conv"])) for n in "qkv")
            unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            q, k = (unit(t.unflatten(-1, (G, dk))).repeat_interleave(H // G, 2) for t in (q, k))
            q, v = q * dk ** -0.5, v.unflatten(-1, (H, dv))
            beta = torch.sigmoid(proj("b"))
            g = torch.exp(-torch.exp(W[p + "mix.A_log"]) * torch.nn.functional.softplus(proj("a") + W[p + "mix.dt_bias"], threshold=700.0))
            S = torch.zeros(x.shape[0], H, dk, dv, dtype=torch.float64, device="cuda")
            o = torch.empty_like(v)
            for t in range(T):
                S.mul_(g[:, t, :, None, None])
                u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[:, :, 0])
                S.addcmul_(k[:, t, :, :, None], u[:, :, None, :])
                o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
            y = (_rms(o, eps) * W[p + "mix.norm"] * silu(proj("g").unflatten(-1, (H, dv)))).flatten(2)
        else:
            if m.get("kv_from") is None:
                shared[i] = _rms(proj("k").unflatten(-1, (G, dk)), eps), proj("v").unflatten(-1, (G, dv))
            k, v = shared[m.get("kv_from", i) if m.get("kv_from") is not None else i]
            y = _causal_attention(_rms(proj("q").unflatten(-1, (H, dk)), eps), k, v, m["scale"], m["mask"]["size"], True)
        x = x + _rms(y @ W[p + "mix.o"].T, eps) * (1.0 + W[p + "norm1"])
        if L.get("mlp"):
            a = torch.relu(x @ W[p + "mlp.up"].T)
            x = x + _rms((a * a) @ W[p + "mlp.down"].T, eps) * (1.0 + W[p + "norm2"])
    return x, lambda r: (_rms(r, eps) * (1.0 + W["final.norm"])) @ W["embed"].T


def _zutazen(W, cfg, tokens):
    eps, T, B = cfg.raw["norm"]["eps"], tokens.shape[1], tokens.shape[0]
    silu = torch.nn.functional.silu
    x = W["embed"][tokens] * cfg.raw["embedding"]["scale"]
    for i, L in enumerate(cfg.raw["layers"]):
        p, m, f = "l%d." % i, L["mixer"], L["mlp"]
        h = _rms(x, eps) * W[p + "norm1"]
        proj = lambda n: h @ W[p + "mix." + n].T  # noqa: E731
        if L["type"] == "retention":
            H, dk, dv = m["heads"], m["dim"], m["vdim"]
            cos, sin = (a[:, None, :] for a in _angles(T, dk, m["rot"]["base"]))

            def half(t):
                a, b = t[..., :dk // 2], t[..., dk // 2:]
                return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

            q, k = (half(proj(n).unflatten(-1, (H, dk))) for n in "qk")
            k, v = k * dk ** -0.5, proj("v").unflatten(-1, (H, dv))
            t = torch.arange(T, dtype=torch.float64, device="cuda")
            ago = t[:, None] - t[None, :]
            o = torch.empty(B, T, H, dv, dtype=torch.float64, device="cuda")
            for j in range(H):
                mix = torch.where(ago >= 0, float(m["decay"][j]) ** ago.clamp(min=0), 0.0)
                for b in range(0, B, 16):
                    o[b:b + 16, :, j] = ((q[b:b + 16, :, j] @ k[b:b + 16, :, j].transpose(1, 2)) * mix) @ v[b:b + 16, :, j]
            y = (_rms(o, eps).flatten(2) * silu(proj("g"))) @ W[p + "mix.o"].T
        elif L["type"] == "rglru":
            n = m["blocks"]
            gate = torch.nn.functional.gelu(proj("y") + W[p + "mix.y.b"], approximate="tanh")
            u = _conv(proj("x") + W[p + "mix.x.b"], W[p + "mix.conv"]) + W[p + "mix.conv.b"]
            blocks = lambda q: torch.sigmoid(torch.einsum("bij,...bj->...bi", W[p + "mix." + q], u.unflatten(-1, (n, -1))) + W[p + "mix." + q + ".b"]).flatten(-2)  # noqa: E731
            log_a = -8.0 * blocks("ra") * torch.nn.functional.softplus(W[p + "mix.lam"], threshold=700.0)
            a, new = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * blocks("ri") * u
            S = torch.zeros_like(u[:, 0])
            for t in range(T):
                S = a[:, t] * S + new[:, t]
                u[:, t] = S
            y = (u * gate) @ W[p + "mix.o"].T
        else:
            H, d, r, dv, c = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            cos, sin = _angles(T, r, m["rot"]["base"])
            q, lat = proj("q").unflatten(-1, (H, d + r)), proj("dkv")
            q = torch.cat([q[..., :d], _turn_pairs(q[..., d:], cos[:, None, :], sin[:, None, :])], -1)
            kr = _turn_pairs(lat[..., c:], cos, sin)[:, :, None, :].expand(B, T, H, r)
            lat = _rms(lat[..., :c], eps) * W[p + "mix.dkv.norm"]
            k = torch.cat([(lat @ W[p + "mix.uk"].T).unflatten(-1, (H, d)), kr], -1)
            o = _causal_attention(q, k, (lat @ W[p + "mix.uv"].T).unflatten(-1, (H, dv)), m["scale"], m["mask"]["size"], False)
            y = (o * torch.sigmoid(proj("g"))) @ W[p + "mix.o"].T
        x = x + y
        h = _rms(x, eps) * W[p + "norm2"]
        if f["kind"] == "dense":
            a = torch.relu(h @ W[p + "mlp.gate"].T + W[p + "mlp.gate.b"]) * (h @ W[p + "mlp.up"].T + W[p + "mlp.up.b"])
            x = x + a @ W[p + "mlp.down"].T + W[p + "mlp.down.b"]
        else:
            rows = h.flatten(0, 1)
            score, chosen = torch.sigmoid(rows @ W[p + "mlp.router"].T).topk(f["router"]["top"], -1)
            y = torch.zeros_like(rows)
            for e in range(f["router"]["experts"]):
                at, which = torch.nonzero(chosen == e, as_tuple=True)
                q, r = p + "mlp.e%d." % e, rows[at] * score[at, which][:, None]
                y.index_add_(0, at, (silu(r @ W[q + "gate"].T) * (r @ W[q + "up"].T)) @ W[q + "down"].T)
            x = x + y.view_as(x)
    return x, lambda r: (_rms(r, eps) * W["final.norm"]) @ W["head"].T


@torch.no_grad()
def _forward(model, tokens):
    """The residual stream [B, T, width] behind the last layer, and the head as a function of rows."""
    W = _Wide(model)
    form = _hybrid if isinstance(W.cfg, synth.ModelConfig) else _zozonex if isinstance(W.cfg, zozonex.ZozonexConfig) else _zutazen
    return form(W, W.cfg, torch.from_numpy(tokens.astype(np.int64)).cuda())


def exact(case, seed):
    prompts, replies, lengths = _texts(case, seed)
    op, T, B = case["op"], case["prompt"], case["batch"]
    if op == "generate":
        if case["new"] * B * (T + case["new"]) > 100_000:
            return None
        text = prompts
        for _ in range(case["new"]):          # whole sequences again for every token: no cache that could be wrong
            x, head = _forward(case["model"], text)
            text = np.concatenate([text, head(x[:, -1]).argmax(-1, keepdim=True).cpu().numpy().astype(np.uint32)], 1)
        x, head = _forward(case["model"], text)
        return {"tokens": text[:, T:].astype(np.int64), "logits": head(x[:, -1]).cpu().numpy()}
    if case.get("ragged"):                    # each reply behind its own prompt; what stands behind it is never looked at
        text, at = np.concatenate([prompts, replies], 1), np.arange(B)
        text[at, lengths] = replies[:, 0]
        x, head = _forward(case["model"], text)
        first, logits = head(x[at, lengths - 1]), head(x[at, lengths.astype(np.int64)])
        return {"first": first.cpu().numpy(), "tokens": logits.argmax(-1)[None].cpu().numpy(), "logits": logits.cpu().numpy()}
    if op in ("step", "serve", "prefill"):
        x, head = _forward(case["model"], np.concatenate([prompts, replies], 1))
        n = replies.shape[1]
        tokens = None if case.get("top_k") else np.stack([head(x[:, T + i]).argmax(-1).cpu().numpy() for i in range(n)])
        out = {"tokens": tokens, "logits": head(x[:, -1]).cpu().numpy()}
        if op != "step":
            out["first"] = head(x[:, T - 1]).cpu().numpy()
        return out
    x, head = _forward(case["model"], prompts)
    if op == "score":
        rows = [torch.log_softmax(head(x[b, :-1]), -1).cpu().numpy() for b in range(B)]
        return {"logprobs": np.stack([r[np.arange(T - 1), prompts[b, 1:].astype(np.int64)] for b, r in enumerate(rows)])}
    return {"logits": head(x[0, [a + w for a, _, want in _portions(case) for w in want]]).cpu().numpy()}
