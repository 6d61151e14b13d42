"""Workloads of the engine's model step: what a serving process has the models do, one forward a pass.

A case names a model shape (``config.preset``, cut to its first ``layers`` layers where the whole would not fit beside
copies of itself), the storage of its projections and one step of the serving loop:

* ``decode``: one token for each of ``rows`` running sequences, staged and replayed as the engine does (``set_rows``,
  ``decode``).  Context lengths lie between ``context`` and ``longest``.
* ``prefill``: ``tokens`` prompt tokens of ``rows`` sequences in one forward (``prefill_group``), each behind ``history``
  tokens that are cached already.  A sequence without history starts from a zeroed slot.
* ``mixed``: a forward over ``rows`` running sequences and ``portions`` portions of prompts, ``tokens`` tokens in all, the
  step of the families that batch both (``forward_batch``).

Weights, cached keys and values, recurrent states and tokens are drawn from the seed at the magnitudes that the shapes'
random-init weights produce; the caches' pages are in random order, as in a pool that has been in use.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from coffin_b200.config import LINEAR, first_layers, preset
from coffin_b200.models import build_model
from coffin_b200.weights.init import LM, random_state_dict
from coffin_b200.weights.quant import QWeight, W4A8Weight, is_quantizable

PAGE = 64
BUCKETS = (1, 2, 4, 8, 16, 32, 64)
DEV = "cuda"


# ---------------------------------------------------------------------------------------------- the cases
def _decode(model, layers, rows, context, longest, weights="bf16"):
    return {"kind": "decode", "model": model, "layers": layers, "weights": weights, "rows": rows, "context": context, "longest": longest}


def _prefill(model, layers, rows, tokens, history, weights="bf16"):
    return {"kind": "prefill", "model": model, "layers": layers, "weights": weights, "rows": rows, "tokens": tokens, "history": history}


def _mixed(model, layers, rows, context, longest, portions, tokens, history):
    return {"kind": "mixed", "model": model, "layers": layers, "weights": "bf16", "rows": rows, "context": context, "longest": longest,
            "portions": portions, "tokens": tokens, "history": history}


def listed():
    cases = {
        # one token of the smallest shape: launches and latency, nothing to stream
        "tiny-decode-1": _decode("tiny", 4, 1, 65, 65),
        # single-stream generation, the headline workload's step
        "4b-decode-1": _decode("qwen35-4b", 32, 1, 2111, 2111),
        # a few sequences of very different length, long ones among them: the widest step of the GEMV projections
        "4b-decode-8": _decode("qwen35-4b", 32, 8, 517, 16391),
        # a full batch of running sequences
        "4b-decode-64": _decode("qwen35-4b", 32, 64, 1031, 2047),
        # time to first token of a 2048-token prompt
        "4b-prefill-2048": _prefill("qwen35-4b", 32, 1, 2048, 0),
        # short suffixes behind a shared system prompt, grouped into one forward
        "4b-prefill-suffixes": _prefill("qwen35-4b", 32, 5, 811, 1024),
        # a late chunk of a long document, odd length
        "4b-prefill-deep": _prefill("qwen35-4b", 32, 1, 1901, 16384),
        # the 27B shape with int8 projections: 32 sequences at 4096 tokens, and a chunk of such a prompt
        "27b-int8-decode-32": _decode("qwen35-27b", 4, 32, 4096, 4607, "int8"),
        "27b-int8-prefill": _prefill("qwen35-27b", 4, 1, 2048, 2048, "int8"),
        # the routed shape with int4 projections and experts: 64 sequences at about 1024 tokens, and a prompt of that length
        "35b-a3b-w4-decode-64": _decode("qwen35-35b-a3b", 8, 64, 1024, 1279, "w4a8"),
        "35b-a3b-w4-prefill": _prefill("qwen35-35b-a3b", 8, 1, 1024, 0, "w4a8"),
        # running sequences and prompt portions in one forward (latent attention, state-space layers)
        "sukisun-mixed": _mixed("sukisun-4b", 8, 29, 301, 2047, 2, 643, 0),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("tiny", "decode", "decode", "decode", "prefill", "prefill", "prefill", "int8-decode", "int8-prefill", "w4-decode", "w4-prefill", "mixed"))
    if kind == "tiny":
        n = _log(rng, 16, 190)
        return _decode("tiny", 4, _log(rng, 1, 8), n, rng.randint(n, 190))
    if kind in ("decode", "int8-decode", "w4-decode"):
        rows = _log(rng, 1, 32 if kind == "int8-decode" else 64)
        most = min({"decode": 16384, "int8-decode": 4607, "w4-decode": 2047}[kind], 131072 // rows)
        n = _log(rng, 64, most)
        size = {"decode": ("qwen35-4b", 32, "bf16"), "int8-decode": ("qwen35-27b", 4, "int8"), "w4-decode": ("qwen35-35b-a3b", 8, "w4a8")}[kind]
        return _decode(size[0], size[1], rows, n, rng.randint(n, most), size[2])
    if kind in ("prefill", "int8-prefill", "w4-prefill"):
        rows = _log(rng, 1, 8)
        tokens = _log(rng, 16 * rows, 2048)
        most = {"prefill": 16384, "int8-prefill": 4096, "w4-prefill": 2048}[kind] // rows
        history = rng.choice((0, _log(rng, 64, most)))
        size = {"prefill": ("qwen35-4b", 32, "bf16"), "int8-prefill": ("qwen35-27b", 4, "int8"), "w4-prefill": ("qwen35-35b-a3b", 8, "w4a8")}[kind]
        return _prefill(size[0], size[1], rows, tokens, history, size[2])
    n = _log(rng, 64, 2047)
    return _mixed("sukisun-4b", 8, _log(rng, 1, 48), n, rng.randint(n, 2047), rng.randint(1, 3), _log(rng, 96, 1024), rng.choice((0, _log(rng, 64, 1024))))


# ---------------------------------------------------------------------------------------------- what a case consists of
def _spread(n, lo, hi):
    """``n`` lengths from lo to hi, in no order, hi among them."""
    if n == 1:
        return [hi]
    return [lo + round((hi - lo) * ((i * 5 % n if n % 5 else i) / (n - 1))) for i in range(n)]


def _shares(total, n):
    """``total`` split into ``n`` uneven parts of at least two."""
    w = [1.0 + (i * 7 % 5) for i in range(n)]
    parts = [max(2, int(total * x / sum(w))) for x in w]
    parts[-1] += total - sum(parts)
    return parts


def _segments(case):
    """``(tokens, cached tokens before them)`` of every sequence of the step, in the order of the slots."""
    if case["kind"] == "prefill":
        return [(n, case["history"]) for n in _shares(case["tokens"], case["rows"])]
    ones = [(1, n - 1) for n in _spread(case["rows"], case["context"], case["longest"])]
    if case["kind"] == "mixed":
        ones += [(n, case["history"]) for n in _shares(case["tokens"], case["portions"])]
    return ones


def _config(case):
    cfg = preset(case["model"])
    return cfg if case["layers"] == cfg.num_hidden_layers else first_layers(cfg, case["layers"])


def _pages(case):
    return [(n + before + PAGE - 1) // PAGE for n, before in _segments(case)]


def _gen(seed, tag):
    return torch.Generator(device=DEV).manual_seed(seed * 7919 + tag)


def _tables(case, seed):
    """Block table of every sequence: blocks of a pool of ``sum + 1`` in random order."""
    pages = _pages(case)
    order = torch.randperm(sum(pages) + 1, generator=torch.Generator().manual_seed(seed * 7919 + 1)).tolist()
    out, at = [], 0
    for p in pages:
        out.append(order[at:at + p])
        at += p
    return out


def _tokens(case, seed, cfg):
    g = torch.Generator().manual_seed(seed * 7919 + 2)
    return [torch.randint(0, cfg.vocab_size, (n,), generator=g) for n, _ in _segments(case)]


def _weights(case, seed, cfg):
    """A checkpoint of the shape: random-init bf16 tensors, projections as int8 or int4 containers where the case says so.
    In the hybrid shapes a sublayer adds to its residual as little as one of a trained model does: rows of the embedding are about
    one, and what leads back to the residual is divided by the square root of the number of sublayers."""
    sd = random_state_dict(cfg, seed, dtype=torch.bfloat16, device=DEV)
    if not case["model"].startswith("sukisun"):
        sd[LM + "embed_tokens.weight"].mul_(50)
        for key, t in sd.items():
            if key.endswith(("out_proj.weight", "o_proj.weight", "down_proj.weight", "experts.down_proj")):
                t.mul_((2 * preset(case["model"]).num_hidden_layers) ** -0.5)
    if case["weights"] == "bf16":
        return sd
    g = _gen(seed, 3)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV)
    for key, t in sd.items():
        if not is_quantizable(key, t):
            continue
        *lead, n, k = t.shape
        std = float(t.reshape(-1, k)[:8].float().std())
        if case["weights"] == "int8":
            wq = (t.float() * (32 / std)).round_().clamp_(-127, 127).to(torch.int8)
            sd[key] = QWeight(wq, std / 32 * (0.8 + 0.4 * rand(*lead, n)))
        else:
            q = ((t.transpose(-1, -2).float() * (2.4 / std)).round_().clamp_(-8, 7) + 8).to(torch.uint8)
            packed = q[..., 0::2, :] | (q[..., 1::2, :] << 4)
            sd[key] = W4A8Weight(packed.contiguous(), std / 2.4 * (0.8 + 0.4 * rand(*lead, k // 128, n)), k)
    return sd


def _wide(t, sub=None):
    """Weight ``[.., N, K]`` (expert ``sub`` of a stack) in 64 bits."""
    if isinstance(t, QWeight):
        wq, sc = (t.wq, t.scale) if sub is None else (t.wq[sub], t.scale[sub])
        return wq.double() * sc.double()[..., None]
    if isinstance(t, W4A8Weight):
        p, sc = (t.packed, t.scale) if sub is None else (t.packed[sub], t.scale[sub])
        codes = torch.stack([p & 15, p >> 4], 1).reshape(-1, p.shape[1])[:t.k].double() - 8
        return (codes * sc.double().repeat_interleave(128, 0)[:t.k]).t()
    return (t if sub is None else t[sub]).double()


def _hybrid_caches(case, seed, cfg):
    """Cached keys and values ``[layers, pool rows, heads, dim]``, recurrent states and convolution rows of all slots."""
    c, n, rows = cfg, len(_segments(case)), (sum(_pages(case)) + 1) * PAGE
    g = _gen(seed, 4)
    nl, nf = len(c.linear_layers), len(c.full_layers)
    k = torch.empty(nf, rows, c.num_key_value_heads, c.head_dim, dtype=torch.bfloat16, device=DEV)
    v = torch.empty_like(k)
    for j in range(nf):
        t = torch.randn(k[j].shape, generator=g, device=DEV)
        k[j] = t * torch.rsqrt(t.square().mean(-1, keepdim=True))           # keys are normed
        v[j] = torch.randn(k[j].shape, generator=g, device=DEV) * (0.02 * c.hidden_size ** 0.5)
    state = 0.05 * torch.randn(nl, n, c.linear_num_value_heads, c.linear_key_head_dim, c.linear_value_head_dim, generator=g, device=DEV)
    ring = (0.02 * c.hidden_size ** 0.5 * torch.randn(nl, n, 16, c.lin_conv_dim, generator=g, device=DEV)).bfloat16()
    return k, v, state, ring


def _suki_caches(case, seed, cfg):
    """Per layer: ``(latents | rotated key part)`` pool rows, or the state-space matrix and convolution rows of all slots."""
    n, rows, g, out = len(_segments(case)), (sum(_pages(case)) + 1) * PAGE, _gen(seed, 4), []
    for spec in cfg.layers:
        m = spec.mixer
        if spec.kind == "mamba2":
            out.append((0.05 * torch.randn(n, m.heads, m.state, m.vdim, generator=g, device=DEV),
                        torch.randn(n, 16, m.conv_width, generator=g, device=DEV).bfloat16()))
        else:
            out.append(torch.randn(rows, m.kv_rank + m.rot_dim, generator=g, device=DEV).bfloat16() if m.kv_from is None else None)
    return out


# ---------------------------------------------------------------------------------------------- the program
def prepare(case, seed):
    cfg, segs, tables = _config(case), _segments(case), _tables(case, seed)
    longest = max(n + b for n, b in segs)
    model = build_model(cfg, _weights(case, seed, cfg), device=DEV, max_seq=longest + 65, num_slots=len(segs), num_blocks=sum(_pages(case)) + 1,
                        max_chunk=2048, free_source=True)
    toks = _tokens(case, seed, cfg)
    if case["model"].startswith("sukisun"):
        for L, cached in zip(model.layers, _suki_caches(case, seed, cfg)):
            if L.mixer.state:
                L.mixer.state["S"].copy_(cached[0])
                L.mixer.state["ring"].copy_(cached[1])
            elif cached is not None:
                L.mixer.pool.copy_(cached)
    else:
        for t, u in zip((model.kpool, model.vpool, model.state, model.ring), _hybrid_caches(case, seed, cfg)):
            t.copy_(u)
    st = {"case": case, "model": model, "tables": tables, "tokens": toks, "segs": segs}
    if case["kind"] == "decode":
        st["bucket"] = next(b for b in BUCKETS if b >= len(segs))
        model.capture(st["bucket"])
        st["tokens"] = [int(t[0]) for t in toks]
    elif case["kind"] == "prefill":
        st["items"] = [(t.to(DEV), before, i, torch.tensor(bt, dtype=torch.int32, device=DEV))
                       for i, (t, (n, before), bt) in enumerate(zip(toks, segs, tables))]
    else:
        st["items"] = [(t.tolist(), before, i, bt) for i, (t, (n, before), bt) in enumerate(zip(toks, segs, tables))]
    return st


def run(state):
    m, case, segs = state["model"], state["case"], state["segs"]
    if case["kind"] == "decode":
        m.set_rows(state["bucket"], state["tokens"], [b for _, b in segs], list(range(len(segs))), state["tables"])
        logits = m.decode(state["bucket"])[1][:len(segs)]
    else:
        for i, (n, before) in enumerate(segs):
            if not before:
                m.zero_state(i)
        if case["kind"] == "prefill":
            logits = m.prefill_group(state["items"])
        else:
            logits = m.forward_batch(state["items"], [[n - 1] for n, _ in segs])
    if case["model"].startswith("sukisun"):
        kept = [dict(L.mixer.state) if L.mixer.state else L.mixer.pool if spec.mixer.kv_from is None else None
                for L, spec in zip(m.layers, m.cfg.layers)]
        return {"logits": logits, "layers": kept}
    return {"logits": logits, "keys": m.kpool, "values": m.vpool, "states": m.state, "rows": m.ring}


# ---------------------------------------------------------------------------------------------- what it cannot do without
def _bytes_of(t):
    if isinstance(t, (int, float)):
        return t
    return t.numel() * t.element_size()


def work(case):
    cfg, segs = _config(case), _segments(case)
    rows, outs = sum(n for n, _ in segs), len(segs)
    seen = sum(n * before + n * (n + 1) // 2 for n, before in segs)         # query-key pairs
    cached, wrote = sum(b for _, b in segs), rows
    H, V = cfg.hidden_size, cfg.vocab_size
    if case["model"].startswith("sukisun"):
        size, mults, move, flops = 2, 0, 0, 0
        for spec in cfg.layers:
            m = spec.mixer
            if spec.kind == "mamba2":
                mults += H * (m.inner + m.conv_width + m.heads) + H * m.inner
                move += 2 * outs * m.heads * m.state * m.vdim * 4
                flops += rows * m.heads * m.state * m.vdim * 5
            else:
                own = m.kv_from is None
                mults += H * m.q_rank + m.q_rank * m.heads * (m.dim + m.rot_dim) + own * H * (m.kv_rank + m.rot_dim) + H * m.heads
                mults += m.heads * m.kv_rank * (m.dim + m.vdim) + H * m.heads * m.vdim
                move += (cached + own * wrote) * (m.kv_rank + m.rot_dim) * 2
                flops += 2 * seen * m.heads * (m.dim + m.rot_dim + m.vdim)
            mults += 2 * H * spec.ff
        return {"bytes": size * (mults + H * V) + move + outs * V * 4, "flops": 2 * rows * mults + 2 * outs * H * V + flops}
    c = cfg
    size = {"bf16": 2.0, "int8": 1.0, "w4a8": 0.5 + 4 / 128}[case["weights"]]
    lin = H * (c.lin_conv_dim + c.lin_vdim + 2 * c.linear_num_value_heads) + H * c.lin_vdim
    att = H * c.head_dim * (3 * c.num_attention_heads + 2 * c.num_key_value_heads)
    mults = len(c.linear_layers) * lin + len(c.full_layers) * att
    weights = mults
    if c.is_moe:
        e, s = 3 * H * c.moe_intermediate_size, 3 * H * c.shared_expert_intermediate_size
        mults += c.num_hidden_layers * (c.num_experts_per_tok * e + s + H * c.num_experts)
        chosen = c.num_experts * (1 - (1 - c.num_experts_per_tok / c.num_experts) ** rows)
        weights += c.num_hidden_layers * (chosen * e + s + 2 / size * H * c.num_experts)
    else:
        mults += c.num_hidden_layers * 3 * H * c.intermediate_size
        weights = mults
    per = c.linear_num_value_heads * c.linear_key_head_dim * c.linear_value_head_dim
    kv = 2 * c.num_key_value_heads * c.head_dim * 2
    move = len(c.linear_layers) * outs * per * 4 * 2 + len(c.full_layers) * (cached + wrote) * kv + outs * V * 4 + rows * H * 2
    flops = 2 * rows * mults + 2 * outs * H * V + len(c.full_layers) * 4 * seen * c.num_attention_heads * c.head_dim + len(c.linear_layers) * rows * per * 6
    return {"bytes": size * (weights + H * V) + move, "flops": flops}


def tolerance(case):
    """Four times what the logits are off against 64 bits (the worst of the outputs): bf16 residuals and activations over 32 layers
    give 0.016, int8 activations over 4 layers 0.02, int4 weights over 8 layers 0.012, the 4-layer shape 0.005; at most 0.03."""
    return {"rel": 0.02 if case["model"] == "tiny" else 0.03, "max": 0.5}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _conv(x, taps, before, bias=None):
    """Causal depthwise convolution + SiLU: x ``[T, C]``, taps ``[C, n]`` oldest first, ``before [n - 1, C]`` the rows ahead of x."""
    seq = torch.cat([before, x])
    y = (seq.unfold(0, taps.shape[1], 1) * taps).sum(-1)
    return F.silu(y if bias is None else y + bias)


def _before(ring, pos, taps):
    """The raw rows ahead of position ``pos`` from a ring indexed by position modulo 16 (zeros ahead of the start)."""
    rows = [ring[p % 16] if p >= 0 else torch.zeros_like(ring[0]) for p in range(pos - taps + 1, pos)]
    return torch.stack(rows)


def _attend(q, k, v, pos0, scale):
    """Causal attention of q ``[T, H, d]`` at positions from ``pos0`` over k, v ``[S, G, d]``; blocks of queries."""
    T, H, d = q.shape
    G, out = k.shape[1], []
    kt, vt = k.permute(1, 2, 0), v.transpose(0, 1)                          # [G, d, S], [G, S, e]
    for t in range(0, T, 256):
        n = min(256, T - t)
        s = (q[t:t + n].view(n, G, H // G, d).permute(1, 2, 0, 3).reshape(G, -1, d) @ kt) * scale
        at = pos0 + t + torch.arange(n, device=q.device)
        hide = (torch.arange(k.shape[0], device=q.device)[None, :] > at[:, None]).repeat(H // G, 1)
        o = torch.softmax(s.masked_fill_(hide, -math.inf), -1) @ vt
        out.append(o.view(G, H // G, n, -1).permute(2, 0, 1, 3).reshape(n, H, -1))
    return torch.cat(out)


def _turned(x, pos0, dims, base, halves):
    """The first ``dims`` entries of x ``[T, H, n]`` rotated: entry i with i + dims / 2, or neighbours."""
    T = x.shape[0]
    a = (pos0 + torch.arange(T, device=x.device).double())[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device).double() / dims)
    c, s = a.cos()[:, None], a.sin()[:, None]
    out = x.clone()
    i, j = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    u, v = x[..., i], x[..., j]
    out[..., i], out[..., j] = u * c - v * s, v * c + u * s
    return out


def _rows_of(table, n):
    t = torch.tensor(table, device=DEV).repeat_interleave(PAGE) * PAGE + torch.arange(PAGE, device=DEV).repeat(len(table))
    return t[:n]


def _delta_scan(q, k, v, beta, g, S):
    """Gated delta rule token by token; q, k ``[T, H, dk]``, v ``[T, H, dv]``; S ``[H, dk, dv]`` is updated."""
    out, decay = torch.empty_like(v), g.exp()
    for t in range(q.shape[0]):
        S.mul_(decay[t, :, None, None])
        d = (v[t] - torch.bmm(k[t, :, None], S)[:, 0]) * beta[t, :, None]
        S.baddbmm_(k[t, :, :, None], d[:, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    return out


def _experts(c, sd, p, h):
    prob = torch.softmax(h @ _wide(sd[p + "gate.weight"]).t(), -1)
    w, idx = torch.topk(prob, c.num_experts_per_tok, -1)
    if c.norm_topk_prob:
        w = w / w.sum(-1, keepdim=True)
    out, I = torch.zeros_like(h), c.moe_intermediate_size
    for e in idx.unique().tolist():
        t, j = (idx == e).nonzero(as_tuple=True)
        gu = h[t] @ _wide(sd[p + "experts.gate_up_proj"], e).t()
        out.index_add_(0, t, w[t, j, None] * ((F.silu(gu[:, :I]) * gu[:, I:]) @ _wide(sd[p + "experts.down_proj"], e).t()))
    q = p + "shared_expert."
    s = (F.silu(h @ _wide(sd[q + "gate_proj.weight"]).t()) * (h @ _wide(sd[q + "up_proj.weight"]).t())) @ _wide(sd[q + "down_proj.weight"]).t()
    return out + torch.sigmoid(h @ _wide(sd[p + "shared_expert_gate.weight"]).t()) * s


def _exact_hybrid(case, seed):
    c = _config(case)
    sd, segs, tables, toks = _weights(case, seed, c), _segments(case), _tables(case, seed), _tokens(case, seed, c)
    keys, values, states, ring = (t.double() for t in _hybrid_caches(case, seed, c))
    ends = torch.tensor([n for n, _ in segs]).cumsum(0).tolist()
    parts = [slice(e - n, e) for e, (n, _) in zip(ends, segs)]
    for i, (n, before) in enumerate(segs):
        if case["kind"] != "decode" and not before:
            states[:, i] = 0
            ring[:, i] = 0
    x = sd[LM + "embed_tokens.weight"][torch.cat(toks).to(DEV)].double()
    nk, nv, dk, dv, nh, ng, hd = (c.linear_num_key_heads, c.linear_num_value_heads, c.linear_key_head_dim, c.linear_value_head_dim,
                                  c.num_attention_heads, c.num_key_value_heads, c.head_dim)
    norm = lambda x, key: _rms(x, c.rms_norm_eps) * (1 + _wide(sd[key]))
    jl = jf = 0
    for li, kind in enumerate(c.layer_types):
        p = f"{LM}layers.{li}."
        h = norm(x, p + "input_layernorm.weight")
        outs = []
        if kind == LINEAR:
            p += "linear_attn."
            qkv, z, b, a = (h @ _wide(sd[p + f"in_proj_{s}.weight"]).t() for s in ("qkv", "z", "b", "a"))
            taps = _wide(sd[p + "conv1d.weight"]).view(c.lin_conv_dim, -1)
            beta, g = torch.sigmoid(b), -torch.exp(_wide(sd[p + "A_log"])) * F.softplus(a + _wide(sd[p + "dt_bias"]))
            for i, (s, (n, before)) in enumerate(zip(parts, segs)):
                y = _conv(qkv[s], taps, _before(ring[jl, i], before, taps.shape[1]))
                q, k, v = torch.split(y, [nk * dk, nk * dk, nv * dv], 1)
                q, k = (t.view(n, nk, dk).repeat_interleave(nv // nk, 1) for t in (q, k))
                q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
                outs.append(_delta_scan(q * dk ** -0.5, k, v.reshape(n, nv, dv), beta[s], g[s], states[jl, i]))
                last = torch.arange(max(0, n - 16), n, device=DEV)
                ring[jl, i, (before + last) % 16] = qkv[s][last]
            o = _rms(torch.cat(outs), c.rms_norm_eps) * _wide(sd[p + "norm.weight"]) * F.silu(z.view(-1, nv, dv))
            x = x + o.reshape(-1, nv * dv) @ _wide(sd[p + "out_proj.weight"]).t()
            jl += 1
        else:
            p += "self_attn."
            q, gate = (h @ _wide(sd[p + "q_proj.weight"]).t()).view(-1, nh, 2 * hd).split(hd, -1)
            k, v = ((h @ _wide(sd[p + s + "_proj.weight"]).t()).view(-1, ng, hd) for s in "kv")
            q, k = (norm(t, p + s + "_norm.weight") for t, s in ((q, "q"), (k, "k")))
            for s, (n, before), bt in zip(parts, segs, tables):
                at = _rows_of(bt, before + n)
                qr, kr = (_turned(t[s], before, c.rotary_dim, c.rope_theta, True) for t in (q, k))
                keys[jf, at[before:]], values[jf, at[before:]] = kr, v[s]
                outs.append(_attend(qr, keys[jf, at], values[jf, at], before, hd ** -0.5))
            x = x + (torch.cat(outs) * torch.sigmoid(gate)).reshape(-1, nh * hd) @ _wide(sd[p + "o_proj.weight"]).t()
            jf += 1
        p = f"{LM}layers.{li}."
        h = norm(x, p + "post_attention_layernorm.weight")
        p += "mlp."
        if c.is_moe:
            x = x + _experts(c, sd, p, h)
        else:
            u = F.silu(h @ _wide(sd[p + "gate_proj.weight"]).t()) * (h @ _wide(sd[p + "up_proj.weight"]).t())
            x = x + u @ _wide(sd[p + "down_proj.weight"]).t()
    last = norm(x[[e - 1 for e in ends]], LM + "norm.weight")
    logits = last @ _wide(sd[LM + "embed_tokens.weight" if c.tie_word_embeddings else "lm_head.weight"]).t()
    return {"logits": list(logits) if case["kind"] == "prefill" else logits, "keys": keys, "values": values, "states": states, "rows": ring}


def _ssd_scan(x, B, C, dt, decay, D, S):
    """x ``[T, H, e]``, B and C ``[T, G, N]``, dt and decay ``[T, H]``; S ``[H, N, e]`` is updated."""
    per, out = x.shape[1] // B.shape[1], torch.empty_like(x)
    for t in range(x.shape[0]):
        S.mul_(decay[t, :, None, None])
        S.baddbmm_(B[t].repeat_interleave(per, 0)[:, :, None], (dt[t, :, None] * x[t])[:, None])
        out[t] = torch.bmm(C[t].repeat_interleave(per, 0)[:, None], S)[:, 0] + D[:, None] * x[t]
    return out


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt(d.square().mean(-1, keepdim=True) + eps) * w


def _exact_suki(case, seed):
    c = _config(case)
    W = {k: t.double() for k, t in _weights(case, seed, c).items()}
    segs, tables, toks, eps = _segments(case), _tables(case, seed), _tokens(case, seed, c), c.rms_norm_eps
    ends = torch.tensor([n for n, _ in segs]).cumsum(0).tolist()
    parts = [slice(e - n, e) for e, (n, _) in zip(ends, segs)]
    caches = [tuple(t.double() for t in u) if isinstance(u, tuple) else u.double() if u is not None else None for u in _suki_caches(case, seed, c)]
    for i, (n, before) in enumerate(segs):
        if case["kind"] != "decode" and not before:
            for u in caches:
                if isinstance(u, tuple):
                    u[0][i] = 0
                    u[1][i] = 0
    x = W["embed"][torch.cat(toks).to(DEV)] * c.embedding_scale
    planes = [x]
    for li, spec in enumerate(c.layers):
        p, m, outs = f"l{li}.", spec.mixer, []
        h, q = _layer_norm(x, W[p + "norm1"], eps), p + "mix."
        if spec.kind == "mamba2":
            S, ring = caches[li]
            z, xbc, dt = torch.split(h @ W[q + "in"].t(), [m.inner, m.conv_width, m.heads], 1)
            dt = F.softplus(dt + W[q + "dt_bias"])
            decay, gn = torch.exp(-torch.exp(W[q + "A_log"]) * dt), m.groups * m.state
            cbx = lambda t: torch.cat([t[..., m.inner + gn:], t[..., m.inner:m.inner + gn], t[..., :m.inner]], -1)     # the ring's order
            xbx = lambda t: torch.cat([t[..., 2 * gn:], t[..., gn:2 * gn], t[..., :gn]], -1)
            for i, (s, (n, before)) in enumerate(zip(parts, segs)):
                y = _conv(xbc[s], W[q + "conv"], xbx(_before(ring[i], before, m.conv)), W[q + "conv.b"])
                u, B, C = torch.split(y, [m.inner, gn, gn], 1)
                outs.append(_ssd_scan(u.reshape(n, m.heads, m.vdim), B.reshape(n, m.groups, m.state), C.reshape(n, m.groups, m.state), dt[s], decay[s],
                                      W[q + "D"], S[i]))
                last = torch.arange(max(0, n - m.conv + 1), n, device=DEV)
                ring[i, (before + last) % 16] = cbx(xbc[s][last])
            y = torch.cat(outs).reshape(-1, m.inner) * F.silu(z)
            y = _rms(y.view(-1, m.norm_groups, m.inner // m.norm_groups), eps).reshape(-1, m.inner) * W[q + "norm"]
        else:
            H, n0, r, R = m.heads, m.dim, m.rot_dim, m.kv_rank
            pool = caches[li if m.kv_from is None else m.kv_from]
            t = (_rms(h @ W[q + "dq"].t(), eps) * W[q + "dq.norm"]) @ W[q + "uq"].t()
            t, gate = t.view(-1, H, n0 + r), torch.sigmoid(h @ W[q + "g"].t())
            uk, uv = W[q + "uk"].view(H, n0, R), W[q + "uv"].view(H, m.vdim, R)
            low = h @ W[q + "dkv"].t() if m.kv_from is None else None
            for s, (n, before), bt in zip(parts, segs, tables):
                at = _rows_of(bt, before + n)
                if low is not None:
                    new = low[s]
                    pool[at[before:]] = torch.cat([_rms(new[:, :R], eps) * W[q + "dkv.norm"],
                                                   _turned(new[:, None, R:], before, m.rot_dims, m.rot_base, False)[:, 0]], 1)
                qr = _turned(t[s][..., n0:], before, m.rot_dims, m.rot_base, False)
                qa = torch.cat([torch.einsum("thn,hnr->thr", t[s][..., :n0], uk), qr], -1)
                o = _attend(qa, pool[at][:, None], pool[at][:, None, :R], before, m.scale)
                outs.append(torch.einsum("thr,her->the", o, uv) * gate[s][..., None])
            y = torch.cat(outs).reshape(-1, H * m.vdim)
        x = x + y @ W[q + "o"].t()
        if spec.ff is not None:
            u = _layer_norm(x, W[p + "norm2"], eps) @ W[p + "mlp.up"].t()
            a, b = F.softplus(W[p + "mlp.act"]).tolist()
            u = torch.where(u > 0, a * u * u, (0.5 + b) * (torch.expm1(u.clamp(max=0)) - u)) + u / 2
            x = x + u @ W[p + "mlp.down"].t()
        planes.append(x)
        x = sum(w * t for w, t in zip(W[p + "dwa"], planes))
    logits = _layer_norm(x[[e - 1 for e in ends]], W["final.norm"], eps) @ W["embed"].t()
    kept = [{"S": u[0], "ring": u[1]} if isinstance(u, tuple) else u for u in caches]
    return {"logits": logits, "layers": kept}


def exact(case, seed):
    with torch.no_grad():
        return _exact_suki(case, seed) if case["model"].startswith("sukisun") else _exact_hybrid(case, seed)
