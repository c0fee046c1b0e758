"""The calls that a program serving one of the framework's models makes, as cases to measure.

A case is one forward pass on one GPU: a decode step (one token for each sequence at position `context`, through a CUDA graph that the
program captured once, or eagerly) or a prompt pass (`tokens` positions of each sequence from 0 on, eagerly; logits of all positions,
which is what the reference's forward returns, or of the last one).  Presets are the framework's own.  Weights are random and keep
the scale of their input, so that a deep model's values stay those of a trained one; caches hold random rows and states of the
scale that the layers write.  Position and token ids are copied in for every step, as a decode loop does.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("ladder-residual-inference_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import gpt_fast  # noqa: E402

_FAMILIES = {"ladder": gpt_fast.GPTLadder, "dense": gpt_fast.GPTDense, "parallel": gpt_fast.GPTParallel, "desync": gpt_fast.GPTDesync,
             "patevik": gpt_fast.GPTPatevik, "migosun": gpt_fast.GPTMigosun}
_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
_SPARE = 64  # positions that the caches have beyond the measured ones: a program goes on generating


def _case(name, family, preset, dtype, mode, batch, tokens, context=0, logits="last"):
    return {"name": name, "family": family, "preset": preset, "dtype": dtype, "mode": mode, "batch": batch, "tokens": tokens,
            "context": context, "logits": logits}


def listed():
    return [
        # one user of the smallest model, called as the reference's driver does without flags: launches and host time
        _case("step-110m-eager", "dense", "stories110M", "fp16", "eager", 1, 1, 200),
        # one user of the small ladder model: a chain of short kernels
        _case("step-1b", "ladder", "ladder-llama-1b", "bf16", "graph", 1, 1, 1023),
        # the headline: one user, 8B, a 1024-token prompt behind it
        _case("step-8b", "ladder", "llama-3-8b", "bf16", "graph", 1, 1, 1024),
        # a served batch of the same model
        _case("step-8b-16", "ladder", "llama-3-8b", "bf16", "graph", 16, 1, 1024),
        # a large odd-shaped batch in the type of the reference's driver; every head has its own keys, parallel blocks
        _case("step-3b-40", "parallel", "llama-3.2-3b", "fp16", "graph", 40, 1, 700),
        # a few short prompts of ragged length, logits of every position
        _case("prompt-1b-ragged", "desync", "ladder-llama-1b", "fp16", "eager", 3, 333, 0, "all"),
        # the prompt pass of one user as the reference computes it
        _case("prompt-8b", "ladder", "llama-3-8b", "bf16", "eager", 1, 2048, 0, "all"),
        # a batch of long prompts: the largest call
        _case("prompt-8b-long", "dense", "llama-3-8b", "bf16", "eager", 4, 4096),
        # a few users of the mixture-of-experts design
        _case("step-patevik", "patevik", "patevik-1b", "bf16", "graph", 4, 1, 1500),
        # a prompt through its recurrences, windows and experts
        _case("prompt-patevik", "patevik", "patevik-1b", "bf16", "eager", 1, 2048),
        # a served batch of the design with residual streams
        _case("step-migosun", "migosun", "migosun-8b", "bf16", "graph", 16, 1, 1024),
        # prompts of ragged length through its recurrences
        _case("prompt-migosun", "migosun", "migosun-1b", "bf16", "eager", 2, 1500),
    ]


# family, preset, longest sequence, most positions in the caches, most prompt tokens
_RANGE = [("dense", "stories110M", 2048, 65536, 8192), ("ladder", "ladder-llama-1b", 2048, 65536, 8192),
          ("desync", "ladder-llama-1b", 2048, 65536, 8192), ("parallel", "llama-3.2-3b", 2048, 32768, 8192),
          ("ladder", "llama-3-8b", 8192, 65536, 8192), ("dense", "llama-3-8b", 8192, 65536, 8192),
          ("patevik", "patevik-1b", 4096, 32768, 4096), ("migosun", "migosun-1b", 4096, 32768, 4096),
          ("migosun", "migosun-8b", 4096, 32768, 2048)]


def draw(rng):
    def spread(lo, hi):
        return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))

    family, preset, longest, positions, prompt = rng.choice(_RANGE)
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    kind = rng.choice(("graph", "graph", "eager", "prompt", "prompt"))
    if kind != "prompt":
        batch = spread(1, 64)
        context = spread(16, min(longest, positions // batch) - _SPARE - 1)
        c = _case("", family, preset, dtype, kind, batch, 1, context)
    else:
        batch = spread(1, 8)
        tokens = spread(8, min(longest - _SPARE, prompt // batch))
        c = _case("", family, preset, dtype, "eager", batch, tokens, 0, rng.choice(("all", "last")))
    del c["name"]
    return c


# ---- weights and caches ---------------------------------------------------------------------------------------------------------
def _fill(model, family, gen):
    """Random weights.  Matrices keep the scale of their input; those that write the residual are smaller by the square root of the
    number of sublayers, as initialisations of deep models have it."""
    cfg = model.config
    depth = (2 * cfg.n_layer) ** -0.5
    for name, p in model.named_parameters():
        leaf = name.rsplit(".", 2)
        leaf = leaf[-2] if leaf[-1] == "weight" else leaf[-1]
        if leaf in ("norm", "attention_norm", "ffn_norm", "pre_norm", "q_norm", "k_norm", "latent_norm"):
            p.normal_(1.0, 0.1, generator=gen)
        elif leaf == "post_norm":
            p.normal_(0.1, 0.02, generator=gen)
        elif leaf in ("gate_bias", "f_bias", "a2_bias", "sink"):
            p.normal_(0.0, 0.5, generator=gen)
        elif leaf == "lower":
            p.copy_(torch.linspace(0.0, 0.99, p.numel(), device=p.device))
        elif leaf == "a_log":
            p.copy_(torch.linspace(-4.0, 0.0, p.numel(), device=p.device))
        elif leaf == "dt_bias":
            p.copy_(torch.linspace(-3.0, 1.0, p.numel(), device=p.device))
        elif leaf == "w_in":
            p.normal_(1.0 / p.numel(), 0.1 / p.numel(), generator=gen)
        elif leaf == "w_out":
            p.normal_(1.0, 0.1, generator=gen)
        elif leaf == "w_mix":
            p.normal_(0.0, 0.02, generator=gen)
            p.add_(torch.eye(p.shape[0], device=p.device, dtype=p.dtype))
        elif leaf.startswith("conv_"):
            p.normal_(0.0, 0.5, generator=gen)
        elif leaf == "tok_embeddings":
            p.normal_(0.0, cfg.dim ** -0.5 if family == "migosun" else 1.0, generator=gen)
        elif leaf in ("wo", "w2"):
            # a tied table has rows of length one: what joins its residual has their scale
            p.normal_(0.0, depth * p.shape[-1] ** -0.5 * (cfg.dim ** -0.5 if family == "migosun" else 1.0), generator=gen)
        else:
            p.normal_(0.0, p.shape[-1] ** -0.5, generator=gen)
    if family in ("patevik", "migosun"):
        for block in model.layers:
            for br in (block.mixer, block.mlp):
                if br is not None and br.in_proj is not None:
                    br.in_proj.weight[br.gate_rows + br.sublayer.in_rows:].zero_()
    if family == "patevik":
        _decided_routers(model, gen)


def _decided_routers(model, gen):
    """A trained router is decided about nearly every token; one of random numbers has ties that two right implementations settle
    differently.  Every token's embedding leans on the directions of two experts, and the routers' rows on one each."""
    d, n = model.config.dim, model.layers[0].mlp.sublayer.experts
    w = model.tok_embeddings.weight
    lean = (torch.randint(0, 2, (n, d), device=w.device, generator=gen) * 2 - 1).to(torch.float32)
    for at in range(0, w.shape[0], 16384):
        rows = w[at:at + 16384]
        pair = torch.rand(rows.shape[0], n, device=w.device, generator=gen).topk(2, dim=1).indices
        rows.copy_(0.7 * rows.float() + 0.5 * lean[pair].sum(1))
    for block in model.layers:
        rows = block.mlp.in_proj.weight[d:d + n]
        rows.copy_(0.2 * rows.float() + 6.0 / d * lean)


def _subs(block):
    m = block.mixer.sublayer
    return (m.left, m.right) if m.kind == "parallel" else (m,)


def _fill_caches(model, family, context, gen):
    """Cache rows of earlier positions and recurrent states as earlier steps leave them."""
    def rows(t, dim, scale=1.0):
        t.narrow(dim, 0, context).normal_(0.0, scale, generator=gen)

    for block in model.layers:
        if family not in ("patevik", "migosun"):
            rows(block.attention.kv_cache.k_cache, 2)
            rows(block.attention.kv_cache.v_cache, 2)
            continue
        for m in _subs(block):
            if m.kind == "latent_attention":
                rows(m.kv_cache.rows, 1)
            elif m.kind == "chunked_attention":
                rows(m.kv_cache.k_cache, 2)
                rows(m.kv_cache.v_cache, 2)
            else:
                m.kv_cache.state.normal_(0.0, 0.3, generator=gen)
                if m.kind == "gated_delta":
                    m.conv_state.ring.normal_(0.0, 1.0, generator=gen)


class _State:
    pass


def _model(case, seed):
    family = case["family"]
    gen = torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))
    with torch.device("meta"):
        model = _FAMILIES[family].from_name(case["preset"])
    model = model.to(dtype=_DTYPES[case["dtype"]]).to_empty(device="cuda").eval()
    with torch.no_grad():
        _fill(model, family, gen)
    first = case["context"]
    with torch.device("cuda"):
        model.setup_caches(max_batch_size=case["batch"], max_seq_length=first + case["tokens"] + _SPARE)
    with torch.no_grad():
        if first:
            _fill_caches(model, family, first, gen)
    ids = torch.randint(0, model.config.vocab_size, (case["batch"], case["tokens"]), device="cuda", generator=gen)
    return model, ids


def prepare(case, seed):
    s = _State()
    s.case = case
    s.model, s.ids = _model(case, seed)
    first, n = case["context"], case["tokens"]
    if n > 1:
        s.pos = torch.arange(n, device="cuda")
        return s
    s.ids = s.ids.to(torch.int32)
    s.pos = torch.tensor([first], dtype=torch.int32, device="cuda")
    if case["mode"] == "graph":
        s.tok, s.at = s.ids.clone(), s.pos.clone()
        kept = [t.clone() for t in s.model.recurrent_state()]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side), torch.no_grad():
            s.model(s.tok, s.at)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        for t, t0 in zip(s.model.recurrent_state(), kept):
            t.copy_(t0)
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph), torch.no_grad():
            s.logits = s.model(s.tok, s.at)
    return s


def _some(n):
    """Layers whose caches are returned: all of them meet in the logits."""
    return sorted({0, n // 2, n - 1})


def _kept(model, family, first, n):
    """What a pass leaves in the caches of some layers: the rows that it writes, and whole states."""
    out = []
    for i in _some(len(model.layers)):
        block = model.layers[i]
        if family not in ("patevik", "migosun"):
            c = block.attention.kv_cache
            out += [c.k_cache[:, :, first:first + n], c.v_cache[:, :, first:first + n]]
            continue
        for m in _subs(block):
            if m.kind == "latent_attention":
                out.append(m.kv_cache.rows[:, first:first + n])
            elif m.kind == "chunked_attention":
                out += [m.kv_cache.k_cache[:, :, first:first + n], m.kv_cache.v_cache[:, :, first:first + n]]
            else:
                out.append(m.kv_cache.state)
                if m.kind == "gated_delta":
                    out.append(m.conv_state.ring)
    return out


def run(state):
    s, case = state, state.case
    if case["mode"] == "graph":
        s.tok.copy_(s.ids)
        s.at.copy_(s.pos)
        s.graph.replay()
        logits = s.logits
    elif case["tokens"] == 1 or case["logits"] == "all":
        logits = s.model(s.ids, s.pos)
    else:
        logits = s.model.prefill_last(s.ids, s.pos)
    return {"logits": logits, "kept": _kept(s.model, case["family"], case["context"], case["tokens"])}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------
def _pairs(n, first, window=0, chunk=0):
    """(query, key) pairs of n queries from position `first` on, and how many keys are read at all."""
    pairs, lowest = 0, first + n
    for p in range(first, first + n):
        lo = max(0, p - window + 1 if window else 0, p // chunk * chunk if chunk else 0)
        pairs += p - lo + 1
        lowest = min(lowest, lo)
    return pairs, first + n - lowest


def work(case):
    with torch.device("meta"):
        model = _FAMILIES[case["family"]].from_name(case["preset"])
    cfg, family, B, n, first = model.config, case["family"], case["batch"], case["tokens"], case["context"]
    rows = B * n
    out_rows = rows if n == 1 or case["logits"] == "all" else B
    nbytes = rows * (cfg.dim * 2 + 8) + cfg.vocab_size * cfg.dim * 2 + out_rows * cfg.vocab_size * 2
    flops = 2 * out_rows * cfg.vocab_size * cfg.dim
    for name, p in model.named_parameters():
        if name.startswith(("tok_embeddings", "output")):
            continue
        if p.dim() == 3:  # experts: those that some token chooses, and the products of the chosen ones
            e, top = p.shape[0], model.layers[0].mlp.sublayer.top
            nbytes += 2 * p.numel() * (1 - (1 - top / e) ** rows)
            flops += 2 * rows * top * p.numel() // e
        else:
            nbytes += 2 * p.numel()
            flops += 2 * rows * p.numel() if p.dim() == 2 else 0
    for block in model.layers:
        if family not in ("patevik", "migosun"):
            pairs, keys = _pairs(n, first)
            nbytes += 4 * B * cfg.n_local_heads * cfg.head_dim * keys
            flops += 4 * B * cfg.n_head * cfg.head_dim * pairs
            continue
        for m in _subs(block):
            if m.kind == "latent_attention":
                pairs, keys = _pairs(n, first, window=m.window)
                nbytes += 2 * B * (m.rank + m.rot_dim) * keys
                flops += 2 * B * m.heads * (m.dim + m.rot_dim + m.vdim) * pairs
            elif m.kind == "chunked_attention":
                pairs, keys = _pairs(n, first, chunk=m.chunk)
                nbytes += 2 * B * m.kv_heads * (m.dim + m.vdim) * keys
                flops += 2 * B * m.heads * (m.dim + m.vdim) * pairs
            else:
                nbytes += 4 * B * m.heads * m.dim * m.vdim * (2 if first else 1)
                flops += (8 if m.kind == "gated_delta" else 6) * rows * m.heads * m.dim * m.vdim
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    # About four times what one pass is off from 64 bits: bf16 keeps 8 bits and fp16 11, a Llama schedule rounds its residual at every
    # addition (0.014 and 0.0018 measured), the other designs keep it in 32 bits (0.003 and 0.0006).
    wide = case["family"] in ("patevik", "migosun")
    rel = (0.012 if wide else 0.03) if case["dtype"] == "bf16" else (0.0024 if wide else 0.007)
    return {"rel": rel, "max": 13 * rel}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _mm(x, w):
    return x @ w.double().T


def _softmax_over(q, k, v, scale, first, window=0, chunk=0, sink=None):
    """q [n, H, d] at positions from `first` on, k [keys, G, d], v [keys, G, e] from position 0 on -> [n, H * e]"""
    n, H = q.shape[:2]
    each = H // k.shape[1]
    pos, at = torch.arange(first, first + n, device=q.device)[:, None], torch.arange(k.shape[0], device=q.device)[None]
    hidden = at > pos
    if window:
        hidden |= at <= pos - window
    if chunk:
        hidden |= at // chunk != pos // chunk
    out = torch.empty(n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for g in range(k.shape[1]):
        heads = slice(g * each, (g + 1) * each)
        score = (q[:, heads].transpose(0, 1) @ k[:, g].T * scale).masked_fill_(hidden, float("-inf"))
        if sink is not None:
            score = torch.cat([score, sink[heads].double()[:, None, None].expand(each, n, 1)], dim=-1)
        score = torch.softmax(score, dim=-1)[..., : k.shape[0]]
        out[:, heads] = (score @ v[:, g]).transpose(0, 1)
    return out.reshape(n, -1)


def _with_history(cache, new, first):
    """Rows of the cache [G, positions, d] before `first`, then the new ones [n, G, d] -> [first + n, G, d]"""
    return torch.cat([cache[:, :first].transpose(0, 1).double(), new])


def _llama_attention(att, w, cfg, h, B, n, first, kept):
    nh, nkv, hd = cfg.n_head, cfg.n_local_heads, cfg.head_dim
    q, k, v = _mm(h, w).view(B, n, nh + 2 * nkv, hd).split((nh, nkv, nkv), dim=2)
    # the table of angles is part of the model: evaluated in 32 bits and rounded to its type, as the reference does
    freqs = 1.0 / (cfg.rope_base ** (torch.arange(0, hd, 2).float() / hd))
    ang = torch.outer(torch.arange(first, first + n), freqs)
    cos, sin = (f(ang).to(w.dtype).to(h.device).double()[None, :, None] for f in (torch.cos, torch.sin))

    def turned(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cos - b * sin, b * cos + a * sin], dim=-1).flatten(-2)

    q, k = turned(q), turned(k)
    if kept is not None:
        kept += [k.transpose(1, 2), v.transpose(1, 2)]
    c = att.kv_cache
    return torch.cat([_softmax_over(q[b], _with_history(c.k_cache[b], k[b], first), _with_history(c.v_cache[b], v[b], first),
                                    hd ** -0.5, first) for b in range(B)])


def _llama(model, family, ids, first, kept):
    cfg, (B, n) = model.config, ids.shape
    r = model.tok_embeddings.weight[ids.view(-1)].double()
    A = M = torch.zeros_like(r)
    keep = _some(len(model.layers))

    def mlp(h, w1, w2):
        u, g = _mm(h, w1).chunk(2, dim=-1)
        return _mm(torch.nn.functional.silu(g) * u, w2.weight)

    for i, la in enumerate(model.layers):
        at, out = la.attention, kept if i in keep else None
        if family == "parallel":
            h = _rms(r, la.attention_norm.weight, cfg.norm_eps)
            w, nq = at.wqkv1.weight, (cfg.n_head + 2 * cfg.n_local_heads) * cfg.head_dim
            r = r + _mm(_llama_attention(at, w[:nq], cfg, h, B, n, first, out), at.wo.weight) + mlp(h, w[nq:], at.w2)
            continue
        ff = la.feed_forward
        # a ladder block adds a sublayer's result one sublayer later
        r = r + A
        a = _mm(_llama_attention(at, at.wqkv.weight, cfg, _rms(r, la.attention_norm.weight, cfg.norm_eps), B, n, first, out), at.wo.weight)
        r = r + M if family == "ladder" else r + a
        m = mlp(_rms(r, la.ffn_norm.weight, cfg.norm_eps), ff.w1.weight, ff.w2)
        if family == "ladder":
            A, M = a, m
        else:
            r = r + m
    return _rms(r + A + M, model.norm.weight, cfg.norm_eps)


def _halves(x, first, dims, base):
    """Rotates the pairs (i, i + dims / 2) of the first `dims` elements; x [B, n, heads, d]."""
    half = dims // 2
    i = torch.arange(half, dtype=torch.float64, device=x.device)
    ang = torch.outer(torch.arange(first, first + x.shape[1], dtype=torch.float64, device=x.device), base ** (-2.0 * i / dims))[None, :, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin(), x[..., dims:]], dim=-1)


def _glu(x, w1, w2, glu):
    u, g = _mm(x, w1).chunk(2, dim=-1)
    g = g.clamp(max=glu[1])
    return _mm(g * torch.sigmoid(glu[0] * g) * (u.clamp(-glu[1], glu[1]) + glu[2]), w2)


def _moe(m, h, logits):
    score, ids = torch.sigmoid(logits).topk(m.top, dim=-1)
    out = torch.zeros_like(h)
    for e in range(m.experts):
        row, slot = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            out.index_add_(0, row, _glu(score[row, slot, None] * h[row], m.w1[e], m.w2[e], m.glu))
    return out


def _states(first, state):
    return state.double() if first else torch.zeros_like(state, dtype=torch.float64)


def _recur(q, k, v, g, state, beta=None):
    """state <- g state + k u^T with u = v, or the delta rule's beta (v - state^T k) on the decayed state; o = state^T q.
    q, k, g [B, n, H, C], v [B, n, H, E], beta [B, n, H], state [B, H, C, E]"""
    out = torch.empty_like(v)
    for t in range(q.shape[1]):
        state = g[:, t, :, :, None] * state
        u = v[:, t, :, None]
        if beta is not None:
            u = beta[:, t, :, None, None] * (u - k[:, t, :, None] @ state)
        state = state + k[:, t, :, :, None] * u
        out[:, t] = (q[:, t, :, None] @ state)[:, :, 0]
    return out, state


def _latent(m, p, B, n, first, eps, kept):
    H, dn, dr, r, c = m.heads, m.dim, m.rot_dim, m.rank, m.kv_cache.rows
    q = p[:, : m.q_rows].view(B, n, H, dn + dr)
    q = torch.cat([q[..., :dn], _halves(q[..., dn:], first, dr, m.rot_base)], dim=-1)
    lat = _rms(p[:, m.q_rows: m.q_rows + r], m.latent_norm, eps).view(B, n, r)
    rot = _halves(p[:, m.q_rows + r:].reshape(B, n, 1, dr), first, dr, m.rot_base)[:, :, 0]
    rows = torch.cat([lat, rot], dim=-1)
    if kept is not None:
        kept.append(rows)
    out = []
    for b in range(B):
        seen = torch.cat([c[b, :first].double(), rows[b]])
        kv = _mm(seen[:, :r], m.expand.weight)
        k = torch.cat([kv[:, : H * dn].view(-1, H, dn), seen[:, None, r:].expand(-1, H, dr)], dim=-1)
        out.append(_softmax_over(q[b], k, kv[:, H * dn:].view(-1, H, m.vdim), m.scale, first, window=m.window))
    return torch.cat(out)


def _hgrn2(m, p, B, n, first, eps, kept):
    H, C, E = m.heads, m.dim, m.vdim
    q, f, v = p.split((H * C, H * C, H * E), dim=-1)
    low = m.lower.double()
    f = (low + (1 - low) * torch.sigmoid(f + m.f_bias.double())).view(B, n, H, C)
    o, state = _recur(torch.nn.functional.silu(q).view(B, n, H, C), 1 - f, v.view(B, n, H, E), f, _states(first, m.kv_cache.state))
    if kept is not None:
        kept.append(state)
    return _rms(o, m.norm, eps).reshape(B * n, -1)


def _patevik(model, ids, first, kept):
    cfg, (B, n) = model.config, ids.shape
    d, eps, keep = cfg.dim, cfg.norm_eps, _some(len(model.layers))
    x = model.tok_embeddings.weight[ids.view(-1)].double()
    for i, block in enumerate(model.layers):
        for br in (block.mixer, block.mlp):
            h, m = _rms(x, br.pre_norm, eps), br.sublayer
            p = _mm(h, br.in_proj.weight[: d + m.in_rows])
            if m.kind == "moe":
                y = _moe(m, h, p[:, d:])
            else:
                run_ = _latent if m.kind == "latent_attention" else _hgrn2
                y = _mm(run_(m, p[:, d:], B, n, first, eps, kept if i in keep else None), m.wo.weight)
            x = x + _rms(torch.sigmoid(p[:, :d] + br.gate_bias.double()) * y, br.post_norm, eps)
    return _rms(x, model.norm.weight, eps)


def _grouped(m, q, k, v, B, n, first, eps, kept):
    q = _halves(_rms(q, m.q_norm, eps).view(B, n, m.heads, m.dim), first, m.rot_dims, m.rot_base)
    k = _halves(_rms(k, m.k_norm, eps).view(B, n, m.kv_heads, m.dim), first, m.rot_dims, m.rot_base)
    v = v.reshape(B, n, m.kv_heads, m.vdim)
    if kept is not None:
        kept += [k.transpose(1, 2), v.transpose(1, 2)]
    c = m.kv_cache
    return torch.cat([_softmax_over(q[b], _with_history(c.k_cache[b], k[b], first), _with_history(c.v_cache[b], v[b], first), m.scale,
                                    first, chunk=m.chunk, sink=m.sink) for b in range(B)])


def _delta(m, q, k, v, a1, g1, beta, B, n, first, eps, kept):
    H, C, E, T = m.heads, m.dim, m.vdim, m.taps
    x = torch.cat([q, k, v], dim=-1).view(B, n, -1)
    ring = m.conv_state.ring.double()
    past = torch.zeros(B, T - 1, x.shape[-1], dtype=x.dtype, device=x.device)
    for j in range(1, T):
        if first - j >= 0:
            past[:, T - 1 - j] = ring[:, (first - j) % T]
    whole = torch.cat([past, x], dim=1)
    taps = torch.cat([m.conv_q, m.conv_k, m.conv_v]).double()
    y = torch.nn.functional.silu(sum(taps[:, j] * whole[:, j:j + n] for j in range(T)))
    if kept is not None:
        ring = ring.clone()
        for s in range(max(0, n - T), n):
            ring[:, (first + s) % T] = x[:, s]
    qk = m.kv_heads * C

    def unit(t):
        t = t.reshape(B, n, m.kv_heads, C)
        return (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // m.kv_heads, dim=2)

    z = _mm(a1, m.a2) + m.dt_bias.double()
    g = torch.exp(-torch.exp(m.a_log.double())[:, None] * torch.nn.functional.softplus(z).view(B, n, H, C))
    o, state = _recur(unit(y[..., :qk]) * C ** -0.5, unit(y[..., qk:2 * qk]), y[..., 2 * qk:].reshape(B, n, H, E), g,
                      _states(first, m.kv_cache.state), torch.sigmoid(beta).view(B, n, H))
    if kept is not None:
        kept += [state, ring]
    return _rms(o, m.norm, eps).reshape(B * n, -1) * torch.sigmoid(_mm(g1, m.g2))


def _gla(m, q, k, v, gate, a1, B, n, first, eps, kept):
    H, C, E = m.heads, m.dim, m.vdim
    g = torch.exp(torch.nn.functional.logsigmoid(_mm(a1, m.a2) + m.a2_bias.double()) / m.tau).view(B, n, H, C)
    o, state = _recur((q * C ** -0.5).view(B, n, H, C), k.reshape(B, n, H, C), v.reshape(B, n, H, E), g, _states(first, m.kv_cache.state))
    if kept is not None:
        kept.append(state)
    return _rms(o, m.norm, eps).reshape(B * n, -1) * torch.nn.functional.silu(gate)


def _migosun(model, ids, first, kept):
    cfg, (B, n) = model.config, ids.shape
    eps, keep = cfg.norm_eps, _some(len(model.layers))
    x = (model.tok_embeddings.weight[ids.view(-1)].double() * cfg.embed_scale)[None].repeat(cfg.streams, 1, 1)
    for i, block in enumerate(model.layers):
        out = kept if i in keep else None
        for br in (block.mixer, block.mlp):
            if br is None:
                continue
            h, m = _rms(torch.einsum("s,snd->nd", br.w_in.double(), x), br.pre_norm, eps), br.sublayer
            if m.kind == "glu":
                y = _glu(h, m.w1, m.w2, m.glu)
            else:
                p = _mm(h, br.in_proj.weight[: m.in_rows]).split([r.padded for r in m.parts()], dim=-1)
                if m.kind == "parallel":
                    y = torch.cat([m.scales[0] * _grouped(m.left, *p[:3], B, n, first, eps, out),
                                   m.scales[1] * _delta(m.right, *p[3:], B, n, first, eps, out)], dim=-1)
                else:
                    y = _gla(m, *p, B, n, first, eps, out)
                y = _mm(y, m.wo.weight)
            x = torch.einsum("st,snd->tnd", br.w_mix.double(), x) + br.w_out.double()[:, None, None] * y
    return _rms(x.sum(0), model.norm.weight, eps)


@torch.no_grad()
def exact(case, seed):
    model, ids = _model(case, seed)
    family, (B, n), first, kept = case["family"], ids.shape, case["context"], []
    if family == "patevik":
        h = _patevik(model, ids, first, kept)
    elif family == "migosun":
        h = _migosun(model, ids, first, kept)
    else:
        h = _llama(model, family, ids, first, kept)
    h = h.view(B, n, -1)
    if n > 1 and case["logits"] == "last":
        h = h[:, -1:]
    w = model.output.weight
    logits = torch.empty(*h.shape[:2], w.shape[0], dtype=torch.float64, device=h.device)
    for at in range(0, w.shape[0], 16384):
        logits[..., at:at + 16384] = _mm(h, w[at:at + 16384])
    return {"logits": logits, "kept": kept}
