"""Inputs and 64-bit results for the tests of kernels whose CTAs share tiles between rows (attention of prompt rows, recurrences)."""
import types

import torch

DEV = "cuda:0"
UNIT = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}
TYPES = [torch.bfloat16, torch.float16]


def rel(got, ref):
    got, ref = got.double(), ref.double()
    assert bool(torch.isfinite(got).all())
    return float((got - ref).norm() / ref.norm())


def ints(v):
    return torch.tensor(list(v), dtype=torch.int32, device=DEV)


def normal(*shape, seed, dtype=torch.float32):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV).to(dtype)


def table(totals, bs, seed):
    per = [-(-n // bs) for n in totals]
    ids = torch.randperm(sum(per), generator=torch.Generator().manual_seed(seed)).tolist()
    bt = torch.zeros(len(totals), max(per), dtype=torch.int32)
    at = 0
    for s, n in enumerate(per):
        bt[s, :n] = torch.tensor(ids[at:at + n])
        at += n
    return bt.to(DEV), sum(per)


def token_state(portions, decodes):
    """portions: (tokens, position of the first); decodes: positions of single decoded tokens."""
    rows = portions + [(1, p) for p in decodes]
    return rows, types.SimpleNamespace(
        token_seq_ids=ints(i for i, (n, _) in enumerate(rows) for _ in range(n)),
        token_positions=ints(p + j for n, p in rows for j in range(n)), num_prefill_tokens=sum(n for n, _ in portions), num_prefill_seqs=len(portions))


def angles(positions, dims):
    f = torch.tensor([50.0 ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=DEV)
    a = positions.double()[:, None] * f
    return a.cos().float().contiguous(), a.sin().float().contiguous()


def segments(lens, firsts, decoded=False):
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    return types.SimpleNamespace(
        batch_size=len(lens), num_prefill_seqs=0 if decoded else len(lens), num_prefill_tokens=0 if decoded else sum(lens),
        seq_ids=ints(range(len(lens))), seg_starts=ints(starts), token_seq_ids=ints(i for i, n in enumerate(lens) for _ in range(n)),
        token_positions=ints(f + j for n, f in zip(lens, firsts) for j in range(n)))


def turn(x, cos, sin, dims, halves=False):
    """The first `dims` entries of [..., d] turned, pairs as neighbours or as halves; cos, sin broadcast over [..., dims / 2]."""
    y = x.clone()
    if halves:
        a, b = x[..., :dims // 2], x[..., dims // 2:dims]
        y[..., :dims // 2], y[..., dims // 2:dims] = a * cos - b * sin, b * cos + a * sin
    else:
        a, b = x[..., 0:dims:2], x[..., 1:dims:2]
        y[..., 0:dims:2], y[..., 1:dims:2] = a * cos - b * sin, b * cos + a * sin
    return y


# ---------------------------------------------------------------- latent attention
def latent_case(dtype, portions, decodes, H, r, dr, dims, window, sink, bs=16, gated=True):
    rows, st = token_state(portions, decodes)
    T = st.token_positions.shape[0]
    bt, nb = table([n + p for n, p in rows], bs, T + r)
    cos, sin = angles(st.token_positions, dims) if dims else (None, None)
    return types.SimpleNamespace(
        rows=rows, st=st, bt=bt, bs=bs, cache=normal(nb, 2, bs, r + dr, seed=r, dtype=dtype), q=normal(T, H, r, seed=T, dtype=dtype),
        qr=normal(T, H, 3 + dr, seed=T + 1, dtype=dtype)[:, :, 3:], gate=normal(T, H, seed=T + 2, dtype=dtype) if gated else None, cos=cos, sin=sin,
        dims=dims, window=window, scale=(r + dr) ** -0.5, sink=normal(H, seed=9) if sink else None)


def latent_run(c, cache=None):
    from swiftllm_b200.worker.kernels.latent_attn import latent_attention
    out = torch.empty_like(c.q)
    latent_attention(c.q, c.qr, c.gate, c.cache if cache is None else cache, 1, c.bt, c.st, out, c.dims, c.window, c.scale, c.cos, c.sin, c.sink)
    return out


def cache_rows(c, slot, s):
    """The cache rows of sequence s of a case, in order."""
    n, p = c.rows[s]
    bs = c.cache.shape[2]
    return c.cache[c.bt[s, :-(-(n + p) // bs)].long(), slot].flatten(0, 1)[:n + p]


def attend(score, seen, value, sink):
    """score [n, H, L], seen [n, L] or [n, H, L], value [L, H, e]; sink [H]: score of a key without a value, or None."""
    score = score.masked_fill(~(seen if seen.dim() == 3 else seen[:, None]), float("-inf"))
    if sink is not None:
        score = torch.cat((score, sink[None, :, None].expand(score.shape[0], -1, 1)), 2)
    return torch.einsum("nhl,lhe->nhe", torch.softmax(score, 2)[:, :, :value.shape[0]], value)


def latent_exact(c):
    out, at, r = [], 0, c.q.shape[2]
    for s, (n, p) in enumerate(c.rows):
        t = slice(at, at + n)
        at += n
        k = cache_rows(c, 1, s).double()
        qr = c.qr[t].double()
        if c.dims:
            qr = turn(qr, c.cos[t, None].double(), c.sin[t, None].double(), c.dims)
        score = torch.einsum("nhd,ld->nhl", torch.cat((c.q[t].double(), qr), 2), k) * c.scale
        qp, kp = p + torch.arange(n, device=DEV)[:, None], torch.arange(n + p, device=DEV)[None]
        seen = (kp <= qp) & ((qp - kp < c.window) if c.window > 0 else True)
        y = attend(score, seen, k[:, None, :r].expand(-1, score.shape[1], -1), None if c.sink is None else c.sink.double())
        out.append(y if c.gate is None else y * torch.sigmoid(c.gate[t].double())[:, :, None])
    return torch.cat(out)


# ---------------------------------------------------------------- window attention
def window_case(dtype, portions, decodes, H, G, dk, dv, rot, window, opts):
    from swiftllm_b200.worker.kernels.window_attn import AttnOptions, shared_row_width
    rows, st = token_state(portions, decodes)
    T, opts = st.token_positions.shape[0], dict(opts)
    bt, nb = table([n + p for n, p in rows], 16, T + dk)
    shared, prenorm, turned = opts.pop("shared", False), opts.pop("prenorm", False), opts.pop("turned_values", False)
    gated, sink = opts.pop("gate", True), opts.pop("sink", not shared)
    kt = opts.get("key_turned", 0)
    if shared:
        cache = normal(nb, 1, 16, shared_row_width(G, dk, kt), seed=dk, dtype=dtype)
        inv = normal(nb, 1, 16, G, seed=dk + 1).abs() * 0.2 + 0.9
        cache[..., :2 * G] = inv.contiguous().view(dtype).view(nb, 1, 16, 2 * G)
        opts["shared_kv"] = True
    else:
        cache = normal(nb, 1, 16, G * dk + G // opts.get("vshare", 1) * dv, seed=dk, dtype=dtype)
    if prenorm:
        opts.update(q_norm=1 + 0.1 * normal(dk, seed=4), prenorm_eps=1e-5)
    for name in ("slopes", "sinks"):
        if opts.pop(name, False):
            opts[name] = normal(H, seed=5).abs() * 0.1
    opt = AttnOptions(**opts)
    proj = normal(T, H * dk + H * dv, seed=T, dtype=dtype)
    gate = proj[:, H * dk:H * dk + (H if opt.gate_per_head else H * dv)] if gated else None
    cos, sin = angles(st.token_positions, rot) if rot else (None, None)
    vcos, vsin = angles(st.token_positions, dv) if turned else (None, None)
    return types.SimpleNamespace(rows=rows, st=st, bt=bt, cache=cache, q=proj[:, :H * dk], gate=gate, H=H, G=G, dk=dk, dv=dv, rot=rot,
                                 window=window, sink=sink, opt=opt, cos=cos, sin=sin, vcos=vcos, vsin=vsin)


def window_run(c, cache=None, st=None):
    from swiftllm_b200.worker.kernels.window_attn import window_attention
    out = torch.empty(c.q.shape[0], c.H * c.dv, dtype=torch.float32 if c.opt.out_f32 else c.q.dtype, device=DEV)
    window_attention(c.q, c.gate, c.cache if cache is None else cache, 0, c.bt, st or c.st, out, c.H, c.G, c.dk, c.dv, c.rot, c.window,
                     c.dk ** -0.5, c.sink, c.cos, c.sin, c.opt, c.vcos, c.vsin)
    return out


def window_columns(c):
    """(first key column, entries of a key head, first value column, value heads) of a cache row."""
    if c.opt.shared_kv:
        first = (2 * c.G + 7) // 8 * 8
        return first, c.dk + c.opt.key_turned, first, c.G
    return 0, c.dk, c.G * c.dk, c.G // c.opt.vshare


def window_exact(c):
    o, H, G, dk, dv = c.opt, c.H, c.G, c.dk, c.dv
    k0, kw, v0, gv = window_columns(c)
    out, at = [], 0
    for s, (n, p) in enumerate(c.rows):
        t = slice(at, at + n)
        at += n
        row = cache_rows(c, 0, s)
        L = n + p
        q = c.q[t].double().unflatten(1, (H, dk))
        if o.q_norm is not None:
            q = q / (q.square().mean(2, keepdim=True) + o.prenorm_eps).sqrt() * o.q_norm.double()
        if c.rot:
            q = turn(q, c.cos[t, None].double(), c.sin[t, None].double(), c.rot, o.pair_halves)
        if o.qk_norm_eps >= 0:
            q = q / (q.square().mean(2, keepdim=True) + o.qk_norm_eps).sqrt()
        heads = row[:, k0:k0 + G * kw].double().unflatten(1, (G, kw))
        k = heads[:, :, o.key_turned:o.key_turned + dk]
        if o.shared_kv:
            k = k * row[:, :2 * G].contiguous().view(torch.float32).double()[:, :, None]
            v = heads[:, :, :dv]
        else:
            v = row[:, v0:].double().unflatten(1, (gv, dv)).repeat_interleave(o.vshare, 1)
        k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
        score = torch.einsum("nhd,lhd->nhl", q, k) * dk ** -0.5
        if o.softcap > 0:
            score = o.softcap * torch.tanh(score / o.softcap)
        qp, kp = p + torch.arange(n, device=DEV)[:, None], torch.arange(L, device=DEV)[None]
        if o.slopes is not None:
            score = score - o.slopes.double()[None, :, None] * (qp - kp)[:, None].double()
        seen = kp <= qp
        if c.window > 0:
            seen = seen & ((qp - kp < c.window) | (kp < o.keep_first))
        if o.chunk > 0:
            seen = seen & (kp >= qp // o.chunk * o.chunk)
        sink = o.sinks.double() if o.sinks is not None else torch.zeros(H, dtype=torch.float64, device=DEV) if c.sink else None
        y = attend(score, seen, v, sink) * o.out_scale
        if c.vcos is not None:                               # values were stored turned by their position: turned back by the query's
            y = turn(y, c.vcos[t, None].double(), -c.vsin[t, None].double(), dv, o.pair_halves)
        if c.gate is not None:
            g = torch.sigmoid(c.gate[t].double())
            y = y * (g[:, :, None] if o.gate_per_head else g.unflatten(1, (H, dv)))
        out.append(y.flatten(1))
    return torch.cat(out)
