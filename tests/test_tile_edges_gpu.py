"""GPU: the tensor-core attention kernels and the vector paths of the per-channel kernels at the edges of their tiles: lengths around a
step of 80 keys and a tile of 128 rows, prompt portions that begin and end inside a CTA's tokens, head counts and sizes that fill a tile
only in part, states and taps with remainders.  Attention is compared with 64-bit arithmetic or with the fp32 CUDA-core kernel of
the same operation, vector paths with the plain path, which views that are not aligned take.

Tolerances (2-norm of the difference over 2-norm of the result): an output rounded to 16 bits is off by at most half a unit in the last
place, 2^-9 (bf16) or 2^-12 (fp16) of its value; attention rounds its softmax weights as well, so two units bound both roundings and
two kernels of one operation differ by at most two units each."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
UNIT = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}
TYPES = [torch.bfloat16, torch.float16]


def _rel(got, ref):
    got, ref = got.double(), ref.double()
    assert bool(torch.isfinite(got).all())
    return float((got - ref).norm() / ref.norm())


def _ints(v):
    return torch.tensor(list(v), dtype=torch.int32, device=DEV)


def _normal(*shape, seed, dtype=torch.float32):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV).to(dtype)


def _table(totals, bs, seed):
    per = [-(-n // bs) for n in totals]
    ids = torch.randperm(sum(per), generator=torch.Generator().manual_seed(seed)).tolist()
    bt = torch.zeros(len(totals), max(per), dtype=torch.int32)
    at = 0
    for s, n in enumerate(per):
        bt[s, :n] = torch.tensor(ids[at:at + n])
        at += n
    return bt.to(DEV), sum(per)


# ---------------------------------------------------------------- causal attention of prompts
def _causal(q, k, v, first):
    s = torch.einsum("nhd,lhd->hnl", q.double(), k.double()) * q.shape[-1] ** -0.5
    see = torch.arange(k.shape[0], device=DEV)[None, :] <= first + torch.arange(q.shape[0], device=DEV)[:, None]
    return torch.einsum("hnl,lhd->nhd", torch.softmax(s.masked_fill(~see, float("-inf")), dim=-1), v.double())


def _llama_state(lens, prefix=None):
    starts = [sum(lens[:i]) for i in range(len(lens))]
    return types.SimpleNamespace(prefill_seq_start_locs=_ints(starts), prefill_seq_lens=_ints(lens), softmax_scale=128 ** -0.5,
                                 num_prefill_seqs=len(lens), max_prefill_len=max(lens), seq_ids=_ints(range(len(lens))),
                                 prefill_prefix_lens=None if prefix is None else _ints(prefix))


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens", [(1, 79, 80, 81), (127, 128, 129), (159, 160, 161, 2), (240, 255, 256, 257), (385, 400)])
def test_packed_prompts_around_steps_and_tiles(dtype, lens):
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention
    H, G, T = 4, 2, sum(lens)
    qkv = _normal(T, (H + 2 * G) * 128, seed=T, dtype=dtype)
    q, k, v = (x.unflatten(1, (-1, 128)) for x in qkv.split([H * 128, G * 128, G * 128], dim=1))
    out = torch.empty(T, H, 128, dtype=dtype, device=DEV)
    prefill_attention(q, k, v, out, None, None, _llama_state(lens))
    at = 0
    for n in lens:
        s = slice(at, at + n)
        at += n
        ref = _causal(q[s], k[s].repeat_interleave(H // G, 1), v[s].repeat_interleave(H // G, 1), 0)
        assert _rel(out[s], ref) < UNIT[dtype], n


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens,prefix", [((1, 80, 81), (79, 0, 160)), ((128, 129), (1, 95)), ((257, 16), (63, 4000)), ((512,), (3584,))])
def test_prompt_portions_around_steps_and_tiles(dtype, lens, prefix):
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention_paged
    H, G, T = 4, 2, sum(lens)
    totals = [a + b for a, b in zip(lens, prefix)]
    bt, nb = _table(totals, 16, T)
    kc, vc = (_normal(nb, 1, G, 16, 128, seed=T + i, dtype=dtype) for i in (1, 2))
    q = _normal(T, H, 128, seed=T, dtype=dtype)
    out = torch.empty_like(q)
    prefill_attention_paged(q, kc, vc, bt, out, None, types.SimpleNamespace(block_size=16), _llama_state(lens, prefix), 0)
    at = 0
    for s, (n, total) in enumerate(zip(lens, totals)):
        k, v = (c[bt[s, :-(-total // 16)].long(), 0].transpose(1, 2).flatten(0, 1)[:total].repeat_interleave(H // G, 1) for c in (kc, vc))
        assert _rel(out[at:at + n], _causal(q[at:at + n], k, v, total - n)) < UNIT[dtype], (n, total)
        at += n


# ---------------------------------------------------------------- rows that are queries with their own position
PORTIONS = [[(1, 0), (3, 5), (130, 0)], [(64, 17), (65, 0)], [(31, 200), (33, 63), (2, 0)], [(200, 90)]]


def _token_state(portions, decodes):
    rows = portions + [(1, p) for p in decodes]
    return rows, types.SimpleNamespace(
        token_seq_ids=_ints(i for i, (n, _) in enumerate(rows) for _ in range(n)),
        token_positions=_ints(p + j for n, p in rows for j in range(n)), num_prefill_tokens=sum(n for n, _ in portions))


def _angles(positions, dims):
    f = torch.tensor([50.0 ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=DEV)
    a = positions.double()[:, None] * f
    return a.cos().float().contiguous(), a.sin().float().contiguous()


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("portions", PORTIONS)
@pytest.mark.parametrize("H,r,dr,dims,window,sink,bs", [
    (16, 512, 64, 64, 0, True, 16), (1, 64, 16, 8, 50, False, 16), (5, 192, 48, 48, 0, False, 8), (40, 256, 64, 32, 70, False, 16),
    (70, 320, 16, 16, 0, True, 4), (16, 512, 0, 0, 64, False, 16)])
def test_latent_rows_share_tiles(dtype, portions, H, r, dr, dims, window, sink, bs):
    from swiftllm_b200 import _lib
    from swiftllm_b200.worker.kernels.latent_attn import latent_attention
    rows, st = _token_state(portions, [77, 0])
    T = st.token_positions.shape[0]
    bt, nb = _table([n + p for n, p in rows], bs, T + r)
    cache = _normal(nb, 2, bs, r + dr, seed=r, dtype=dtype)
    q, qr = _normal(T, H, r, seed=T, dtype=dtype), _normal(T, H, 3 + dr, seed=T + 1, dtype=dtype)[:, :, 3:]
    gate = _normal(T, H, seed=T + 2, dtype=dtype)
    cos, sin = _angles(st.token_positions, dims) if dims else (None, None)
    outs = []
    for simt in (0, 1):
        old = _lib.lib().sllm_latent_attention_set_simt(simt)
        try:
            out = torch.empty_like(q)
            latent_attention(q, qr, gate, cache, 1, bt, st, out, dims, window, (r + dr) ** -0.5, cos, sin,
                             _normal(H, seed=9) if sink else None)
            outs.append(out)
        finally:
            _lib.lib().sllm_latent_attention_set_simt(old)
    assert _rel(*outs) < 2 * UNIT[dtype]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("portions", PORTIONS)
@pytest.mark.parametrize("H,G,dk,dv,rot,window,opts", [
    (16, 4, 128, 128, 64, 100, {}), (3, 1, 64, 128, 32, 0, {"out_f32": True}), (4, 4, 16, 48, 16, 33, {"pair_halves": True, "qk_norm_eps": 1e-5}),
    (6, 2, 80, 112, 0, 0, {"softcap": 5.0, "out_scale": 0.5}), (8, 4, 64, 128, 32, 0, {"vshare": 2, "chunk": 64, "prenorm": True}),
    (4, 2, 128, 128, 64, 50, {"pair_halves": True, "turned_values": True}),
    (8, 2, 128, 128, 0, 90, {"shared": True, "keep_first": 4, "slopes": True, "gate_per_head": True, "prenorm": True}),
    (8, 2, 96, 96, 0, 90, {"shared": True, "key_turned": 16, "sinks": True, "gate_per_head": True}),
    (40, 1, 64, 64, 64, 40, {"gate": False})])
def test_window_rows_share_tiles(dtype, portions, H, G, dk, dv, rot, window, opts):
    from swiftllm_b200 import _lib
    from swiftllm_b200.worker.kernels.window_attn import AttnOptions, shared_row_width, window_attention
    rows, st = _token_state(portions, [77, 0])
    T, opts = st.token_positions.shape[0], dict(opts)
    bt, nb = _table([n + p for n, p in rows], 16, T + dk)
    shared, prenorm, turned = opts.pop("shared", False), opts.pop("prenorm", False), opts.pop("turned_values", False)
    gated = opts.pop("gate", True)
    kt = opts.get("key_turned", 0)
    if shared:
        cache = _normal(nb, 1, 16, shared_row_width(G, dk, kt), seed=dk, dtype=dtype)
        inv = _normal(nb, 1, 16, G, seed=dk + 1).abs() * 0.2 + 0.9
        cache[..., :2 * G] = inv.contiguous().view(dtype).view(nb, 1, 16, 2 * G)
        opts["shared_kv"] = True
    else:
        cache = _normal(nb, 1, 16, G * dk + G // opts.get("vshare", 1) * dv, seed=dk, dtype=dtype)
    if prenorm:
        opts.update(q_norm=1 + 0.1 * _normal(dk, seed=4), prenorm_eps=1e-5)
    for name in ("slopes", "sinks"):
        if opts.pop(name, False):
            opts[name] = _normal(H, seed=5).abs() * 0.1
    opt = AttnOptions(**opts)
    proj = _normal(T, H * dk + H * dv, seed=T, dtype=dtype)
    q = proj[:, :H * dk]
    gate = (proj[:, H * dk:H * dk + (H if opt.gate_per_head else H * dv)]) if gated else None
    cos, sin = _angles(st.token_positions, rot) if rot else (None, None)
    vcos, vsin = _angles(st.token_positions, dv) if turned else (None, None)
    outs = []
    for simt in (0, 1):
        old = _lib.lib().sllm_window_attention_set_simt(simt)
        try:
            out = torch.empty(T, H * dv, dtype=torch.float32 if opt.out_f32 else dtype, device=DEV)
            window_attention(q, gate, cache, 0, bt, st, out, H, G, dk, dv, rot, window, dk ** -0.5, not shared, cos, sin, opt, vcos, vsin)
            outs.append(out)
        finally:
            _lib.lib().sllm_window_attention_set_simt(old)
    assert _rel(*outs) < 2 * UNIT[dtype]


# ---------------------------------------------------------------- per-channel kernels: vector path against the plain one
def _segments(lens, firsts):
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    return types.SimpleNamespace(
        batch_size=len(lens), num_prefill_seqs=len(lens), num_prefill_tokens=sum(lens), seq_ids=_ints(range(len(lens))), seg_starts=_ints(starts),
        token_seq_ids=_ints(i for i, n in enumerate(lens) for _ in range(n)),
        token_positions=_ints(f + j for n, f in zip(lens, firsts) for j in range(n)))


LENS = [((1, 2, 3, 40), (0, 7, 2, 0)), ((16, 17, 15), (1, 0, 3)), ((65,), (0,))]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens,firsts", LENS)
@pytest.mark.parametrize("C,taps,wide", [(4, 4, False), (516, 3, False), (1024, 4, True)])
def test_short_convolution_in_pieces(dtype, lens, firsts, C, taps, wide):
    from swiftllm_b200.worker.kernels.scan_ops import short_conv
    st, T = _segments(lens, firsts), sum(lens)
    tin = torch.float32 if wide else dtype
    base = _normal(T, C + 8, seed=C, dtype=tin)
    w, b = _normal(C, taps, seed=1) * 0.4, _normal(C, seed=2)
    outs = []
    for off in (0, 1):                                  # a view that is not aligned takes the plain path
        x = torch.zeros_like(base)[:, off:off + C]
        x.copy_(base[:, :C])
        tail = _normal(len(lens), taps - 1, C, seed=3, dtype=tin)
        outs.append((short_conv(x, w, b, tail, st, dtype, add_input=wide, silu=True, move_tail=True), tail))
    assert _rel(outs[0][0], outs[1][0]) < UNIT[dtype] and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens,firsts", LENS + [((32, 33, 31, 64), (0, 5, 0, 1))])
@pytest.mark.parametrize("C,N", [(8, 16), (40, 16), (2048, 16), (24, 8), (16, 24), (32, 64)])
def test_selective_scan_in_pieces(dtype, lens, firsts, C, N):
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    st, T = _segments(lens, firsts), sum(lens)
    base = _normal(T, 2 * C + 2 * N + 8, seed=C + N, dtype=dtype)
    dt, bias = _normal(T, C, seed=1), _normal(C, seed=2) - 3
    A, D = -(_normal(C, N, seed=3).abs() + 0.1), _normal(C, seed=4)
    outs = []
    for off in (0, 1):
        x = torch.zeros_like(base)[:, off:off + C]
        x.copy_(base[:, :C])
        state = _normal(len(lens), C, N, seed=5)
        y = selective_scan(x, dt, bias, A, base[:, 2 * C:], 0, N, D, base[:, C:2 * C], state, st)
        outs.append((y, state))
    # the states take no 16-bit rounding: both paths add the same 32-bit terms
    assert _rel(outs[0][0], outs[1][0]) < UNIT[dtype] and _rel(outs[0][1], outs[1][1]) < 1e-6
