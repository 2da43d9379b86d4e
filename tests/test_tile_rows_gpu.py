"""GPU: rows that share tiles with other rows (csrc/latent_attn_tc.cu, window_attn_tc.cu, prefill_attn_paged.cu, scan_ops.cu) take nothing
from keys that they do not see, and agree with 64-bit arithmetic in every part of a tile."""
import pytest
import torch

from tile_cases import DEV, TYPES, UNIT, attend, ints, normal, rel, segments, table
from tile_cases import latent_case, latent_exact, latent_run, window_case, window_columns, window_exact, window_run

pytestmark = pytest.mark.gpu


# ---------------------------------------------------------------- selective scan
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("C,N", [(2048, 16), (24, 8)])
def test_selective_scan_gate_is_the_plain_one(dtype, C, N):
    # without input to the state the output is silu(gate), rounded once: the vector path, the plain path (which a view that is not
    # aligned takes) and decoded tokens give the same bits only if they take the same exponential and quotient
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    T = 64
    one, zero = torch.ones(C, device=DEV), torch.zeros(T, 2 * N, dtype=dtype, device=DEV)
    z = normal(T, C + 8, seed=C, dtype=dtype) * 6
    A, dt = -torch.ones(C, N, device=DEV), torch.zeros(T, C, device=DEV)
    outs = []
    for off, decoded in ((0, False), (1, False), (0, True)):
        st = segments([1] * T, range(T), True) if decoded else segments([T], [0])
        gate = torch.zeros_like(z)[:, off:off + C]
        gate.copy_(z[:, :C])
        outs.append(selective_scan(torch.ones(T, C, dtype=dtype, device=DEV), dt, one, A, zero, 0, N, one, gate,
                                   torch.zeros(st.batch_size, C, N, device=DEV), st))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


# ---------------------------------------------------------------- keys that are not finite reach nobody who does not see them
def _poisoned(c, spots, cols, value):
    """The case's cache with `value` in columns `cols` of the rows of (sequence, position)s."""
    cache = c.cache.clone()
    bs = cache.shape[2]
    for s, p in spots:
        cache[int(c.bt[s, p // bs]), :, p % bs, cols] = value
    return cache


def _sees(c, spots, keep=0, chunk=0):
    """[rows] whether a row sees one of the (sequence, position)s."""
    out = []
    for s, (n, first) in enumerate(c.rows):
        for q in range(first, first + n):
            out.append(any(s == t and p <= q and (c.window <= 0 or q - p < c.window or p < keep) and (chunk <= 0 or p >= q // chunk * chunk)
                           for t, p in spots))
    return torch.tensor(out, device=DEV)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("H,r,dr,window,portions", [
    (16, 512, 64, 0, [(130, 5), (7, 90)]), (16, 512, 64, 33, [(130, 5), (7, 90)]), (1, 64, 16, 0, [(130, 0), (64, 3)]),
    (5, 192, 48, 20, [(100, 0)]), (16, 512, 64, 0, [(1200, 0)])])
def test_latent_keys_reach_only_rows_that_see_them(dtype, value, H, r, dr, window, portions):
    c = latent_case(dtype, portions, [77, 0], H, r, dr, dr, window, sink=True)
    spots = [(0, 43), (0, 66), (0, portions[0][0] - 2)]
    clean, got = latent_run(c), latent_run(c, _poisoned(c, spots, [3, r - 1], value))
    sees = _sees(c, spots)
    # a row that does not see the key: the same tiles, the same splits, zeros in place of a key with the weight 0
    assert torch.equal(got[~sees], clean[~sees])
    assert bool((~torch.isfinite(got[sees])).flatten(1).any(1).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("where", ["keys", "values"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("H,G,dk,dv,rot,window,opts", [
    (16, 4, 128, 128, 64, 33, {}), (4, 4, 80, 48, 16, 0, {"pair_halves": True, "out_f32": True}),
    (8, 4, 64, 128, 32, 0, {"vshare": 2, "chunk": 64}), (4, 2, 128, 128, 64, 50, {"pair_halves": True, "turned_values": True}),
    (8, 2, 128, 128, 0, 40, {"shared": True, "keep_first": 4, "slopes": True, "gate_per_head": True}),
    (8, 2, 96, 96, 0, 0, {"shared": True, "key_turned": 32, "sinks": True, "gate_per_head": True}), (64, 1, 64, 64, 64, 40, {"gate": False})])
def test_window_keys_reach_only_rows_that_see_them(dtype, where, value, H, G, dk, dv, rot, window, opts):
    # 700 tokens of 64 heads a group fill both tiles of a CTA; with fewer heads a CTA has half a tile
    c = window_case(dtype, [(700, 5), (7, 90)], [77, 0], H, G, dk, dv, rot, window, opts)
    k0, kw, v0, _ = window_columns(c)
    spots = [(0, 43), (0, 66), (0, 299), (0, 300), (0, 702)]
    cols = [k0 + kw - 1] if where == "keys" else [v0 + 3, v0 + dv - 1]
    clean, got = window_run(c), window_run(c, _poisoned(c, spots, cols, value))
    sees = _sees(c, spots, c.opt.keep_first, c.opt.chunk)
    assert torch.equal(got[~sees], clean[~sees])
    if where == "values" or value != value:                  # (a score of -infinity is a weight of 0)
        assert bool((~torch.isfinite(got[sees])).any(1).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,G,d", [(16, 4, 128), (4, 4, 80)])
def test_window_gate_of_prompt_rows_is_that_of_decoded_rows(dtype, H, G, d):
    # a window of one token and scores whose factors are applied beforehand (slopes): the weight is exactly 1 and O the value itself, so
    # the fp32 output is the value times the gate.  Decoded rows round the quotient exactly; half a unit more is one unit now and then
    c = window_case(dtype, [(150, 5)], [], H, G, d, d, 16, 1, {"out_f32": True, "sink": False, "slopes": True})
    prompt = window_run(c)
    c.st.num_prefill_tokens = 0
    decoded = window_run(c)
    assert float((prompt != decoded).float().mean()) < 0.01
    assert bool(((prompt - decoded).abs() <= 2.0 ** -22 * decoded.abs()).all())


# ---------------------------------------------------------------- portions whose keys are split between CTAs
def _split_case(dtype, lens, prefix, H=4, G=2):
    T, totals = sum(lens) + 3, [a + b for a, b in zip(lens, prefix)]              # three rows belong to no sequence
    bt, nb = table(totals, 16, T)
    kc, vc = (normal(nb, 1, G, 16, 128, seed=T + i, dtype=dtype) for i in (1, 2))
    return normal(T, H, 128, seed=T, dtype=dtype), kc, vc, bt


def _split_run(q, kc, vc, bt, lens, prefix, splits):
    from swiftllm_b200 import _lib
    T, H, D = q.shape
    starts = ints(sum(lens[:i]) for i in range(len(lens)))
    out, n = torch.full_like(q, 7.0), ints(lens)
    ws = torch.full((splits * T * H * (D + 2),), float("nan"), device=DEV)        # what nobody wrote is not read
    seqs, pre = ints(range(len(lens))), ints(prefix)
    _lib.check(_lib.lib().sllm_prefill_attention_paged_split(
        q.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), bt.data_ptr(), seqs.data_ptr(), starts.data_ptr(), n.data_ptr(),
        pre.data_ptr(), D ** -0.5, len(lens), max(lens), T, 0, 1, H, kc.shape[2], 16, D, bt.shape[1], kc.shape[0], H * D,
        _lib.dtype_tag(q.dtype), _lib.stream(), splits, ws.data_ptr()))
    torch.cuda.synchronize()
    return out


SPLIT_SHAPES = [((1, 300, 81), (0, 1000, 4000)), ((512,), (3584,)), ((257, 16, 1), (63, 4000, 700)), ((80, 130), (0, 31))]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("splits", [2, 3, 16, 64])
def test_split_keys_leave_other_rows_alone(dtype, splits):
    lens, prefix = SPLIT_SHAPES[0]
    q, kc, vc, bt = _split_case(dtype, lens, prefix)
    assert bool((_split_run(q, kc, vc, bt, lens, prefix, splits)[sum(lens):] == 7).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("splits", [1, 2, 5, 16])
def test_split_of_keys_that_are_not_finite_is_not_lost(dtype, splits):
    # every key of the first splits is NaN: so is every row, however the keys were split
    lens, prefix = (33,), (2000,)
    q, kc, vc, bt = _split_case(dtype, lens, prefix)
    kc[bt[0, :80].long()] = float("nan")
    assert bool(torch.isnan(_split_run(q, kc, vc, bt, lens, prefix, splits)[:33]).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,r,dr,dims,window,portions", [
    (16, 512, 64, 64, 0, [(130, 5), (7, 90), (1, 3)]), (16, 512, 64, 32, 100, [(600, 200), (95, 0)]), (1, 64, 16, 8, 50, [(130, 0), (65, 70)]),
    (5, 192, 48, 48, 0, [(33, 63), (64, 0)]), (40, 256, 64, 32, 70, [(31, 200), (2, 0)]), (70, 320, 0, 0, 0, [(20, 44)])])
def test_latent_rows_against_64_bits(dtype, H, r, dr, dims, window, portions):
    # weights and output are rounded to 16 bits, and the turned queries: three roundings of at most half a unit, that add as squares
    c = latent_case(dtype, portions, [77, 0, 500], H, r, dr, dims, window, sink=True)
    assert rel(latent_run(c), latent_exact(c)) < UNIT[dtype]


# CTAs of two full tiles: 16 heads on 4 groups need more than 36 x 64 prompt rows on 148 SMs, one group of 64 heads more than 147 x 4.
# Sequences end inside tile A (33 tokens), inside tile B (63) and beside whole CTAs
FULL = [(33, 0), (63, 5), (1, 0), (700, 90), (1500, 30), (95, 0)]
SHORT = [(1, 0), (3, 5), (130, 0), (65, 17)]
WINDOWS = [
    (16, 4, 128, 128, 64, 100, {}, FULL), (64, 1, 64, 64, 64, 40, {"gate": False}, [(3, 0), (1, 7), (600, 90), (2, 0), (5, 200)]),
    (16, 4, 128, 128, 0, 90, {"shared": True, "keep_first": 4, "slopes": True, "gate_per_head": True, "prenorm": True}, FULL),
    (16, 4, 128, 128, 0, 300, {"shared": True, "key_turned": 32, "sinks": True, "gate_per_head": True}, FULL),
    (16, 4, 128, 128, 64, 0, {"pair_halves": True, "turned_values": True, "qk_norm_eps": 1e-5, "softcap": 5.0, "sink": False}, FULL),
    (16, 4, 64, 128, 32, 0, {"vshare": 2, "chunk": 64, "prenorm": True, "out_f32": True, "gate": False}, FULL),
    (16, 4, 80, 112, 16, 50, {"softcap": 5.0, "out_scale": 0.5, "slopes": True}, FULL),
    (16, 4, 128, 128, 64, 100, {}, SHORT), (3, 1, 64, 128, 32, 0, {"out_f32": True}, SHORT),
    (4, 4, 80, 48, 16, 33, {"pair_halves": True, "qk_norm_eps": 1e-5}, SHORT), (4, 4, 16, 48, 16, 33, {"pair_halves": True}, SHORT), (8, 2, 96, 96, 0, 90, {"shared": True, "key_turned": 16}, SHORT)]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,G,dk,dv,rot,window,opts,portions", WINDOWS)
def test_window_rows_against_64_bits(dtype, H, G, dk, dv, rot, window, opts, portions):
    # as above: queries after norm and rotation, weights, and the output
    c = window_case(dtype, portions, [77, 0], H, G, dk, dv, rot, window, opts)
    got, ref = window_run(c), window_exact(c)
    at = 0
    for n, p in c.rows:                                      # a fault in a short sequence does not hide behind a long one
        assert rel(got[at:at + n], ref[at:at + n]) < UNIT[dtype], (n, p)
        at += n


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("splits", [1, 2, 3, 7, 16, 64])
@pytest.mark.parametrize("lens,prefix", SPLIT_SHAPES)
def test_split_keys_against_64_bits(dtype, splits, lens, prefix):
    # splits beyond the steps, one-row portions beside long ones, boundaries inside a query block's diagonal
    q, kc, vc, bt = _split_case(dtype, lens, prefix)
    got, at, H = _split_run(q, kc, vc, bt, lens, prefix, splits), 0, q.shape[1]
    for s, (n, p) in enumerate(zip(lens, prefix)):
        k, v = (c[bt[s, :-(-(n + p) // 16)].long(), 0].transpose(1, 2).flatten(0, 1)[:n + p].repeat_interleave(H // kc.shape[2], 1).double()
                for c in (kc, vc))
        score = torch.einsum("nhd,lhd->nhl", q[at:at + n].double(), k) * 128 ** -0.5
        seen = torch.arange(n + p, device=DEV)[None] <= p + torch.arange(n, device=DEV)[:, None]
        assert rel(got[at:at + n], attend(score, seen, v, None)) < UNIT[dtype], (n, p)
        at += n


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens,prefix", SPLIT_SHAPES)
def test_portions_of_a_step_split_their_keys(dtype, lens, prefix):
    # the entry point that the worker calls, with the length that it gives: the split count is its own
    import types
    from swiftllm_b200.worker.kernels.prefill_attn import _key_splits, prefill_attention_paged
    q, kc, vc, bt = _split_case(dtype, lens, prefix)
    longest = max(a + b for a, b in zip(lens, prefix))
    st = types.SimpleNamespace(
        num_prefill_seqs=len(lens), num_prefill_tokens=sum(lens), max_prefill_len=max(lens), seq_ids=ints(range(len(lens))), prefill_seq_lens=ints(lens),
        prefill_seq_start_locs=ints(sum(lens[:i]) for i in range(len(lens))), prefill_prefix_lens=ints(prefix), softmax_scale=128 ** -0.5,
        max_prefill_kv_len=longest)
    splits = _key_splits(4 * len(lens), max(lens), longest)
    assert splits > 1 or longest < 1280
    out = torch.full_like(q, 7.0)
    prefill_attention_paged(q, kc, vc, bt, out, None, types.SimpleNamespace(block_size=16), st, 0)
    assert torch.equal(out, _split_run(q, kc, vc, bt, lens, prefix, splits))


# ---------------------------------------------------------------- selective scan: the instances that other tests do not reach
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("dt_wide", [True, False])
@pytest.mark.parametrize("lens,C,N", [((15, 16, 17, 33), 8192, 16), ((32, 1, 31), 8192, 16), ((33, 70), 64, 16), ((9,), 128, 8)])
def test_selective_scan_lanes_and_step_types(dtype, dt_wide, lens, C, N):
    # four (three) segments of 8192 channels leave two lanes to a channel on 148 SMs; step sizes of the storage type
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    st, T = segments(lens, [0] * (len(lens) - 1) + [5]), sum(lens)
    base = normal(T, 2 * C + 2 * N + 8, seed=C + N, dtype=dtype)
    dt, bias = normal(T, C, seed=1, dtype=torch.float32 if dt_wide else dtype), normal(C, seed=2) - 3
    A, D = -(normal(C, N, seed=3).abs() + 0.1), normal(C, seed=4)
    outs = []
    for off in (0, 1):                                       # a view that is not aligned takes the plain path
        x = torch.zeros_like(base)[:, off:off + C]
        x.copy_(base[:, :C])
        state = normal(len(lens), C, N, seed=5)
        outs.append((selective_scan(x, dt, bias, A, base[:, 2 * C:], 0, N, D, base[:, C:2 * C], state, st), state))
    assert rel(outs[0][0], outs[1][0]) < UNIT[dtype] and rel(outs[0][1], outs[1][1]) < 1e-6


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens,C,N", [((40, 9), 64, 4), ((40, 9), 64, 8), ((33, 8, 20, 15), 2048, 8), ((17, 40), 8192, 4)])
def test_selective_scan_of_few_states_against_32_bit_rows(dtype, lens, C, N):
    # one state a lane, or four: the same steps as fp32 rows of the same values, to the output's rounding
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    st, T = segments(lens, [0] * (len(lens) - 1) + [5]), sum(lens)
    x, z, bc = (normal(T, n, seed=n + i, dtype=dtype) for i, n in enumerate((C, C, 2 * N)))
    dt, bias, A, D = normal(T, C, seed=1), normal(C, seed=2) - 3, -(normal(C, N, seed=3).abs() + 0.1), normal(C, seed=4)
    outs = []
    for t in (dtype, torch.float32):
        state = normal(len(lens), C, N, seed=5)
        outs.append((selective_scan(x.to(t), dt, bias, A, bc.to(t), 0, N, D, z.to(t), state, st), state))
    assert rel(outs[0][0], outs[1][0]) < UNIT[dtype] and rel(outs[0][1], outs[1][1]) < 1e-6


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("lens,C,taps,wide", [((1, 2, 3, 250, 44), 4096, 4, False), ((17, 184), 5252, 3, False), ((16, 15, 241), 4096, 4, True)])
def test_short_convolution_of_many_rows(dtype, lens, C, taps, wide):
    # 2^20 entries and more go in pieces of four channels, with the sums and the SiLU of the plain path, which other views take
    from swiftllm_b200.worker.kernels.scan_ops import short_conv
    st, T = segments(lens, [0, 7, 2, 0, 1][:len(lens)]), sum(lens)
    tin = torch.float32 if wide else dtype
    base, w, b = normal(T, C + 8, seed=C, dtype=tin), normal(C, taps, seed=1) * 0.4, normal(C, seed=2)
    outs = []
    for off in (0, 1):
        x = torch.zeros_like(base)[:, off:off + C]
        x.copy_(base[:, :C])
        tail = normal(len(lens), taps - 1, C, seed=3, dtype=tin)
        outs.append((short_conv(x, w, b, tail, st, dtype, add_input=wide, silu=True, move_tail=True), tail))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


# ---------------------------------------------------------------- how often a result is rounded
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,T,length", [(16, 64, 2000), (5, 40, 700), (1, 9, 3000)])
def test_latent_decoded_tokens_round_their_weights_finely(dtype, H, T, length):
    # without turned entries nothing but the output is rounded to 16 bits: values spread evenly over a binade's logarithm are then off by
    # unit / sqrt(12) * sqrt(0.75 / (2 ln 2)) = 0.2123 units (root of the mean square, relative); 6 % for the draw.  Weights rounded to
    # 16 bits, but for the largest of every key split, added a sixth
    c = latent_case(dtype, [], [length - 7 * i for i in range(T)], H, 512, 0, 0, 0, sink=False, gated=False)
    assert rel(latent_run(c), latent_exact(c)) < 1.06 * 0.2123 * 2 * UNIT[dtype]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("opts", [{}, {"softcap": 5.0}, {"slopes": True}])
def test_window_weights_sum_to_one(dtype, opts):
    # equal values come out as they are, whatever the weights were rounded to: sum and product take the same weights
    c = window_case(dtype, [(300, 5), (1, 0), (700, 90)], [], 16, 4, 128, 128, 0, 200, {"out_f32": True, "gate": False, "sink": False, **opts})
    c.cache[..., 4 * 128:] = 1.5
    assert float((window_run(c) - 1.5).abs().max()) < 1e-5
