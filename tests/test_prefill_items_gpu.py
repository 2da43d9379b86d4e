"""GPU: prompts whose query blocks persistent CTAs take from the launch's grid: heads of one key/value head side by side in a tile (one to
eight, and groups that are no power of two), more sequences than a warp has lanes, blocks that end inside a tile, many more blocks than SMs,
sequences that share rows, and a stated longest length below a sequence's own.

An output rounded to 16 bits is off by at most half a unit in the last place, and so are the softmax's weights: two units bound both."""
import types

import pytest
import torch

from prefill_grid import prefill_grid
from tile_cases import DEV, TYPES, UNIT, ints, normal, rel, table

pytestmark = pytest.mark.gpu
SHAPES = [(4, 4, (1, 255, 257, 128)), (6, 2, (127, 130, 300)), (8, 4, (63, 64, 65, 129, 511)), (8, 2, (31, 32, 33, 64, 65, 700)),
          (16, 2, (15, 16, 17, 32, 33, 500)), (16, 1, (1, 300, 40)), (12, 2, (200, 31)), (8, 2, tuple(range(1, 75))),
          (32, 8, (1500, 3, 1777, 900, 80, 81))]


def _causal(q, k, v, first):
    s = torch.einsum("nhd,lhd->hnl", q.double(), k.double()) * 128 ** -0.5
    see = torch.arange(k.shape[0], device=DEV)[None, :] <= first + torch.arange(q.shape[0], device=DEV)[:, None]
    return torch.einsum("hnl,lhd->nhd", torch.softmax(s.masked_fill(~see, float("-inf")), dim=-1), v.double())


def _state(lens, starts=None, longest=None, **more):
    starts = [sum(lens[:i]) for i in range(len(lens))] if starts is None else starts
    return types.SimpleNamespace(prefill_seq_start_locs=ints(starts), prefill_seq_lens=ints(lens), softmax_scale=128 ** -0.5, num_prefill_seqs=len(lens),
                                 max_prefill_len=max(lens) if longest is None else longest, seq_ids=ints(range(len(lens))), **more)


def _packed(dtype, H, G, T):
    qkv = normal(T, (H + 2 * G) * 128, seed=T, dtype=dtype)
    return tuple(x.unflatten(1, (-1, 128)) for x in qkv.split([H * 128, G * 128, G * 128], dim=1))


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,G,lens", SHAPES)
def test_packed_prompts(dtype, H, G, lens):
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention
    q, k, v = _packed(dtype, H, G, sum(lens))
    out = torch.full((sum(lens) + 1, H, 128), 7.0, dtype=dtype, device=DEV)
    prefill_attention(q, k, v, out[:-1], None, None, _state(lens))
    at = 0
    for n in lens:
        s = slice(at, at + n)
        at += n
        assert rel(out[s], _causal(q[s], k[s].repeat_interleave(H // G, 1), v[s].repeat_interleave(H // G, 1), 0)) < UNIT[dtype], n
    assert bool((out[-1] == 7.0).all())


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,G,lens", SHAPES)
@pytest.mark.parametrize("splits", [1, 3])
def test_portions(dtype, H, G, lens, splits):
    from swiftllm_b200 import _lib
    prefix = [(97 * i) % 400 for i in range(len(lens))]
    totals, T = [a + b for a, b in zip(lens, prefix)], sum(lens)
    bt, nb = table(totals, 16, T)
    kc, vc = (normal(nb, 2, G, 16, 128, seed=T + i, dtype=dtype) for i in (1, 2))
    q, out, st = normal(T, H, 128, seed=T, dtype=dtype), torch.full((T, H, 128), 7.0, dtype=dtype, device=DEV), _state(lens)
    ws, pre = torch.full((splits * T * H * 130,), float("nan"), device=DEV), ints(prefix)
    _lib.check(_lib.lib().sllm_prefill_attention_paged_split(
        q.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), bt.data_ptr(), st.seq_ids.data_ptr(), st.prefill_seq_start_locs.data_ptr(),
        st.prefill_seq_lens.data_ptr(), pre.data_ptr(), 128 ** -0.5, len(lens), max(lens), T, 1, 2, H, G, 16, 128, bt.shape[1], nb, H * 128,
        _lib.dtype_tag(dtype), _lib.stream(), splits, ws.data_ptr()), "prefill_attention_paged_split")
    at = 0
    for s, (n, total) in enumerate(zip(lens, totals)):
        k, v = (c[bt[s, :-(-total // 16)].long(), 1].transpose(1, 2).flatten(0, 1)[:total].repeat_interleave(H // G, 1) for c in (kc, vc))
        assert rel(out[at:at + n], _causal(q[at:at + n], k, v, total - n)) < UNIT[dtype], (n, total)
        at += n


def test_sequences_that_share_rows_and_a_longest_below():
    # more query blocks than rows / block: a CTA takes several of the grid's; rows past the whole 256 behind the stated longest stay as they are
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention
    H, G, T = 8, 2, 600
    q, k, v = _packed(torch.float16, H, G, T)
    out = torch.full((T, H, 128), 7.0, dtype=torch.float16, device=DEV)
    prefill_attention(q, k, v, out, None, None, _state([600] * 12, [0] * 12, 300))
    ref = _causal(q, k.repeat_interleave(4, 1), v.repeat_interleave(4, 1), 0)
    assert rel(out[:512], ref[:512]) < UNIT[torch.float16] and bool((out[512:] == 7.0).all())


# more sequences than a warp has lanes: several numbers of blocks, sequences without rows among them, one long one among short ones
MANY = [tuple((37 * i) % 150 for i in range(300)), tuple(900 if i == 170 else 1 + i % 9 for i in range(333)), (70,) * 129]


@pytest.mark.parametrize("H,G", [(8, 8), (8, 2), (8, 1)])
@pytest.mark.parametrize("lens", MANY)
def test_many_prompts(H, G, lens):
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention
    T = sum(lens)
    q, k, v = _packed(torch.float16, H, G, T)
    out = torch.full((T + 1, H, 128), 7.0, dtype=torch.float16, device=DEV)
    prefill_attention(q, k, v, out[:-1], None, None, _state(lens))
    at = 0
    for n in lens:
        s = slice(at, at + n)
        at += n
        if n:
            assert rel(out[s], _causal(q[s], k[s].repeat_interleave(H // G, 1), v[s].repeat_interleave(H // G, 1), 0)) < UNIT[torch.float16], n
    assert bool((out[-1] == 7.0).all())


@pytest.mark.parametrize("lens", MANY)
@pytest.mark.parametrize("splits", [1, 2])
def test_many_portions(lens, splits):
    test_portions(torch.bfloat16, 8, 2, tuple(max(n, 1) for n in lens), splits)


# more query blocks than the grid has, because sequences share rows: a CTA goes on by so many, and takes the grid's next only behind its last
def _shared(n):
    g = prefill_grid(64, 8, n, 700, 600, 1, False, torch.cuda.get_device_properties(0).multi_processor_count)
    assert g.many and g.asks and n * -(-600 // g.tokens) > 2 * g.slots
    return g


def test_packed_prompts_that_share_rows_and_take_ctas():
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention
    H, G, T, n = 64, 8, 600, 40
    _shared(n)
    q, k, v = _packed(torch.bfloat16, H, G, T)
    out = torch.full((T, H, 128), 7.0, dtype=torch.bfloat16, device=DEV)
    prefill_attention(q, k, v, out, None, None, _state([T] * n, [0] * n, 700))
    assert rel(out, _causal(q, k.repeat_interleave(8, 1), v.repeat_interleave(8, 1), 0)) < UNIT[torch.bfloat16]


@pytest.mark.parametrize("splits", [1, 3])
def test_portions_that_share_rows_and_take_ctas(splits):
    from swiftllm_b200 import _lib
    H, G, T, n, pre, dtype = 64, 8, 600, 40, 333, torch.float16
    _shared(n)
    bt, nb = table([T + pre], 16, 3)
    kc, vc = (normal(nb, 2, G, 16, 128, seed=i, dtype=dtype) for i in (1, 2))
    q, out = normal(T, H, 128, seed=3, dtype=dtype), torch.full((T, H, 128), 7.0, dtype=dtype, device=DEV)
    ws = torch.full((splits * T * H * 130,), float("nan"), device=DEV)
    zeros, lens, prefix = ints([0] * n), ints([T] * n), ints([pre] * n)
    _lib.check(_lib.lib().sllm_prefill_attention_paged_split(
        q.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), bt.data_ptr(), zeros.data_ptr(), zeros.data_ptr(), lens.data_ptr(), prefix.data_ptr(),
        128 ** -0.5, n, 700, T, 1, 2, H, G, 16, 128, bt.shape[1], nb, H * 128, _lib.dtype_tag(dtype), _lib.stream(), splits, ws.data_ptr()), "portions")
    k, v = (c[bt[0].long(), 1].transpose(1, 2).flatten(0, 1)[:T + pre].repeat_interleave(8, 1) for c in (kc, vc))
    assert rel(out, _causal(q, k, v, pre)) < UNIT[dtype]
