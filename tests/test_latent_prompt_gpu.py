"""GPU: latent attention of prompt rows by tiles of whole cache blocks (csrc/latent_attn_prompt.cu): heads that fill a CTA's rows only in part,
segments that end inside a CTA's tokens, tiles that begin in front of a window and end behind the last key, blocks of 16, 32 and 48 tokens, views
that are not aligned; what lies in the cache outside a segment's keys is never multiplied, and a key that is not finite reaches only rows that see it.

Weights, turned queries and the output are rounded to 16 bits: three roundings of at most half a unit, that add as squares."""
import pytest
import torch

from tile_cases import TYPES, UNIT, latent_case, latent_exact, latent_run, rel

pytestmark = pytest.mark.gpu
# 444 CTAs of 64 rows on 148 SMs, and a few more
CASES = [(16, 0, 16, [(1800, 0)]), (16, 100, 16, [(1201, 3), (63, 0), (1, 40), (700, 1000)]), (32, 33, 32, [(450, 7), (33, 100), (500, 0)]),
         (5, 0, 48, [(1700, 5), (2000, 0)]), (20, 1000, 16, [(530, 1100), (400, 0)]), (64, 0, 16, [(390, 0), (65, 70)]), (2, 70, 16, [(1900, 17)] * 8)]


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,window,bs,portions", CASES)
def test_prompt_rows_against_64_bits(dtype, H, window, bs, portions):
    c = latent_case(dtype, portions, [], H, 512, 64, 64, window, sink=window == 0, bs=bs, gated=window > 0)
    got, ref, at = latent_run(c), latent_exact(c), 0
    for n, p in c.rows:
        assert rel(got[at:at + n], ref[at:at + n]) < UNIT[dtype], (n, p)
        at += n


@pytest.mark.parametrize("H,window,bs,portions", CASES[:4])
def test_rows_behind_the_last_key_and_other_layers_are_not_multiplied(H, window, bs, portions):
    c = latent_case(torch.bfloat16, portions, [], H, 512, 64, 64, window, sink=False, bs=bs)
    clean, cache = latent_run(c), torch.full_like(c.cache, float("nan"))
    for s, (n, p) in enumerate(c.rows):                      # only the positions that a row of the step sees
        for pos in range(max(0, p - window + 1) if window else 0, n + p):
            cache[int(c.bt[s, pos // bs]), 1, pos % bs] = c.cache[int(c.bt[s, pos // bs]), 1, pos % bs]
    assert torch.equal(latent_run(c, cache), clean)


def test_views_that_are_not_aligned():
    from swiftllm_b200.worker.kernels.latent_attn import latent_attention
    c = latent_case(torch.float16, [(1400, 9), (533, 0)], [], 16, 512, 64, 32, 0, sink=True)
    clean = latent_run(c)
    odd = lambda x: torch.cat((x[..., :1], x), -1)[..., 1:]
    out = torch.zeros(c.q.shape[0], 16, 513, dtype=c.q.dtype, device=c.q.device)[:, :, 1:]
    latent_attention(c.q, odd(c.qr.contiguous()), c.gate, c.cache, 1, c.bt, c.st, out, c.dims, 0, c.scale, c.cos, c.sin, c.sink)
    assert torch.equal(out, clean)
    latent_attention(odd(c.q), c.qr, c.gate, c.cache, 1, c.bt, c.st, out, c.dims, 0, c.scale, c.cos, c.sin, c.sink)      # (the kernel of other sizes)
    assert rel(out, clean) < 2 * UNIT[torch.float16]


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("H,window,portions", [(16, 0, [(1800, 5), (7, 90)]), (64, 33, [(200, 5), (300, 90)])])
def test_keys_reach_only_rows_that_see_them(value, H, window, portions):
    # every CTA from the odd key on meets it (64 heads: a token a CTA, whose keys are all its own)
    c = latent_case(torch.bfloat16, portions, [], H, 512, 64, 64, window, sink=True)
    spots, clean, cache, at = [41, 42, 66, 120, 130], latent_run(c), c.cache.clone(), 0
    for pos in spots:
        cache[int(c.bt[0, pos // 16]), :, pos % 16, [3, 511]] = value
    got = latent_run(c, cache)
    q = torch.arange(portions[0][0], device=c.q.device) + portions[0][1]
    sees = torch.zeros(c.q.shape[0], dtype=torch.bool, device=c.q.device)
    for pos in spots:
        sees[:q.shape[0]] |= (q >= pos) & ((q - pos < window) if window else True)
    assert torch.equal(got[~sees], clean[~sees]) and bool((~torch.isfinite(got[sees])).flatten(1).any(1).all())


# 64 tokens a CTA whose runs end anywhere in it; two blocks of heads, the last one in part
@pytest.mark.parametrize("H,window,portions", [(1, 0, [(33 + i % 31, (7 * i) % 90) for i in range(500)] + [(2500, 0), (2101, 33)]),
                                               (1, 100, [(1, 4), (62, 0), (65, 128)] + [(4000, 900)] * 7 + [(500, 3)]), (72, 0, [(150, 20), (90, 0)]), (96, 70, [(233, 10)])])
def test_one_head_and_more_than_64(H, window, portions):
    c = latent_case(torch.bfloat16, portions, [], H, 512, 64, 64, window, sink=False, gated=True)
    got, ref, at = latent_run(c), latent_exact(c), 0
    for n, p in c.rows:
        assert rel(got[at:at + n], ref[at:at + n]) < UNIT[torch.bfloat16], (n, p)
        at += n


@pytest.mark.parametrize("value", [float("nan"), float("-inf")])
def test_more_segments_than_a_cta_keeps_marks_of(value):
    # 32 tokens a CTA, 16 segments of two, three CTAs or more in turn: the 32 marks are looked through in the middle of a CTA's work, and again
    portions = [(2, (5 * i) % 130) for i in range(7200)]
    c = latent_case(torch.bfloat16, portions, [], 2, 512, 64, 64, 0, sink=True)
    clean, cache = latent_run(c), c.cache.clone()
    first = torch.arange(len(portions), device=c.q.device)
    bad = first % 3 != 1
    pos = torch.tensor([p + 1 for _, p in portions], device=c.q.device)      # the second token's own key, which the first does not see
    block = c.bt[first, pos // 16].long()
    cache[block[bad], 1, pos[bad] % 16, 300] = value
    got = latent_run(c, cache).unflatten(0, (-1, 2))
    clean = clean.unflatten(0, (-1, 2))
    assert torch.equal(got[:, 0], clean[:, 0]) and torch.equal(got[~bad], clean[~bad])
    assert bool((~torch.isfinite(got[bad][:, 1])).flatten(1).any(1).all())


@pytest.mark.parametrize("window", [33, 64, 1000])
def test_keys_that_only_some_tokens_of_a_segment_see_through_a_window(window):
    # four tokens a CTA: keys behind the first of them, and keys in front of the last one's window
    n, p = 1800, 5
    c = latent_case(torch.float16, [(n, p), (7, 90)], [], 16, 512, 64, 64, window, sink=True)
    clean, cache, spots = latent_run(c), c.cache.clone(), [41, 42, 203, 1206, 1500]
    for pos in spots:
        cache[int(c.bt[0, pos // 16]), 1, pos % 16, [3, 511]] = float("nan")
    got = latent_run(c, cache)
    q = torch.arange(n, device=c.q.device) + p
    sees = torch.zeros(c.q.shape[0], dtype=torch.bool, device=c.q.device)
    for pos in spots:
        sees[:n] |= (q >= pos) & (q - pos < window)
    assert torch.equal(got[~sees], clean[~sees]) and bool((~torch.isfinite(got[sees])).flatten(1).any(1).all())


@pytest.mark.parametrize("broadcast", ["heads", "tokens", "turned"])
def test_query_views_of_other_strides(broadcast):
    # heads or tokens that share their entries go to the kernel of other sizes; heads outside of tokens stay
    from swiftllm_b200.worker.kernels.latent_attn import latent_attention
    c = latent_case(torch.bfloat16, [(1400, 9), (533, 0)], [], 16, 512, 64, 64, 0, sink=True)
    T = c.q.shape[0]
    view = c.q[:, :1].expand(T, 16, 512) if broadcast == "heads" else c.q[:1].expand(T, 16, 512) if broadcast == "tokens" else \
        c.q.transpose(0, 1).contiguous().transpose(0, 1)
    c.q, out = view.contiguous(), torch.empty_like(c.q)
    clean = latent_run(c)
    latent_attention(view, c.qr, c.gate, c.cache, 1, c.bt, c.st, out, c.dims, 0, c.scale, c.cos, c.sin, c.sink)
    assert torch.equal(out, clean) if broadcast == "turned" else rel(out, clean) < 2 * UNIT[torch.bfloat16]
