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
    # every CTA from the odd key on meets it; more of them than a CTA keeps marks of
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
