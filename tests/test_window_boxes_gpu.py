"""GPU: windowed attention of prompt rows whose keys and values come in boxes of 16 cache rows (csrc/window_attn_tc.cu): a window that begins inside a box, a
last box filled in part, cache blocks of several boxes, and of sizes that hold no whole ones; what lies in the cache outside a segment's keys is
never multiplied.

Queries after their rotation, weights and the output are rounded to 16 bits: three roundings of at most half a unit, that add as squares."""
import pytest
import torch

from tile_cases import DEV, TYPES, UNIT, rel, table, window_case, window_exact, window_run

pytestmark = pytest.mark.gpu
CASES = [(100, [(33, 0), (63, 5), (1, 0), (700, 90), (95, 0)]), (0, [(130, 0), (5, 15), (65, 17)]), (33, [(300, 200)]), (1024, [(64, 1500)]), (16, [(80, 16), (81, 15)])]


def _blocks_of(c, bs):
    """The case's cache in blocks of bs tokens, NaN wherever no row of the step looks."""
    bt, nb = table([n + p for n, p in c.rows], bs, 5)
    cache = torch.full((nb, 1, bs, c.cache.shape[3]), float("nan"), dtype=c.cache.dtype, device=DEV)
    for s, (n, p) in enumerate(c.rows):
        at = torch.arange(max(0, p - c.window + 1) if c.window else 0, n + p, device=DEV)
        cache[bt[s, at // bs].long(), 0, at % bs] = c.cache[c.bt[s, at // 16].long(), 0, at % 16]
    return bt, cache


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("opts", [{}, {"softcap": 5.0}])
@pytest.mark.parametrize("window,portions", CASES)
def test_blocks_of_any_size(dtype, window, portions, opts):
    c = window_case(dtype, portions, [], 16, 4, 128, 128, 64, window, opts)
    ref, clean, at = window_exact(c), window_run(c), 0
    for n, p in c.rows:
        assert rel(clean[at:at + n], ref[at:at + n]) < UNIT[dtype], (n, p)
        at += n
    for bs in (16, 48, 24):
        c.bt, c.cache = _blocks_of(window_case(dtype, portions, [], 16, 4, 128, 128, 64, window, opts), bs)
        got = window_run(c)
        if bs != 24:                                         # (others come row by row, in steps that begin with the window)
            assert torch.equal(got, clean)
        else:
            assert rel(got, ref) < UNIT[dtype]
