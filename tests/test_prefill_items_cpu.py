"""CPU: the numbering of query blocks that persistent prefill CTAs search (pt_block, csrc/prefill_attn_tc_kernel.cuh), in Python as the kernel does it, against a
plain enumeration: blocks of the highest number first, the sequences of a number in order."""
import pytest
import torch

from prefill_grid import WARP, WIDE, Search, prefill_grid


def enumeration(blocks, max_blocks):
    return [(s, b) for b in reversed(range(max_blocks)) for s, n in enumerate(blocks) if n > b]


def _blocks(kind, n):
    g = torch.Generator().manual_seed(n)
    if kind == "one long":
        return [37 if s == n // 2 else 1 for s in range(n)]
    if kind == "empty ones":
        return [s % 3 for s in range(n)]
    return (torch.rand(n, generator=g) * (1 if kind == "single" else 12)).ceil().int().tolist()


@pytest.mark.parametrize("kind", ["single", "spread", "one long", "empty ones"])
@pytest.mark.parametrize("n", [1, 31, 33, 128, 129, 300, 1000])
@pytest.mark.parametrize("heads,by_head", [(1, True), (8, True), (8, False)])
def test_every_cta_finds_its_blocks(kind, n, heads, by_head):
    blocks = _blocks(kind, n)
    most = max(1, max(blocks)) + 1                           # (the caller's longest may be longer than any)
    order = enumeration(blocks, most)
    grid = [(h, r) for r in range(len(order)) for h in range(heads)] if by_head else [(h, r) for h in range(heads) for r in range(len(order))]
    for cta in (0, 1, 147):                                  # ranks of a CTA among 148 that take the grid's next in turn
        search = Search(blocks, most)
        mine = grid[cta::148]
        for _, rank in mine:
            assert search(rank) == order[rank]
        if kind == "single" and heads == 8 and by_head and n > WARP:      # the lengths are read about once a CTA, not several times an item
            assert search.reads <= 2 * (n + WIDE) + WIDE * len(mine)


@pytest.mark.parametrize("H,G,lens", [(16, 16, (1024, 121, 754, 363)), (32, 32, (300, 35, 221, 106)), (24, 4, (1024, 121, 754, 363))])
def test_the_last_items_are_the_shortest(H, G, lens):
    """Portions of one to four items an SM, in the grid's order: what is left for the second round are no long items."""
    g = prefill_grid(H, G, len(lens), max(lens), sum(lens), 1, True)
    order = enumeration([-(-n // g.tokens) for n in lens], g.most)
    assert g.many and g.by_head and 148 < g.heads * g.slots <= 4 * 148
    items = [b for _, b in order for _ in range(g.heads)]
    assert max(items[148:]) <= min(items[:148])


SHAPES = [(64, 8, 1, 16, 16), (64, 8, 1, 64, 64), (32, 8, 4, 16, 45), (32, 8, 1, 300, 300), (32, 8, 1, 512, 512), (16, 4, 1, 64, 64), (24, 4, 4, 64, 150),
          (16, 16, 1, 300, 300), (16, 1, 3, 40, 41), (64, 8, 1, 700, 700), (32, 8, 32, 500, 8000), (6, 2, 2, 1, 2), (48, 8, 7, 333, 334)]


@pytest.mark.parametrize("H,G,n,longest,rows", SHAPES)
def test_blocks_are_counted_as_the_launch_makes_them(H, G, n, longest, rows):
    from swiftllm_b200.worker.kernels.prefill_attn import _blocks
    for tiles, got in zip((1, 2), _blocks(H, G, n, longest, rows)):
        g = prefill_grid(H, G, n, longest, rows, 1, True, sms=1 << 30 if tiles == 1 else 0)
        assert g.tiles == tiles and got == g.heads * min(n * -(-longest // g.tokens), rows // g.tokens + n)


@pytest.mark.parametrize("H,G,n,longest,rows", SHAPES)
@pytest.mark.parametrize("kv_len", [0, 479, 700, 1016, 3300, 5064, 30000])
def test_key_splits_fill_the_sms_and_no_more(H, G, n, longest, rows, kv_len):
    from swiftllm_b200.worker.kernels.prefill_attn import _blocks, _splits
    sms = 148
    splits = _splits(sms, kv_len, *_blocks(H, G, n, longest, rows), True)
    g = prefill_grid(H, G, n, longest, rows, splits, True, sms)
    assert 1 <= splits <= 16 and (splits == 1 or kv_len // splits >= 480)
    if splits > 1:
        assert g.heads * g.slots <= sms or g.heads * n * splits * -(-longest // g.tokens) <= sms
    if splits < min(16, kv_len // 640):                      # keys for more CTAs, but no SMs: at least half of them have one
        assert 2 * splits * _blocks(H, G, n, longest, rows)[0] > sms
