"""The blocks and the grid of a prefill attention launch, as pt_grid of csrc/prefill_attn_tc.cu works them out, and the search for a CTA's blocks, as
pt_block of csrc/prefill_attn_tc_kernel.cuh goes about it."""
import types

WARP, WIDE = 32, 128


def prefill_grid(H, G, seqs, longest, rows, splits, paged, sms=148):
    pack = 1
    while pack < 8 and H // G % (2 * pack) == 0:
        pack *= 2
    heads, up = H // pack, lambda a, b: -(-a // b)
    blocks = lambda tiles: min(seqs * up(longest, tiles * 128 // pack), rows // (tiles * 128 // pack) + seqs)
    ones, short = heads * splits * blocks(1), not paged and longest <= 320
    tiles = 1 if ones <= sms or short and 2 * ones <= 5 * sms else 2
    tokens = tiles * 128 // pack
    slots = min(blocks(tiles) * splits, 65535)
    room = 2 * sms if short else 3 * sms // 2 if paged and heads * slots <= sms else sms
    many = heads * seqs * splits * up(longest, tokens) > room
    return types.SimpleNamespace(pack=pack, heads=heads, tiles=tiles, tokens=tokens, most=up(longest, 256) * 256 // tokens, many=many, slots=slots,
                                 asks=many and (not paged or heads * slots > sms), by_head=many and (not paged or sms < heads * slots <= 4 * sms))


class Search:
    """pt_block with its cursor; `reads`: lengths of sequences past the warp's own 32 that were read."""

    def __init__(self, blocks, max_blocks):
        self.blocks, self.max_blocks, self.reads = [min(b, max_blocks) for b in blocks], max_blocks, 0
        self.total = sum(self.blocks)
        self.block = self.first = self.count = self.s0 = self.before = 0

    def _from(self, b):
        self.reads += max(0, len(self.blocks) - WARP)
        return sum(max(n - b, 0) for n in self.blocks)

    def __call__(self, rank):
        if rank < self.first or rank >= self.first + self.count:
            lo, hi, from_lo, from_hi = 0, self.max_blocks, self.total, 0
            while hi - lo > 1:
                mid = (lo + hi) // 2
                n = self._from(mid)
                if n > rank:
                    lo, from_lo = mid, n
                else:
                    hi, from_hi = mid, n
            self.block, self.first, self.count, self.s0, self.before = lo, from_hi, from_lo - from_hi, 0, 0
        elif rank < self.first + self.before:
            self.s0 = self.before = 0
        r = rank - self.first
        while self.s0 < len(self.blocks):
            n = self.before
            for s in range(self.s0, self.s0 + WIDE):
                self.reads += WARP <= s < len(self.blocks)
                if s < len(self.blocks) and self.blocks[s] > self.block:
                    if n == r:
                        return s, self.block
                    n += 1
            self.before = n
            self.s0 += WIDE
        raise AssertionError("a rank without a sequence")
