"""The blocks and the grid of a prefill attention launch, as pt_grid of csrc/prefill_attn_tc.cu works them out."""
import types


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
