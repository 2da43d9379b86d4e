"""GPU: paged attention whose CTAs walk many items, each finished behind the next one's first tile (csrc/paged_attn_tc.cu): items of one and of several tiles in
turns, sequences without tokens between them and at the end, every width of a group, one split and several.

The softmax's weights and the output are rounded once each, by at most half a unit in the last place: 2^-8 (bf16), 2^-11 (fp16) together."""
import types

import pytest
import torch

from tile_cases import DEV, TYPES, UNIT, ints, normal, rel

pytestmark = pytest.mark.gpu
SOME = (40, 129, 1, 0, 300, 128, 16, 256, 7, 0, 0, 385)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,G,B,sbs", [(8, 8, 130, 0), (12, 6, 170, 0), (32, 8, 230, 0), (16, 2, 501, 0), (16, 1, 950, 0), (32, 8, 60, 128), (16, 2, 220, 256), (6, 2, 2, 0)])
def test_items_behind_one_another(dtype, H, G, B, sbs):
    from swiftllm_b200.worker.kernels.paged_attn import paged_attention
    lens = [SOME[i % len(SOME)] for i in range(B)]
    blocks = [-(-n // 16) for n in lens]
    kc, vc = (normal(sum(blocks), 1, G, 16, 128, seed=i, dtype=dtype) for i in (1, 2))
    table = torch.zeros(B, max(blocks), dtype=torch.int32)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]))
    table, q, out = table.to(DEV), normal(B, H, 128, seed=4, dtype=dtype), torch.full((B, H * 128), 7.0, dtype=dtype, device=DEV)
    st = types.SimpleNamespace(num_decoding_seqs=B, num_prefill_seqs=0, seq_ids=ints(range(B)), decoding_seq_lens=ints(lens), softmax_scale=128 ** -0.5,
                               max_decoding_len=max(lens), paged_attn_seq_block_size=sbs)
    for _ in range(2):
        paged_attention(q, kc, vc, table, None, types.SimpleNamespace(block_size=16), st, 0, out)
    for i, n in enumerate(lens):
        if n == 0:
            continue                                         # (no tokens: nobody's row)
        k, v = (c[table[i, :blocks[i]].long(), 0].transpose(1, 2).flatten(0, 1)[:n].double().repeat_interleave(H // G, 1) for c in (kc, vc))
        w = torch.softmax(torch.einsum("hd,nhd->hn", q[i].double(), k) * 128 ** -0.5, dim=1)
        assert rel(out[i], torch.einsum("hn,nhd->hd", w, v).flatten()) < UNIT[dtype], (i, n)


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("H,G,B,sbs", [(9, 1, 260, 0), (24, 2, 60, 128), (32, 2, 230, 256), (11, 1, 3, 128)])
def test_wide_groups_one_item_after_the_other(dtype, H, G, B, sbs):
    test_items_behind_one_another(dtype, H, G, B, sbs)
