"""GPU: the items of a paged-attention launch (csrc/paged_attn_tc.cu) against 64 bits.  Splits that meet in a cluster: two to eight, splits
that a shorter sequence does not have, every width of a group, the largest launch that takes the path beside the first that does not.
Counted splits: batches around every edge of the scan and of the search, lengths that are whole multiples of a split."""
import types

import pytest
import torch

from swiftllm_b200 import _lib
from test_tile_edges_gpu import _ints, _normal

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lens,H,G,sbs,clustered", [
    ((700,), 32, 8, 0, True), ((700, 1, 257, 256), 8, 2, 0, True), ((300, 2000), 4, 4, 256, True), ((129, 17), 16, 1, 128, True),
    ((1000, 64, 130), 24, 3, 128, True), ((1024,), 16, 2, 128, True), ((1025,), 16, 2, 128, False), ((40,), 4, 2, 16, True),
    ((1900,) * 6, 32, 2, 256, True), ((1900,) * 7, 32, 2, 256, False)])
def test_splits_in_a_cluster(dtype, lens, H, G, sbs, clustered):
    from swiftllm_b200.worker.kernels.paged_attn import paged_attention
    B, g = len(lens), H // G
    blocks = [-(-n // 16) for n in lens]
    kc, vc = (_normal(sum(blocks), 2, G, 16, 128, seed=i, dtype=dtype) for i in (1, 2))
    table = torch.zeros(B + 1, max(blocks), dtype=torch.int32, device=DEV)
    order = torch.randperm(sum(blocks), generator=torch.Generator().manual_seed(3)).to(torch.int32).to(DEV)
    for i, n in enumerate(blocks):
        table[B - i, :n] = order[sum(blocks[:i]):sum(blocks[:i + 1])]
    q = _normal(B, H, 128, seed=4, dtype=dtype)
    st = types.SimpleNamespace(num_decoding_seqs=B, num_prefill_seqs=1, seq_ids=_ints([0] + [B - i for i in range(B)]), decoding_seq_lens=_ints(lens),
                               softmax_scale=128 ** -0.5, max_decoding_len=max(lens), paged_attn_seq_block_size=sbs)
    needed = _lib.lib().sllm_paged_attention_workspace_needed(B, H, 128, max(lens), sbs, G, 16, sum(blocks), 2)
    assert (needed == 0) == clustered and _lib.lib().sllm_paged_attention_workspace_bytes(B, H, 128, max(lens), sbs, G) > 0
    out = torch.full((B, H * 128), float("nan"), dtype=dtype, device=DEV)
    for _ in range(3):
        paged_attention(q, kc, vc, table, None, types.SimpleNamespace(block_size=16), st, 1, out)
    for i, n in enumerate(lens):
        k, v = (c[table[B - i, :blocks[i]].long(), 1].transpose(1, 2).flatten(0, 1)[:n].double().repeat_interleave(g, 1) for c in (kc, vc))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].double(), k) * 128 ** -0.5, dim=1)
        want = torch.einsum("hn,nhd->hd", p, v).flatten()
        # the output and the softmax's weights are rounded once each
        assert float((out[i].double() - want).norm() / want.norm()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11), i


@pytest.mark.parametrize("kind", ["mixed", "whole", "short", "one_long"])
@pytest.mark.parametrize("B", [31, 32, 33, 64, 65, 128, 199, 200, 201])
def test_counted_splits(B, kind):
    """Up to 200 sequences are counted, 201 are numbered; `short`: sequences without a whole split among them and at the end."""
    from swiftllm_b200.worker.kernels.paged_attn import paged_attention
    H, G, sbs, dtype = 8, 2, 256, torch.bfloat16
    some = {"mixed": (700, 256, 1, 255, 257, 512, 1024, 300), "whole": (256, 512, 1024, 768), "short": (17, 255, 900, 16, 1, 200, 3),
            "one_long": (40,)}[kind]
    lens = [some[i % len(some)] for i in range(B)]
    lens[B // 2] = 1500
    blocks = [-(-n // 16) for n in lens]
    kc, vc = (_normal(sum(blocks), 1, G, 16, 128, seed=i, dtype=dtype) for i in (1, 2))
    table = torch.zeros(B, max(blocks), dtype=torch.int32)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]))
    q = _normal(B, H, 128, seed=4, dtype=dtype)
    st = types.SimpleNamespace(num_decoding_seqs=B, num_prefill_seqs=0, seq_ids=_ints(range(B)), decoding_seq_lens=_ints(lens),
                               softmax_scale=128 ** -0.5, max_decoding_len=max(lens), paged_attn_seq_block_size=sbs)
    out = torch.full((B, H * 128), float("nan"), dtype=dtype, device=DEV)
    paged_attention(q, kc, vc, table.to(DEV), None, types.SimpleNamespace(block_size=16), st, 0, out)
    keys, values = (c[:, 0].transpose(1, 2).flatten(0, 1).double().repeat_interleave(H // G, 1) for c in (kc, vc))
    for i, n in enumerate(lens):
        at = 16 * sum(blocks[:i])
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].double(), keys[at:at + n]) * 128 ** -0.5, dim=1)
        want = torch.einsum("hn,nhd->hd", p, values[at:at + n]).flatten()
        assert float((out[i].double() - want).norm() / want.norm()) < 2.0 ** -8, i      # output and weights are rounded once each


@pytest.mark.parametrize("B,G", [(2, 2), (3, 8), (60, 2)])
def test_lengths_above_the_longest_are_cut(B, G):
    """Tokens past the launch's splits are not seen, and nothing is written past the workspace: splits in a cluster, counted splits and the
    merge, with every third length above the stated longest."""
    H, D, st_tokens, longest = 2 * G, 128, 256, 1024
    lens = [3 * longest if i % 3 == 1 else 700 + 13 * i % 300 for i in range(B)]
    blocks = 3 * longest // 16
    kc, vc = (_normal(blocks, 1, G, 16, D, seed=i, dtype=torch.bfloat16) for i in (1, 2))
    table = torch.stack([torch.randperm(blocks, generator=torch.Generator().manual_seed(i)) for i in range(B)]).to(torch.int32).to(DEV)
    q = _normal(B, H, D, seed=4, dtype=torch.bfloat16)
    ids, l = _ints(range(B)), _lib.lib()
    floats = l.sllm_paged_attention_workspace_bytes(B, H, D, longest, st_tokens, G) // 4
    outs = []
    for stated in (lens, [min(n, longest) for n in lens]):
        ws = torch.full((floats + (1 << 20),), 7.0, device=DEV)
        out, n = torch.empty(B, H * D, dtype=torch.bfloat16, device=DEV), _ints(stated)
        _lib.check(l.sllm_paged_attention(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), table.data_ptr(), ids.data_ptr(), n.data_ptr(), out.data_ptr(),
                                          ws.data_ptr(), 4 * floats, D ** -0.5, B, longest, st_tokens, 0, 1, H, G, 16, D, blocks, blocks, H * D,
                                          _lib.dtype_tag(q.dtype), _lib.stream()), "paged_attention")
        assert bool((ws[floats:] == 7.0).all())
        outs.append(out)
    assert bool(torch.isfinite(outs[0]).all()) and torch.equal(outs[0], outs[1])
