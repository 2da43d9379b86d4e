"""GPU: paged attention of small batches whose splits meet in a cluster (csrc/paged_attn_tc.cu) against 64 bits: two to eight splits, splits
that a shorter sequence does not have, every width of a group, and the largest launch that takes the path beside the first that does not."""
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
