"""GPU: launches that begin before the one ahead of them has ended (csrc/common.cuh, launch_early): back to back on buffers that each call
overwrites, and replayed from a graph, they give what they give alone."""
import types

import pytest
import torch

from test_tile_edges_gpu import _ints, _normal

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _decode(seed, H=8, G=2, lens=(1900, 300, 1)):
    from swiftllm_b200.worker.kernels.paged_attn import paged_attention
    blocks = [-(-n // 16) for n in lens]
    kc, vc = (_normal(sum(blocks), 1, G, 16, 128, seed=seed + i, dtype=torch.bfloat16) for i in (0, 1))
    table = torch.zeros(len(lens), max(blocks), dtype=torch.int32, device=DEV)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]), device=DEV)
    q = _normal(len(lens), H, 128, seed=seed + 2, dtype=torch.bfloat16)
    st = types.SimpleNamespace(num_decoding_seqs=len(lens), num_prefill_seqs=0, seq_ids=_ints(range(len(lens))), decoding_seq_lens=_ints(lens),
                               softmax_scale=128 ** -0.5, max_decoding_len=max(lens), paged_attn_seq_block_size=0)
    return lambda out: paged_attention(q, kc, vc, table, None, types.SimpleNamespace(block_size=16), st, 0, out), (len(lens), H * 128)


def _window(seed, H=8, G=2, prompts=(300, 77), decodes=(900, 40, 1500)):
    from swiftllm_b200.worker.kernels.window_attn import window_attention
    rows = [(n, 0) for n in prompts] + [(1, n - 1) for n in decodes]
    T = sum(n for n, _ in rows)
    blocks = [-(-(n + p) // 16) for n, p in rows]
    table = torch.zeros(len(rows), max(blocks), dtype=torch.int32, device=DEV)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]), device=DEV)
    cache = _normal(sum(blocks), 1, 16, 2 * G * 128, seed=seed, dtype=torch.bfloat16)
    proj = _normal(T, 2 * H * 128, seed=seed + 1, dtype=torch.bfloat16)
    st = types.SimpleNamespace(num_tokens=T, num_prefill_tokens=sum(prompts), num_prefill_seqs=len(prompts), num_decoding_seqs=len(decodes),
                               token_seq_ids=_ints(i for i, (n, _) in enumerate(rows) for _ in range(n)),
                               token_positions=_ints(p + j for n, p in rows for j in range(n)), max_prefill_len=max(prompts))
    return lambda out: window_attention(proj[:, :H * 128], proj[:, H * 128:], cache, 0, table, st, out, H, G, 128, 128, 0, 512, 128 ** -0.5,
                                        True, None, None), (T, H * 128)


@pytest.mark.parametrize("make", [_decode, _window])
def test_back_to_back(make):
    calls = [make(seed) for seed in (1, 11, 21)]
    alone = []
    for call, shape in calls:
        out = torch.empty(shape, dtype=torch.bfloat16, device=DEV)
        call(out)
        torch.cuda.synchronize()
        alone.append(out)
    out, kept = torch.empty_like(alone[0]), []
    for k in range(60):                                                  # one output for all: the copy has to see the call before it
        calls[k % 3][0](out)
        kept.append(out.clone())
    for k, got in enumerate(kept):
        assert torch.equal(got, alone[k % 3]), k
    graph = torch.cuda.CUDAGraph()
    outs = [torch.empty_like(out) for _ in range(6)]
    with torch.cuda.graph(graph):
        for k in range(6):
            calls[k % 3][0](out)
            outs[k].copy_(out)
    for _ in range(3):
        for o in outs:
            o.zero_()
        graph.replay()
        for k in range(6):
            assert torch.equal(outs[k], alone[k % 3]), k
