"""GPU: launches that begin before the one ahead of them has ended (csrc/common.cuh, launch_early), or beside it: back to back on buffers
that each call overwrites, and replayed from a graph, they give what they give alone."""
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


def _stepwise_and_back_to_back(load, stages, result):
    """What `result()` is after load(k) and the stages, each waited for, against the same without a wait in between, and from a graph; the inputs
    change from round to round, in the same buffers."""
    alone = []
    for k in range(3):
        load(k)
        for stage in stages:
            torch.cuda.synchronize()
            stage()
        torch.cuda.synchronize()
        alone.append([x.clone() for x in result()])
    kept = []
    for k in range(30):
        load(k % 3)
        for stage in stages:
            stage()
        kept.append([x.clone() for x in result()])
    for k, got in enumerate(kept):
        assert all(torch.equal(a, b) for a, b in zip(got, alone[k % 3])), k
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for stage in stages:
            stage()
    for k in (0, 1, 2, 1, 0):
        load(k)
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(result(), alone[k])), k


def _mixed_window(seed, H, G, prompts, decodes, dtype=torch.bfloat16):
    """A windowed layer's step: norm of the projection, store of its keys and values, attention of prompt and decoded rows."""
    from swiftllm_b200.worker.kernels.rmsnorm import rmsnorm_inplace
    from swiftllm_b200.worker.kernels.window_attn import window_attention, window_kv_store
    rows = [(n, 700) for n in prompts] + [(1, n - 1) for n in decodes]
    T, D = sum(n for n, _ in rows), 128
    blocks = [-(-(n + p) // 16) for n, p in rows]
    table = torch.zeros(len(rows), max(blocks), dtype=torch.int32, device=DEV)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]), device=DEV)
    projs = [_normal(T, 2 * (H + G) * D, seed=seed + k, dtype=dtype) for k in range(3)]
    old = _normal(sum(blocks), 1, 16, 2 * G * D, seed=seed + 7, dtype=dtype)
    proj, cache = torch.empty_like(projs[0]), torch.empty_like(old)
    out = torch.empty(T, H * D, dtype=dtype, device=DEV)
    w = _normal(proj.shape[1], seed=seed + 8, dtype=dtype)
    st = types.SimpleNamespace(num_tokens=T, num_prefill_tokens=sum(prompts), num_prefill_seqs=len(prompts), num_decoding_seqs=len(decodes),
                               token_seq_ids=_ints(i for i, (n, _) in enumerate(rows) for _ in range(n)),
                               token_positions=_ints(p + j for n, p in rows for j in range(n)), max_prefill_len=max(prompts))
    q, gate, k, v = proj[:, :H * D], proj[:, H * D:2 * H * D], proj[:, 2 * H * D:(2 * H + G) * D], proj[:, (2 * H + G) * D:]

    def load(i):
        cache.copy_(old)
        proj.copy_(projs[i])
    stages = [lambda: rmsnorm_inplace(proj, w, 1e-5),
              lambda: window_kv_store(k, v, cache, 0, table, st, G, D, D, 0, None, None),
              lambda: window_attention(q, gate, cache, 0, table, st, out, H, G, D, D, 0, 512, D ** -0.5, True, None, None)]
    return load, stages, lambda: [out, cache]


@pytest.mark.parametrize("prompts,decodes", [((300, 77), (900, 40, 1500)), ((1,), (300,)), ((2048, 33, 700), tuple(range(1, 1200, 30)))])
def test_decoded_rows_beside_prompt_rows(prompts, decodes):
    """The attention reads rows that the launches just ahead of it wrote: the norm's, and the store's into the cache."""
    _stepwise_and_back_to_back(*_mixed_window(31, 16, 4, prompts, decodes))


def test_decoded_rows_beside_prompt_rows_from_threads():
    """Three threads on streams of their own."""
    import threading
    cases = [_mixed_window(50 + 10 * i, 8, 2, (300, 40), (900, 40, 1500)) for i in range(3)]
    want, got, errors = [], [None] * 3, []
    for load, stages, result in cases:
        load(0)
        for stage in stages:
            stage()
        torch.cuda.synchronize()
        want.append([x.clone() for x in result()])

    def work(i):
        try:
            load, stages, result = cases[i]
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for k in range(40):
                    load(k % 3)
                    for stage in stages:
                        stage()
                load(0)
                for stage in stages:
                    stage()
                got[i] = [x.clone() for x in result()]
            stream.synchronize()
        except Exception as e:                           # told to the test
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, b in zip(got, want):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
