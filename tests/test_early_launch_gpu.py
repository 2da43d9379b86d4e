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
    """A windowed layer's step: norm of the projection, store of its keys and values, attention of prompt and decoded rows, norm of both."""
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
    w, w2 = _normal(proj.shape[1], seed=seed + 8, dtype=dtype), _normal(H * D, seed=seed + 9, dtype=dtype)
    st = types.SimpleNamespace(num_tokens=T, num_prefill_tokens=sum(prompts), num_prefill_seqs=len(prompts), num_decoding_seqs=len(decodes),
                               token_seq_ids=_ints(i for i, (n, _) in enumerate(rows) for _ in range(n)),
                               token_positions=_ints(p + j for n, p in rows for j in range(n)), max_prefill_len=max(prompts))
    q, gate, k, v = proj[:, :H * D], proj[:, H * D:2 * H * D], proj[:, 2 * H * D:(2 * H + G) * D], proj[:, (2 * H + G) * D:]

    def load(i):
        cache.copy_(old)
        proj.copy_(projs[i])
    stages = [lambda: rmsnorm_inplace(proj, w, 1e-5),
              lambda: window_kv_store(k, v, cache, 0, table, st, G, D, D, 0, None, None),
              lambda: window_attention(q, gate, cache, 0, table, st, out, H, G, D, D, 0, 512, D ** -0.5, True, None, None),
              lambda: rmsnorm_inplace(out, w2, 1e-5)]
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


def _blocks(totals):
    blocks = [-(-n // 16) for n in totals]
    table = torch.zeros(len(totals), max(blocks), dtype=torch.int32, device=DEV)
    for i, n in enumerate(blocks):
        table[i, :n] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]), device=DEV)
    return table, sum(blocks)


def test_rows_around_the_layers():
    """Gathered rows -> norm (its weight gathered just ahead of it, too) -> SiLU -> rows in front of the head -> greedy token: every kernel
    reads what the one ahead of it wrote."""
    from swiftllm_b200.worker.kernels.rmsnorm import fused_add_rmsnorm_inplace, rmsnorm_inplace
    from swiftllm_b200.worker.kernels.row_ops import add_rmsnorm_rows, argmax_rows, embed_and_zero, gather_two
    T, W, dtype = 5000, 4096, torch.bfloat16
    tables, weights = ([_normal(n, W, seed=s + k, dtype=dtype) for k in range(3)] for n, s in ((300, 1), (40, 11)))
    table, weight = torch.empty_like(tables[0]), torch.empty_like(weights[0])
    ids = (torch.arange(T, device=DEV) * 7 % 300).to(torch.int32)
    rows, picks, s = _ints([4999, 0, 17, 2500]), _ints([3, 39]), {}

    def load(k):
        table.copy_(tables[k])
        weight.copy_(weights[k])

    def norm():
        s["w"], s["w2"] = gather_two(weight, weight, picks)
        fused_add_rmsnorm_inplace(s["x"], s["r"], s["w"][0], 1e-5)

    def head():
        s["last"] = add_rmsnorm_rows(s["x"], s["r"], rows, s["w2"][1], 1e-5)
        rmsnorm_inplace(s["last"], s["w"][1], 1e-5)
        s["token"] = argmax_rows(s["last"])
    stages = [lambda: s.update(zip("xr", embed_and_zero(table, ids))), norm, lambda: _silu(s["x"]), head]
    _stepwise_and_back_to_back(load, stages, lambda: [s["x"], s["r"], s["last"], s["token"]])


def _silu(x):
    from swiftllm_b200.worker.kernels.silu_and_mul import silu_and_mul_inplace
    silu_and_mul_inplace(x)


@pytest.mark.parametrize("lens", [(700,), (1900, 300, 1), tuple(range(40, 1640, 20)), (64,) * 300])
def test_a_decoding_layer(lens):
    """Norm -> rotation and store -> paged attention (splits in a cluster, merged, none) -> norm -> greedy token."""
    from swiftllm_b200.worker.kernels.kvcache_mgmt import rotary_store_kvcache_decode
    from swiftllm_b200.worker.kernels.paged_attn import paged_attention
    from swiftllm_b200.worker.kernels.rmsnorm import rmsnorm_inplace
    from swiftllm_b200.worker.kernels.row_ops import argmax_rows, gather_two
    H, G, D, B, dtype = 8, 2, 128, len(lens), torch.bfloat16
    table, n = _blocks(lens)
    qkvs = [_normal(B, (H + 2 * G) * D, seed=k, dtype=dtype) for k in range(3)]
    old = [_normal(n, 1, G, 16, D, seed=5 + k, dtype=dtype) for k in range(2)]
    angles = [_normal(2000, D // 2, seed=8 + k, dtype=dtype) for k in range(2)]
    qkv, kc, vc = torch.empty_like(qkvs[0]), torch.empty_like(old[0]), torch.empty_like(old[1])
    w, w2 = _normal(qkv.shape[1], seed=10, dtype=dtype), _normal(H * D, seed=11, dtype=dtype)
    out, s = torch.empty(B, H * D, dtype=dtype, device=DEV), {}
    q, k, v = (x.unflatten(1, (-1, D)) for x in qkv.split([H * D, G * D, G * D], dim=1))
    st = types.SimpleNamespace(num_decoding_seqs=B, num_prefill_seqs=0, seq_ids=_ints(range(B)), decoding_seq_lens=_ints(lens),
                               softmax_scale=D ** -0.5, max_decoding_len=max(lens), paged_attn_seq_block_size=0)

    def load(i):
        qkv.copy_(qkvs[i])
        kc.copy_(old[0])
        vc.copy_(old[1])

    def turn():
        st.position_cos, st.position_sin = gather_two(angles[0], angles[1], st.decoding_seq_lens, -1)
        rotary_store_kvcache_decode(q, k, v, kc, vc, table, st, 0)

    def after():
        rmsnorm_inplace(out, w2, 1e-5)
        s["token"] = argmax_rows(out)
    stages = [lambda: rmsnorm_inplace(qkv, w, 1e-5), turn,
              lambda: paged_attention(q, kc, vc, table, None, types.SimpleNamespace(block_size=16), st, 0, out), after]
    _stepwise_and_back_to_back(load, stages, lambda: [out, kc, vc, s["token"]])


@pytest.mark.parametrize("lens,prefix", [((64,), 3000), ((300, 40, 512), 700), ((1000,) * 4, 100)])
def test_a_chunked_prompt(lens, prefix):
    """Norm of the queries -> attention over the cache (split keys and their merge, or none) -> norm."""
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention_paged
    from swiftllm_b200.worker.kernels.rmsnorm import rmsnorm_inplace
    H, G, D, T, dtype = 8, 2, 128, sum(lens), torch.float16
    table, n = _blocks([m + prefix for m in lens])
    qs = [_normal(T, H * D, seed=k, dtype=dtype) for k in range(3)]
    kc, vc = (_normal(n, 1, G, 16, D, seed=5 + k, dtype=dtype) for k in range(2))
    q, w = torch.empty_like(qs[0]), _normal(H * D, seed=10, dtype=dtype)
    out = torch.empty(T, H, D, dtype=dtype, device=DEV)
    st = types.SimpleNamespace(prefill_seq_start_locs=_ints(sum(lens[:i]) for i in range(len(lens))), prefill_seq_lens=_ints(lens),
                               softmax_scale=D ** -0.5, num_prefill_seqs=len(lens), max_prefill_len=max(lens), seq_ids=_ints(range(len(lens))),
                               prefill_prefix_lens=_ints([prefix] * len(lens)), max_prefill_kv_len=max(lens) + prefix, num_prefill_tokens=T)
    stages = [lambda: rmsnorm_inplace(q, w, 1e-5),
              lambda: prefill_attention_paged(q.view(T, H, D), kc, vc, table, out, None, types.SimpleNamespace(block_size=16), st, 0),
              lambda: rmsnorm_inplace(out.view(T, H * D), w, 1e-5)]
    _stepwise_and_back_to_back(lambda k: q.copy_(qs[k]), stages, lambda: [out])


@pytest.mark.parametrize("prompts,decodes", [((), (2000, 300, 40)), ((40,), ()), ((33, 33, 33), (900,)), ((800,), ()), ((), (500,) * 64)])
def test_a_latent_layer(prompts, decodes):
    """Norm of queries and gate -> store of the latent rows -> attention (splits and their merge, shared CTAs, none) -> norm."""
    from swiftllm_b200.worker.kernels.latent_attn import latent_attention, latent_kv_store
    from swiftllm_b200.worker.kernels.rmsnorm import rmsnorm_inplace
    H, r, dr, dtype = 16, 512, 64, torch.bfloat16
    steps = [(n, 300) for n in prompts] + [(1, n - 1) for n in decodes]
    T = sum(n for n, _ in steps)
    table, n = _blocks([a + b for a, b in steps])
    width = H * (r + dr) + H + 8 + r + dr                                # queries | gates | the new row
    projs = [_normal(T, width, seed=k, dtype=dtype) for k in range(3)]
    old = _normal(n, 1, 16, r + dr, seed=5, dtype=dtype)
    proj, cache, w = torch.empty_like(projs[0]), torch.empty_like(old), _normal(width, seed=6, dtype=dtype)
    nw, w2 = _normal(r, seed=7, dtype=dtype), _normal(H * r, seed=8, dtype=dtype)
    out = torch.empty(T, H, r, dtype=dtype, device=DEV)
    st = types.SimpleNamespace(num_tokens=T, num_prefill_tokens=sum(prompts), num_prefill_seqs=len(prompts), num_decoding_seqs=len(decodes),
                               token_seq_ids=_ints(i for i, (a, _) in enumerate(steps) for _ in range(a)),
                               token_positions=_ints(b + j for a, b in steps for j in range(a)))
    q = proj[:, :H * (r + dr)].unflatten(1, (H, r + dr))
    gate, row = proj[:, H * (r + dr):H * (r + dr) + H], proj[:, H * (r + dr) + H + 8:]

    def load(k):
        proj.copy_(projs[k])
        cache.copy_(old)
    stages = [lambda: rmsnorm_inplace(proj, w, 1e-5),
              lambda: latent_kv_store(row, nw, cache, 0, table, st, r, dr, 0, 1e-5, None, None),
              lambda: latent_attention(q[:, :, :r], q[:, :, r:], gate, cache, 0, table, st, out, 0, 0, (r + dr) ** -0.5, None, None),
              lambda: rmsnorm_inplace(out.view(T, H * r), w2, 1e-5)]
    _stepwise_and_back_to_back(load, stages, lambda: [out, cache])


def _prompts(seed, H=32, G=8, lens=(900, 333, 700)):
    from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention
    T = sum(lens)
    qkv = _normal(T, (H + 2 * G) * 128, seed=seed, dtype=torch.bfloat16)
    q, k, v = (x.unflatten(1, (-1, 128)) for x in qkv.split([H * 128, G * 128, G * 128], dim=1))
    st = types.SimpleNamespace(prefill_seq_start_locs=_ints(sum(lens[:i]) for i in range(len(lens))), prefill_seq_lens=_ints(lens), softmax_scale=128 ** -0.5,
                               num_prefill_seqs=len(lens), max_prefill_len=max(lens))
    return lambda out: prefill_attention(q, k, v, out, None, None, st), (T, H, 128)


def _latent_prompts(seed, H=16, n=1700):
    from tile_cases import latent_case
    from swiftllm_b200.worker.kernels.latent_attn import latent_attention
    c = latent_case(torch.bfloat16, [(n, seed)], [], H, 512, 64, 64, 0, sink=True)
    return lambda out: latent_attention(c.q, c.qr, c.gate, c.cache, 1, c.bt, c.st, out, c.dims, 0, c.scale, c.cos, c.sin, c.sink), (n, H, 512)


@pytest.mark.parametrize("make", [_prompts, _latent_prompts])
def test_ctas_that_take_others_back_to_back(make):
    """Grids of more CTAs than SMs, whose CTAs take the next one's place: the launch behind them begins when none is left."""
    test_back_to_back(make)
