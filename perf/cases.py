"""The work that is timed: what a program that serves models with this package has it do, through the package's public entry points.

Every case is a dict of plain values.  `kind` names the entry point; the rest are sizes, storage types and options:

  decode   paged attention of one new token per sequence (Llama worker)
  prefill  causal attention over packed prompts (Llama worker)
  chunk    attention of prompt portions over the paged cache (Llama worker, chunked prompts beside running decodes)
  window   windowed attention with grouped or shared key/value heads, prompt portions and decoded tokens in one step
  latent   latent attention, prompt portions or decoded tokens
  delta, gla   recurrences with a matrix state per head
  scan     short convolution and selective scan of a state-space layer
  llama    a whole decode step of the Llama worker, host lists in, tokens and logits out

Sizes are those of the package's own configurations: Llama-3-8B / 70B heads, and the width-2048 / width-4096 layer shapes of the
other families (16 / 32 heads, a quarter as many key/value heads, 128 entries per head, 512 + 64 latent entries, windows of 1024 /
2048, 128 x 128 states, 16 states per scanned channel, blocks of 16 tokens)."""
import math
from types import SimpleNamespace

import torch

from swiftllm_b200 import EngineConfig, LlamaModel
from swiftllm_b200.model_config import LLAMA3_8B, LlamaModelConfig
from swiftllm_b200.worker.infer_state import LlamaInferState, TokenInferState
from swiftllm_b200.worker.kernels.gla import gated_linear_attention
from swiftllm_b200.worker.kernels.head_decay import delta_rule
from swiftllm_b200.worker.kernels.latent_attn import latent_attention
from swiftllm_b200.worker.kernels.paged_attn import paged_attention
from swiftllm_b200.worker.kernels.prefill_attn import prefill_attention, prefill_attention_paged
from swiftllm_b200.worker.kernels.scan_ops import selective_scan, short_conv
from swiftllm_b200.worker.kernels.window_attn import AttnOptions, shared_row_width, window_attention

BLOCK = 16              # tokens of a cache block: the package's default
DIM = 128               # entries of an attention head
LATENT, LATENT_ROT = 512, 64
KEEP_FIRST = 4
EPS = 1e-5
GLA_TAU = 16.0
SCAN_STATES, SCAN_TAPS = 16, 4
LLAMA_LAYERS = 2

_TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one user's chat: a single short sequence, all of it latency
        dict(name="decode_single", kind="decode", dtype="bf16", heads=32, kv_heads=8, batch=1, longest=700, ragged=False),
        # a server's ordinary step: sequences of many lengths, half precision as the reference ships it
        dict(name="decode_ragged", kind="decode", dtype="fp16", heads=32, kv_heads=8, batch=48, longest=6000, ragged=True),
        # the headline: 256 sequences of 4096 tokens, one layer of Llama-3-8B
        dict(name="decode_full", kind="decode", dtype="bf16", heads=32, kv_heads=8, batch=256, longest=4096, ragged=False),
        # whole long prompts, one layer of Llama-3-8B
        dict(name="prefill_long", kind="prefill", dtype="bf16", heads=32, kv_heads=8, batch=4, longest=4096, ragged=False),
        # prompts as they arrive: a dozen, from a few tokens to a page of text
        dict(name="prefill_ragged", kind="prefill", dtype="fp16", heads=32, kv_heads=8, batch=12, longest=1777, ragged=True),
        # a 512-token portion of a long prompt, as it rides beside running decodes
        dict(name="chunk", kind="chunk", dtype="bf16", heads=32, kv_heads=8, batch=1, longest=512, prefix=3584, ragged=False),
        # a mixed step of a windowed layer: three prompts of different lengths and forty running sequences
        dict(name="window_mixed", kind="window", dtype="bf16", design="grouped", heads=16, kv_heads=4, window=1024, batch=3,
             longest=2048, prefix=0, ragged=True, decodes=40, context=2048),
        # prompts through a latent-attention layer without a window
        dict(name="latent_prompt", kind="latent", dtype="bf16", heads=16, window=0, batch=4, longest=2048, prefix=0, ragged=False,
             decodes=0, context=0),
        # 64 running sequences through the same layer
        dict(name="latent_decode", kind="latent", dtype="bf16", heads=16, window=0, batch=0, longest=0, prefix=0, ragged=False,
             decodes=64, context=2048),
        # prompts through a gated-delta-rule layer
        dict(name="delta_prompt", kind="delta", dtype="bf16", heads=16, batch=4, longest=2048, ragged=False),
        # prompts through a state-space layer: convolution and scan between its projections
        dict(name="scan_prompt", kind="scan", dtype="bf16", channels=4096, batch=4, longest=2048, ragged=False),
        # a whole decode step of a Llama-3-8B-shaped model with two layers, sixteen sequences
        dict(name="llama_step", kind="llama", dtype="bf16", batch=16, longest=1500, ragged=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "chunk", "window", "window", "latent", "latent", "delta", "gla", "scan",
                       "llama"])
    c = dict(kind=kind, dtype=rng.choice(["bf16", "fp16"]), ragged=rng.random() < 0.7)
    if kind == "decode":
        c["heads"], c["kv_heads"] = rng.choice([(32, 8), (64, 8), (16, 4)])
        c["longest"] = _log(rng, 16, 8192)
        c["batch"] = _log(rng, 1, min(256, 500000 // c["longest"]))
    elif kind == "prefill":
        c["heads"], c["kv_heads"] = rng.choice([(32, 8), (64, 8), (16, 4)])
        c["longest"] = _log(rng, 16, 4096)
        c["batch"] = _log(rng, 1, max(1, min(64, 8192 // c["longest"])))
    elif kind == "chunk":
        c["heads"], c["kv_heads"] = rng.choice([(32, 8), (64, 8), (16, 4)])
        c["longest"], c["prefix"] = _log(rng, 16, 1024), rng.randrange(1, 6000)
        c["batch"] = rng.randrange(1, 5)
    elif kind in ("window", "latent"):
        big = rng.random() < 0.4
        c["heads"] = 32 if big else 16
        c["window"] = (2048 if big else 1024) if kind == "window" or rng.random() < 0.4 else 0
        c["batch"], c["longest"] = rng.randrange(0, 4), _log(rng, 32, 2048)
        c["prefix"] = rng.randrange(0, 2000) if rng.random() < 0.4 else 0
        c["decodes"] = _log(rng, 1, 64) if c["batch"] == 0 or rng.random() < 0.6 else 0
        c["context"] = _log(rng, 32, 4096)
        if kind == "window":
            c["kv_heads"] = c["heads"] // 4
            c["design"] = rng.choice(["grouped", "shared"])
    elif kind in ("delta", "gla"):
        c["heads"] = rng.choice([16, 32])
        c["longest"] = _log(rng, 32, 2048)
        c["batch"] = rng.randrange(1, 4)
    elif kind == "scan":
        c["channels"] = rng.choice([4096, 8192])
        c["longest"] = _log(rng, 32, 2048)
        c["batch"] = rng.randrange(1, 4)
    else:
        c["batch"], c["longest"] = _log(rng, 1, 64), _log(rng, 16, 2000)
    return c


# ---------------------------------------------------------------------------------------------------------------- shapes
def _lens(n, longest, ragged):
    """n lengths of at most `longest`: all equal, or spread over the range with `longest` among them."""
    if not ragged:
        return [longest] * n
    return [longest] + [max(1, round(longest * ((0.5 + 0.6180339887 * i) % 1.0))) for i in range(1, n)]


def _step(c):
    """(tokens, position of the first) of every sequence of a step: prompt portions, then one row per running sequence."""
    portions = [(n, c.get("prefix", 0)) for n in _lens(c["batch"], c["longest"], c["ragged"])]
    running = [(1, n - 1) for n in _lens(c.get("decodes", 0), c.get("context", 0), c["ragged"])]
    return portions, running


def _pairs(n, first, window=0):
    """Visible (query, key) pairs of n queries at positions first ..; a window also bounds each query's keys."""
    if window <= 0:
        return n * first + n * (n + 1) // 2
    return sum(min(window, p + 1) for p in range(first, first + n))


def work(c):
    kind = c["kind"]
    if kind == "decode":
        lens = _lens(c["batch"], c["longest"], c["ragged"])
        return dict(bytes=2 * (sum(lens) * c["kv_heads"] * DIM * 2 + 2 * len(lens) * c["heads"] * DIM),
                    flops=4 * c["heads"] * DIM * sum(lens))
    if kind in ("prefill", "chunk"):
        first = c.get("prefix", 0)
        lens = _lens(c["batch"], c["longest"], c["ragged"])
        kv = sum(n + first for n in lens)
        return dict(bytes=2 * (2 * sum(lens) * c["heads"] * DIM + 2 * kv * c["kv_heads"] * DIM),
                    flops=4 * c["heads"] * DIM * sum(_pairs(n, first) for n in lens))
    if kind in ("window", "latent"):
        portions, running = _step(c)
        rows = portions + running
        T = sum(n for n, _ in rows)
        pairs = sum(_pairs(n, p, c["window"]) for n, p in rows)
        seen = sum(n + (p if c["window"] <= 0 else min(p, c["window"])) for n, p in rows)
        if kind == "latent":
            return dict(bytes=2 * (seen * (LATENT + LATENT_ROT) + T * c["heads"] * (2 * LATENT + LATENT_ROT)),
                        flops=2 * c["heads"] * (2 * LATENT + LATENT_ROT) * pairs)
        keys = c["kv_heads"] * DIM * (2 if c["design"] == "grouped" else 1)
        gate = c["heads"] * (DIM if c["design"] == "grouped" else 1)
        return dict(bytes=2 * (seen * keys + T * (2 * c["heads"] * DIM + gate)), flops=4 * c["heads"] * DIM * pairs)
    T = sum(_lens(c["batch"], c["longest"], c["ragged"]))
    if kind == "delta":
        H = c["heads"]
        return dict(bytes=T * (2 * (2 * (H // 2) * DIM + 3 * H * DIM) + 8 * H) + 4 * c["batch"] * H * DIM * DIM,
                    flops=T * H * DIM * DIM * 7)
    if kind == "gla":
        H = c["heads"]
        return dict(bytes=T * H * DIM * (2 * 5 + 4) + 4 * c["batch"] * H * DIM * DIM, flops=T * H * DIM * DIM * 5)
    if kind == "scan":
        C, N = c["channels"], SCAN_STATES
        return dict(bytes=T * C * (2 + 2 + 4 + 2 + 2 + 2) + T * 4 * N + c["batch"] * C * (4 * N + 2 * (SCAN_TAPS - 1)),
                    flops=T * C * (2 * SCAN_TAPS + 7 * N))
    m = LLAMA3_8B
    W, F, V = m["hidden_size"], m["intermediate_size"], m["vocab_size"]
    kv = m["num_key_value_heads"] * DIM
    B = c["batch"]
    lens = _lens(B, c["longest"], c["ragged"])
    weights = LLAMA_LAYERS * (2 * W * W + 2 * W * kv + 3 * W * F) + V * W
    return dict(bytes=2 * (weights + LLAMA_LAYERS * sum(lens) * 2 * kv + B * (W + V)),
                flops=2 * B * weights + LLAMA_LAYERS * 4 * W * sum(lens))


def tolerance(c):
    """About four times what these cases differ from 64 bits: outputs are rounded once to 16 bits, as are the softmax's weights."""
    if c["kind"] == "llama":
        return {"rel": 2.5e-2 if c["dtype"] == "bf16" else 3e-3}
    return {"rel": 9e-3 if c["dtype"] == "bf16" else 1.2e-3}


# ---------------------------------------------------------------------------------------------------------------- inputs
class _Maker:
    """Tensors from a seed, in the order they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32, std=1.0, mean=0.0):
        if math.prod(shape) > 1 << 28:                   # a large cache is made in place, in its own type
            return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=self.gen)
        return (torch.randn(shape, generator=self.gen, device="cuda") * std + mean).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=self.gen, device="cuda") * (hi - lo) + lo

    def order(self, n):
        return torch.randperm(n, generator=self.gen, device="cuda").to(torch.int32)


def _ints(values):
    return torch.tensor(list(values), dtype=torch.int32, device="cuda")


def _block_table(make, totals):
    """A table whose rows hold the blocks of sequences of the given total lengths, in no order; -> (table, number of blocks)."""
    blocks = [-(-n // BLOCK) for n in totals]
    ids = make.order(sum(blocks)).split(blocks)
    table = torch.zeros((len(totals), max(blocks)), dtype=torch.int32, device="cuda")
    for row, mine in zip(table, ids):
        row[:mine.shape[0]] = mine
    return table, sum(blocks)


def _llama_state(c, lens, totals, running):
    """Metadata of a step of `lens` prompt rows each, or of one decoded token per sequence (`running`)."""
    empty = _ints([])
    starts = [sum(lens[:i]) for i in range(len(lens))]
    none = torch.empty((0,), device="cuda")
    chunked = not running and c.get("prefix", 0) > 0
    return LlamaInferState(
        batch_size=len(lens), seq_ids=_ints(range(len(lens))), num_tokens=len(lens) if running else sum(lens),
        softmax_scale=DIM ** -0.5, num_prefill_seqs=0 if running else len(lens), num_prefill_tokens=0 if running else sum(lens),
        prefill_seq_start_locs=empty if running else _ints(starts),
        prefill_seq_start_locs_with_end=empty if running else _ints(starts + [sum(lens)]),
        prefill_seq_lens=empty if running else _ints(lens), max_prefill_len=0 if running else max(lens),
        num_decoding_seqs=len(lens) if running else 0, decoding_seq_lens=_ints(lens) if running else empty,
        max_decoding_len=max(lens) if running else 0, seq_block_size=2048, num_seq_blocks=(max(lens) + 2047) // 2048 if running else 0,
        position_cos=none, position_sin=none, ignore_kvcache=False,
        prefill_prefix_lens=_ints([c["prefix"]] * len(lens)) if chunked else None, max_prefill_kv_len=max(totals) if chunked else 0)


def _token_state(portions, running):
    rows = portions + running
    seqs = [i for i, (n, _) in enumerate(rows) for _ in range(n)]
    places = [p + j for n, p in rows for j in range(n)]
    ends, at = [0], 0
    for n, _ in rows:
        at += n
        ends.append(at)
    return TokenInferState(
        batch_size=len(rows), num_tokens=at, seq_ids=_ints(range(len(rows))), num_prefill_seqs=len(portions), num_decoding_seqs=len(running),
        num_prefill_tokens=sum(n for n, _ in portions), token_seq_ids=_ints(seqs), token_positions=_ints(places),
        output_rows=_ints(e - 1 for e in ends[1:]), max_prefill_len=max([n for n, _ in portions], default=0), seg_starts=_ints(ends))


def _angles(places, dims, base=10000.0):
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device="cuda")
    a = places.double()[:, None] * f[None, :]
    return a.cos().float().contiguous(), a.sin().float().contiguous()


def _inputs(c, seed):
    """The tensors of a case, by name: what both `run` and `exact` start from."""
    make, t, kind = _Maker(seed), _TYPES[c["dtype"]], c["kind"]
    i = SimpleNamespace()
    if kind in ("decode", "prefill", "chunk"):
        H, G = c["heads"], c["kv_heads"]
        i.lens = _lens(c["batch"], c["longest"], c["ragged"])
        i.totals = [n + c.get("prefix", 0) for n in i.lens]
        i.st = _llama_state(c, i.lens, i.totals, kind == "decode")
        rows = len(i.lens) if kind == "decode" else sum(i.lens)
        if kind == "prefill":                            # q, k and v are column slices of one projection, as in the worker
            qkv = make.normal(rows, (H + 2 * G) * DIM, dtype=t)
            i.q, i.k, i.v = (x.unflatten(1, (-1, DIM)) for x in qkv.split([H * DIM, G * DIM, G * DIM], dim=1))
        else:
            i.q = make.normal(rows, (H + 2 * G) * DIM, dtype=t)[:, :H * DIM].unflatten(1, (H, DIM))
            i.table, n = _block_table(make, i.totals)
            i.kc, i.vc = (make.normal(n, 1, G, BLOCK, DIM, dtype=t) for _ in range(2))
        return i
    if kind in ("window", "latent"):
        H = c["heads"]
        i.portions, i.running = _step(c)
        i.rows = i.portions + i.running
        i.st = _token_state(i.portions, i.running)
        T = i.st.num_tokens
        i.table, n = _block_table(make, [k + p for k, p in i.rows])
        if kind == "latent":
            i.q = make.normal(T, H, LATENT, dtype=t)
            i.q_rot = make.normal(T, H, DIM + LATENT_ROT, dtype=t)[:, :, DIM:]
            i.cache = make.normal(n, 1, BLOCK, LATENT + LATENT_ROT, dtype=t)
            i.sink = make.normal(H) if c["window"] == 0 else None
            i.gate = make.normal(T, H, dtype=t) if c["window"] > 0 else None
            i.cos, i.sin = _angles(i.st.token_positions, LATENT_ROT)
            return i
        G = c["kv_heads"]
        if c["design"] == "grouped":
            proj = make.normal(T, (2 * H + 2 * G) * DIM, dtype=t)
            i.q, i.gate = proj[:, :H * DIM], proj[:, (H + 2 * G) * DIM:]
            i.cache = make.normal(n, 1, BLOCK, 2 * G * DIM, dtype=t)
            i.cos, i.sin = _angles(i.st.token_positions, DIM // 2)
        else:
            proj = make.normal(T, (H + G) * DIM + H, dtype=t)
            i.q, i.gate = proj[:, :H * DIM], proj[:, (H + G) * DIM:]
            keys = make.normal(n, 1, BLOCK, G * DIM, dtype=t)
            off = (2 * G + 7) // 8 * 8
            i.cache = torch.zeros((n, 1, BLOCK, shared_row_width(G, DIM)), dtype=t, device="cuda")
            i.cache[..., off:] = keys
            inv = (keys.float().unflatten(3, (G, DIM)).square().mean(4) + EPS).rsqrt()
            i.cache[..., :2 * G] = inv.contiguous().view(t).view(n, 1, BLOCK, 2 * G)
            i.norm = make.normal(DIM, std=0.1, mean=1.0)
            i.slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)], device="cuda")
        return i
    if kind in ("delta", "gla", "scan"):
        lens = _lens(c["batch"], c["longest"], c["ragged"])
        i.lens, i.st = lens, _token_state([(n, 0) for n in lens], [])
        T = sum(lens)
        if kind == "scan":
            C, N = c["channels"], SCAN_STATES
            i.xz = make.normal(T, 2 * C, dtype=t)
            i.taps, i.taps_b = make.normal(C, SCAN_TAPS, std=0.4), make.normal(C, std=0.1)
            i.tail = torch.zeros((len(lens), SCAN_TAPS - 1, C), dtype=t, device="cuda")
            i.dt, i.dt_b = make.normal(T, C, std=0.5), make.uniform(C, lo=-5.0, hi=-2.0)
            i.A = -torch.arange(1, N + 1, device="cuda", dtype=torch.float32).repeat(C, 1) * make.uniform(C, N, lo=0.8, hi=1.2)
            i.bc = make.normal(T, 2 * N + C // 32, dtype=t)
            i.D = make.normal(C, std=0.1, mean=1.0)
            i.state = torch.zeros((len(lens), C, N), device="cuda")
            return i
        H = c["heads"]
        G = H // 2 if kind == "delta" else H
        if kind == "delta":                              # q, k and v leave one convolution; gate is a slice of the projection
            qkv = torch.nn.functional.silu(make.normal(T, (2 * G + H) * DIM)).to(t)
            i.q, i.k, i.v = qkv.split([G * DIM, G * DIM, H * DIM], dim=1)
            i.gate = make.normal(T, (2 * G + 2 * H) * DIM, dtype=t)[:, (2 * G + H) * DIM:]
            i.z = make.normal(T, 2 * H)
            i.bias, i.rate = make.uniform(H, lo=-5.0, hi=-2.0), make.uniform(H, lo=1.0, hi=8.0)
        else:
            proj = make.normal(T, 4 * H * DIM, dtype=t)
            i.q, i.k, i.v, i.gate = proj.split([H * DIM] * 4, dim=1)
            i.z, i.bias = make.normal(T, H * DIM), make.normal(H * DIM, std=0.5)
        i.norm = make.normal(DIM, std=0.1, mean=1.0)
        i.state = torch.zeros((len(lens), H, DIM, DIM), device="cuda")
        return i
    i.lens = _lens(c["batch"], c["longest"], c["ragged"])
    i.config = dict(LLAMA3_8B, num_hidden_layers=LLAMA_LAYERS)
    i.weights = {}
    W, F, V, kv = i.config["hidden_size"], i.config["intermediate_size"], i.config["vocab_size"], i.config["num_key_value_heads"] * DIM
    for name in ("model.embed_tokens", "lm_head"):
        i.weights[name + ".weight"] = make.normal(V, W, dtype=t, std=1.0 if name != "lm_head" else W ** -0.5)
    i.weights["model.norm.weight"] = make.normal(W, dtype=t, std=0.1, mean=1.0)
    for n in range(LLAMA_LAYERS):
        for name, shape in (("self_attn.q_proj", (W, W)), ("self_attn.k_proj", (kv, W)), ("self_attn.v_proj", (kv, W)),
                            ("self_attn.o_proj", (W, W)), ("mlp.up_proj", (F, W)), ("mlp.gate_proj", (F, W)), ("mlp.down_proj", (W, F))):
            i.weights[f"model.layers.{n}.{name}.weight"] = make.normal(*shape, dtype=t, std=shape[1] ** -0.5)
        for name in ("input_layernorm", "post_attention_layernorm"):
            i.weights[f"model.layers.{n}.{name}.weight"] = make.normal(W, dtype=t, std=0.1, mean=1.0)
    blocks = [-(-n // BLOCK) for n in i.lens]
    i.blocks = sum(blocks)
    # keys and values of the tokens before the new one, by sequence; the worker hands out blocks in ascending order
    i.kc, i.vc = (make.normal(i.blocks, LLAMA_LAYERS, kv // DIM, BLOCK, DIM, dtype=t) for _ in range(2))
    i.ids = torch.randint(0, V, (len(i.lens),), generator=make.gen, device="cuda").tolist()
    return i


def prepare(case, seed):
    c, i = case, _inputs(case, seed)
    kind = c["kind"]
    s = SimpleNamespace(c=c, i=i)
    if kind == "decode":
        s.out = torch.empty((c["batch"], c["heads"] * DIM), dtype=i.q.dtype, device="cuda")
    elif kind in ("prefill", "chunk"):
        s.out = torch.empty(i.q.shape, dtype=i.q.dtype, device="cuda")
    elif kind == "window":
        s.out = torch.empty((i.st.num_tokens, c["heads"] * DIM), dtype=i.q.dtype, device="cuda")
        if c["design"] == "shared":
            s.options = AttnOptions(q_norm=i.norm, prenorm_eps=EPS, slopes=i.slopes, keep_first=KEEP_FIRST, gate_per_head=True,
                                    shared_kv=True)
    elif kind == "latent":
        s.out = torch.empty((i.st.num_tokens, c["heads"], LATENT), dtype=i.q.dtype, device="cuda")
    elif kind == "llama":
        config = LlamaModelConfig(i.config)
        ec = EngineConfig(model_path="", use_dummy=False, block_size=BLOCK, gpu_mem_utilization=0.9, num_cpu_blocks=0,
                          max_seqs_in_block_table=64, max_blocks_per_seq=512, max_batch_size=64, max_tokens_in_batch=4096,
                          dtype={"bf16": "bfloat16", "fp16": "float16"}[c["dtype"]], use_cuda_graph=True)
        s.model = LlamaModel(ec, config)
        s.model.load_weights(lambda key, shape, dtype: i.weights[key])
        s.model.init_kvcache_and_swap(i.blocks)
        s.model.post_layer.keep_logits = True
        s.seqs = list(range(c["batch"]))
        for seq, n in zip(s.seqs, i.lens):               # the sequences' blocks, one sequence after the other
            s.model.gpu_block_manager.allocate_blocks_for_seqs(_ints([seq]), _ints([n]), seq_ids_list=[seq], target_lens_list=[n],
                                                               want_new_blocks=False)
        with torch.inference_mode():                     # the caches are tensors of the model's own inference mode
            s.model.k_cache.copy_(i.kc)
            s.model.v_cache.copy_(i.vc)
        i.kc = i.vc = i.weights = None
        s.tokens = [[t] for t in i.ids]
        s.model.forward(s.tokens, s.seqs, i.lens)        # a server captures the step of a batch size before it takes requests
    return s


def run(state):
    s, c, i = state, state.c, state.i
    kind = c["kind"]
    ec = SimpleNamespace(block_size=BLOCK)
    if kind == "decode":
        paged_attention(i.q, i.kc, i.vc, i.table, None, ec, i.st, 0, s.out)
        return s.out
    if kind == "prefill":
        prefill_attention(i.q, i.k, i.v, s.out, None, ec, i.st)
        return s.out
    if kind == "chunk":
        prefill_attention_paged(i.q, i.kc, i.vc, i.table, s.out, None, ec, i.st, 0)
        return s.out
    if kind == "window":
        H, G = c["heads"], c["kv_heads"]
        if c["design"] == "grouped":
            window_attention(i.q, i.gate, i.cache, 0, i.table, i.st, s.out, H, G, DIM, DIM, DIM // 2, c["window"], DIM ** -0.5, True,
                             i.cos, i.sin)
        else:
            window_attention(i.q, i.gate, i.cache, 0, i.table, i.st, s.out, H, G, DIM, DIM, 0, c["window"], DIM ** -0.5, False, None,
                             None, s.options)
        return s.out
    if kind == "latent":
        latent_attention(i.q, i.q_rot, i.gate, i.cache, 0, i.table, i.st, s.out, LATENT_ROT, c["window"], (DIM + LATENT_ROT) ** -0.5,
                         i.cos, i.sin, i.sink)
        return s.out
    if kind == "delta":
        H = c["heads"]
        y = delta_rule(i.q, i.k, i.v, i.z[:, H:], i.z[:, :H], i.bias, i.rate, i.norm, EPS, i.gate, i.state, i.st, H, H // 2, DIM, DIM)
        return y, i.state
    if kind == "gla":
        y = gated_linear_attention(i.q, i.k, i.v, i.z, i.bias, GLA_TAU, i.norm, EPS, i.gate, i.state, i.st, c["heads"], DIM, DIM)
        return y, i.state
    if kind == "scan":
        C, N = c["channels"], SCAN_STATES
        x = short_conv(i.xz[:, :C], i.taps, i.taps_b, i.tail, i.st, i.xz.dtype, silu=True, move_tail=True)
        y = selective_scan(x, i.dt, i.dt_b, i.A, i.bc, C // 32, C // 32 + N, i.D, i.xz[:, C:], i.state, i.st)
        return x, y, i.state, i.tail
    tokens = s.model.forward_async(s.tokens, s.seqs, i.lens)
    return s.model.post_layer.last_logits, tokens


# ---------------------------------------------------------------------------------------------------------------- in 64 bits
def _rows_of(cache, table_row, n):
    """The first n cache rows of a sequence, in order: [n, ...] of a cache [blocks, 1, BLOCK, ...]."""
    ids = table_row[:-(-n // BLOCK)].long()
    return cache[ids, 0].flatten(0, 1)[:n]


def _turn(x, cos, sin):
    """Neighbouring pairs of the last axis turned; cos, sin broadcast over it."""
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * cos - b * sin, b * cos + a * sin), dim=-1).flatten(-2)


def _attend(q, k, v, first, window=0, keep=0, scale=1.0, sink=None, bias=None):
    """q [n, H, d] at positions first .., k [L, H, d], v [L, H, e] -> [n, H, e]; sink: score of a key without a value, per head."""
    out = []
    L = k.shape[0]
    kp = torch.arange(L, device=q.device)
    step = max(1, (1 << 27) // (L * q.shape[1]))
    kt, vt = k.permute(1, 2, 0), v.transpose(0, 1)
    for at in range(0, q.shape[0], step):
        x = q[at:at + step]
        qp = torch.arange(first + at, first + at + x.shape[0], device=q.device)[:, None]
        seen = kp[None, :] <= qp
        if window > 0:
            seen &= (qp - kp[None, :] < window) | (kp[None, :] < keep)
        sc = torch.matmul(x.transpose(0, 1), kt) * scale                     # [H, n, L]
        if bias is not None:
            sc = sc - bias[:, None, None] * (qp - kp[None, :])[None].double()
        sc = sc.masked_fill(~seen[None], float("-inf"))
        if sink is not None:
            sc = torch.cat((sc, sink[:, None, None].expand(-1, x.shape[0], 1)), dim=2)
        p = torch.softmax(sc, dim=2)[:, :, :L]
        out.append(torch.matmul(p, vt).transpose(0, 1))
    return torch.cat(out)


def _exact_llama(c, i):
    m = i.config
    H, G, W = m["num_attention_heads"], m["num_key_value_heads"], m["hidden_size"]
    w = lambda key: i.weights[key + ".weight"].double()

    def norm(x, key):
        return x / (x.square().mean(1, keepdim=True) + m["rms_norm_eps"]).sqrt() * w(key)
    places = torch.tensor([n - 1 for n in i.lens], dtype=torch.float64, device="cuda")
    f = torch.tensor([m["rope_theta"] ** (-2.0 * j / DIM) for j in range(DIM // 2)], dtype=torch.float64, device="cuda")
    ang = places[:, None] * f
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def turn(x):
        a, b = x[..., :DIM // 2], x[..., DIM // 2:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)
    x = w("model.embed_tokens")[torch.tensor(i.ids, device="cuda")]
    for n in range(LLAMA_LAYERS):
        at = f"model.layers.{n}."
        h = norm(x, at + "input_layernorm")
        q = turn((h @ w(at + "self_attn.q_proj").t()).unflatten(1, (H, DIM)))
        k = turn((h @ w(at + "self_attn.k_proj").t()).unflatten(1, (G, DIM)))
        v = (h @ w(at + "self_attn.v_proj").t()).unflatten(1, (G, DIM))
        out, block = [], 0
        for s, total in enumerate(i.lens):
            nb = -(-total // BLOCK)
            kk, vv = (cache[block:block + nb, n].transpose(1, 2).flatten(0, 1)[:total].double() for cache in (i.kc, i.vc))
            block += nb
            kk[-1], vv[-1] = k[s], v[s]
            out.append(_attend(q[s:s + 1], kk.repeat_interleave(H // G, 1), vv.repeat_interleave(H // G, 1), total - 1, scale=DIM ** -0.5))
        x = x + torch.cat(out).flatten(1) @ w(at + "self_attn.o_proj").t()
        h = norm(x, at + "post_attention_layernorm")
        x = x + (torch.nn.functional.silu(h @ w(at + "mlp.gate_proj").t()) * (h @ w(at + "mlp.up_proj").t())) @ w(at + "mlp.down_proj").t()
    return norm(x, "model.norm") @ w("lm_head").t(), None


def exact(case, seed):
    c, kind = case, case["kind"]
    i = _inputs(c, seed)
    if kind == "llama":
        return _exact_llama(c, i)
    if kind in ("decode", "prefill", "chunk"):
        H, G = c["heads"], c["kv_heads"]
        out, at = [], 0
        for s, (n, total) in enumerate(zip(i.lens, i.totals)):
            if kind == "prefill":
                q, k, v = (x[at:at + n].double() for x in (i.q, i.k, i.v))
                at += n
            else:
                rows = 1 if kind == "decode" else n
                q = i.q[at:at + rows].double()
                at += rows
                k, v = (cache[i.table[s, :-(-total // BLOCK)].long(), 0].transpose(1, 2).flatten(0, 1)[:total].double()
                        for cache in (i.kc, i.vc))
            g = H // G
            parts = [_attend(q[:, j * g:(j + 1) * g], k[:, j:j + 1].expand(-1, g, -1), v[:, j:j + 1].expand(-1, g, -1),
                             total - q.shape[0], scale=DIM ** -0.5) for j in range(G)]
            out.append(torch.cat(parts, dim=1))
        out = torch.cat(out)
        return out.flatten(1) if kind == "decode" else out
    if kind in ("window", "latent"):
        H, out, at = c["heads"], [], 0
        for s, (n, first) in enumerate(i.rows):
            mine = slice(at, at + n)
            at += n
            rows = _rows_of(i.cache, i.table[s], first + n)
            if kind == "latent":
                cos, sin = (x[mine].double()[:, None] for x in (i.cos, i.sin))
                q = torch.cat((i.q[mine].double(), _turn(i.q_rot[mine].double(), cos, sin)), dim=2)
                k = rows.double()[:, None].expand(-1, H, -1)
                o = _attend(q, k, k[:, :, :LATENT], first, c["window"], scale=(DIM + LATENT_ROT) ** -0.5,
                            sink=None if i.sink is None else i.sink.double())
                out.append(o if i.gate is None else o * torch.sigmoid(i.gate[mine].double())[:, :, None])
                continue
            G = c["kv_heads"]
            q = i.q[mine].double().unflatten(1, (H, DIM))
            if c["design"] == "grouped":
                cos, sin = (x[mine].double()[:, None] for x in (i.cos, i.sin))
                q = torch.cat((_turn(q[:, :, :DIM // 2], cos, sin), q[:, :, DIM // 2:]), dim=2)
                k, v = (x.unflatten(1, (G, DIM)).double().repeat_interleave(H // G, 1) for x in rows.chunk(2, dim=1))
                o = _attend(q, k, v, first, c["window"], scale=DIM ** -0.5, sink=torch.zeros(H, dtype=torch.float64, device="cuda"))
                out.append(o.flatten(1) * torch.sigmoid(i.gate[mine].double()))
                continue
            off = (2 * G + 7) // 8 * 8
            inv = rows[:, :2 * G].contiguous().view(torch.float32).double()
            v = rows[:, off:].unflatten(1, (G, DIM)).double()
            k = (v * inv[:, :, None]).repeat_interleave(H // G, 1)
            q = q / (q.square().mean(2, keepdim=True) + EPS).sqrt() * i.norm.double()
            o = _attend(q, k, v.repeat_interleave(H // G, 1), first, c["window"], KEEP_FIRST, DIM ** -0.5, bias=i.slopes.double())
            out.append((o * torch.sigmoid(i.gate[mine].double())[:, :, None]).flatten(1))
        return torch.cat(out)
    B, longest = len(i.lens), max(i.lens)

    def padded(x):                                       # [T, ...] -> [B, longest, ...] in 64 bits, zeros behind a sequence's end
        return torch.nn.utils.rnn.pad_sequence([y.double() for y in x.split(i.lens)], batch_first=True)

    def packed(x):
        return torch.cat([x[b, :n] for b, n in enumerate(i.lens)])
    live = (torch.arange(longest, device="cuda")[None, :] < _ints(i.lens)[:, None]).double()
    if kind == "scan":
        C, N = c["channels"], SCAN_STATES
        xin, z = padded(i.xz[:, :C]), i.xz[:, C:].double()
        full = torch.cat((torch.zeros((B, SCAN_TAPS - 1, C), dtype=torch.float64, device="cuda"), xin), dim=1)
        x = sum(full[:, j:j + longest] * i.taps[:, j].double() for j in range(SCAN_TAPS)) + i.taps_b.double()
        x = torch.nn.functional.silu(x)
        tail = torch.stack([full[b, n:n + SCAN_TAPS - 1] for b, n in enumerate(i.lens)])
        # what the scan reads is the convolution's result in the storage type
        xr = x.to(i.xz.dtype).double()
        dt = torch.nn.functional.softplus(padded(i.dt) + i.dt_b.double()) * live[:, :, None]
        bc, A = padded(i.bc), i.A.double()
        S = torch.zeros((B, C, N), dtype=torch.float64, device="cuda")
        y = torch.empty((B, longest, C), dtype=torch.float64, device="cuda")
        for t in range(longest):
            d = dt[:, t, :, None]
            S = torch.exp(d * A) * S + d * xr[:, t, :, None] * bc[:, t, None, C // 32:C // 32 + N]
            y[:, t] = (S * bc[:, t, None, C // 32 + N:]).sum(2)
        y = packed(y) + packed(xr) * i.D.double()
        return packed(x), y * torch.nn.functional.silu(z), S, tail
    H = c["heads"]
    v, gate = padded(i.v).unflatten(2, (H, DIM)), i.gate.double().unflatten(1, (H, DIM))
    S = torch.zeros((B, H, DIM, DIM), dtype=torch.float64, device="cuda")
    o = torch.empty((B, longest, H, DIM), dtype=torch.float64, device="cuda")
    if kind == "gla":
        q, k = (padded(x).unflatten(2, (H, DIM)) for x in (i.q, i.k))
        decay = torch.sigmoid(padded(i.z) + i.bias.double()).pow(1.0 / GLA_TAU).unflatten(2, (H, DIM))
        for t in range(longest):
            a = torch.where(live[:, t, None, None] > 0, decay[:, t], torch.ones_like(decay[:, t]))
            S = a[..., None] * S + k[:, t][..., None] * v[:, t][:, :, None]
            o[:, t] = torch.matmul(q[:, t][:, :, None], S)[:, :, 0] * DIM ** -0.5
    else:
        def unit(x):
            x = x.unflatten(2, (H // 2, DIM)).repeat_interleave(2, 2)
            return x / (x.square().sum(3, keepdim=True) + 1e-6).sqrt()
        q, k = unit(padded(i.q)) * DIM ** -0.5, unit(padded(i.k))
        beta = torch.sigmoid(padded(i.z[:, :H])) * live[:, :, None]
        g = torch.exp(-i.rate.double() * torch.nn.functional.softplus(padded(i.z[:, H:]) + i.bias.double()) * live[:, :, None])
        for t in range(longest):
            S = g[:, t, :, None, None] * S
            u = beta[:, t, :, None] * (v[:, t] - torch.matmul(k[:, t][:, :, None], S)[:, :, 0])
            S = S + k[:, t][..., None] * u[:, :, None]
            o[:, t] = torch.matmul(q[:, t][:, :, None], S)[:, :, 0]
    o = packed(o)
    o = o / (o.square().mean(2, keepdim=True) + EPS).sqrt() * i.norm.double()
    return (o * torch.nn.functional.silu(gate)).flatten(1), S
