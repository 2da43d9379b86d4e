"""Reference: swiftllm/worker/kernels/prefill_attn.py (prefill_attention :102-139); also replaces the
vllm_flash_attn.flash_attn_varlen_func call at swiftllm/worker/layers/transformer_layer.py:86-96."""
import functools

import torch

from swiftllm_b200 import _lib
from swiftllm_b200.worker.infer_state import LlamaInferState


def prefill_attention(
    q: torch.Tensor,    # [num_prefill_tokens, num_q_heads, head_dim]
    k: torch.Tensor,    # [num_prefill_tokens, num_kv_heads, head_dim]
    v: torch.Tensor,    # [num_prefill_tokens, num_kv_heads, head_dim]
    o: torch.Tensor,    # [num_prefill_tokens, num_q_heads, head_dim]
    model_config,
    engine_config,
    infer_state: LlamaInferState,
):
    assert o.is_contiguous()
    qs, ks, vs = _lib.row_stride(q), _lib.row_stride(k), _lib.row_stride(v)
    _lib.require_device(q)
    Tp, nq, D = q.shape
    nkv = k.shape[1]
    if infer_state.num_prefill_seqs == 0:
        return
    _lib.check(_lib.lib().sllm_prefill_attention(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
        infer_state.prefill_seq_start_locs.data_ptr(), infer_state.prefill_seq_lens.data_ptr(),
        infer_state.softmax_scale, infer_state.num_prefill_seqs, infer_state.max_prefill_len, Tp, nq, nkv, D, qs, ks, vs,
        _lib.dtype_tag(q.dtype), _lib.stream()), "prefill_attention")


_SM_COUNT = {}


def _key_splits(heads: int, longest: int, kv_len: int, blocks=None) -> int:
    """CTAs that share a query block's keys when the portions alone leave SMs idle: as many as find an SM at once, each with at least eight steps of 80
    keys, or six where eight leave half of the SMs idle (shorter ones do not pay for the merge).  `blocks`: the launch's query blocks if they have
    one tile, and two (None: a block for 256 rows of a head).  Measured on B200, us, splits counted by 256 rows of a head / by the blocks, in which
    heads lie side by side: 16 tokens at 5000, 64 / 8 heads, 35.2 / 17.8; four portions of up to 16 at 5000, 32 / 8 heads, 62.8 / 24.8; 300 at 3000,
    32 / 8 heads, 36.3 / 30.6; 64 at 5000, 16 / 4 heads, 19.2 / 17.8; 512 at 3584, 32 / 8 heads, 43.8 both."""
    dev = torch.cuda.current_device()
    if dev not in _SM_COUNT:
        _SM_COUNT[dev] = torch.cuda.get_device_properties(dev).multi_processor_count
    return _splits(_SM_COUNT[dev], kv_len, *(blocks or (heads * -(-longest // 256),) * 2), blocks is not None)


@functools.lru_cache(maxsize=1024)
def _splits(sms: int, kv_len: int, ones: int, twos: int, fewer_steps: bool) -> int:
    most = kv_len // 640
    if fewer_steps and most > 1 and ones * most <= sms // 2:
        most = kv_len // 480
    one, two = (min(sms // max(1, b), most, 16) for b in (ones, twos))
    if two <= max(1, one):
        return max(1, one)
    # Blocks of two tiles leave room for more splits.  In tenths of a microsecond: a step takes them 12 and blocks of one tile 9; splits and their merge
    # come to 95 and 50 (64 / 8 heads, 128 tokens at 5000: two splits of one tile 38.3 us, four of two 33.6; 16 / 4 heads, 512 at 2000: 23.8 and 26.2)
    steps, of_one = -(-kv_len // 80), 9 if one else 12                 # (more blocks of one tile than SMs: a launch without splits has two)
    alone = of_one * -(-steps // max(1, one)) + (50 if one > 1 else 0)
    return two if 12 * -(-steps // two) + 95 < alone else max(1, one)


@functools.lru_cache(maxsize=1024)
def _blocks(nq: int, nkv: int, seqs: int, longest: int, rows: int):
    return tuple(_lib.lib().sllm_prefill_attention_blocks(nq, nkv, seqs, longest, rows, tiles) for tiles in (1, 2))


def prefill_attention_paged(
    q: torch.Tensor,            # [num_prefill_tokens, num_q_heads, head_dim]  (the chunks' queries, packed)
    k_cache: torch.Tensor,      # [num_blocks, num_layers, num_kv_heads, block_size, head_dim]
    v_cache: torch.Tensor,
    block_table: torch.Tensor,  # [max_seqs, max_blocks_per_seq] int32
    o: torch.Tensor,            # [num_prefill_tokens, num_q_heads, head_dim]
    model_config,
    engine_config,
    infer_state: LlamaInferState,
    cur_layer: int,
):
    """Chunked ("prefix-aware") prefill attention (no counterpart in the reference, whose prefill attention
    never reads the KV cache): the chunk's queries sit at positions prefill_prefix_lens[i] + t of their sequence and attend
    to positions <= their own, keys / values read from the paged cache (the chunk's own K/V are stored first)."""
    assert o.is_contiguous() and k_cache.is_contiguous() and v_cache.is_contiguous() and block_table.is_contiguous()
    assert block_table.dtype == torch.int32 and infer_state.seq_ids.dtype == torch.int32
    prefix = infer_state.prefill_prefix_lens
    assert prefix is not None and prefix.dtype == torch.int32 and prefix.is_contiguous()
    qs = _lib.row_stride(q)
    _lib.require_device(q)
    Tp, nq, D = q.shape
    if infer_state.num_prefill_seqs == 0:
        return
    num_blocks, num_layers, nkv, bs, _ = k_cache.shape
    n, longest = infer_state.num_prefill_seqs, infer_state.max_prefill_len
    nsplit = _key_splits(nq * n, longest, getattr(infer_state, "max_prefill_kv_len", 0), _blocks(nq, nkv, n, longest, Tp)) \
        if D == 128 and bs == 16 else 1
    ws = torch.empty((nsplit * Tp * nq * (D + 2),), dtype=torch.float32, device=q.device) if nsplit > 1 else None
    _lib.check(_lib.lib().sllm_prefill_attention_paged_split(
        q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), o.data_ptr(), block_table.data_ptr(),
        infer_state.seq_ids.data_ptr(), infer_state.prefill_seq_start_locs.data_ptr(), infer_state.prefill_seq_lens.data_ptr(),
        prefix.data_ptr(), infer_state.softmax_scale, infer_state.num_prefill_seqs, infer_state.max_prefill_len, Tp,
        cur_layer, num_layers, nq, nkv, bs, D, block_table.shape[1], num_blocks, qs,
        _lib.dtype_tag(q.dtype), _lib.stream(), nsplit, _lib.ptr(ws)), "prefill_attention_paged")
