"""Latent attention over the paged latent cache (csrc/latent_attn.cu).  Cache layout [num_blocks, slots, block_size, r + dr]:
per token and caching layer ONE row [normed latent | rotated key part] shared by all heads."""
import torch

from swiftllm_b200 import _lib


def latent_kv_store(dkv: torch.Tensor, norm_weight: torch.Tensor, cache: torch.Tensor, slot: int, block_table: torch.Tensor,
                    infer_state, r: int, dr: int, rot_dims: int, eps: float, cos: torch.Tensor, sin: torch.Tensor):
    """dkv [T, r + dr] (row-strided): RMS-norm the first r columns, rotate the rest, write the tokens' cache rows."""
    assert dkv.dim() == 2 and dkv.stride(1) == 1 and dkv.shape[1] == r + dr and cache.is_contiguous() and cache.dtype == dkv.dtype
    _lib.require_device(dkv)
    T = dkv.shape[0]
    _lib.check(_lib.lib().sllm_latent_kv_store(
        dkv.data_ptr(), dkv.stride(0) if T > 1 else max(dkv.stride(0), r + dr), norm_weight.data_ptr(), _lib.ptr(cos), _lib.ptr(sin),
        infer_state.token_seq_ids.data_ptr(), infer_state.token_positions.data_ptr(), block_table.data_ptr(), block_table.shape[1],
        cache.data_ptr(), cache.shape[1], slot, cache.shape[2], T, r, dr, rot_dims, eps, _lib.dtype_tag_f32(dkv.dtype),
        _lib.stream()), "latent_kv_store")


_SM_COUNT = {}


def _num_splits(rows: int, H: int, r: int, dr: int, window: int, dtype, portions: bool, seqs: int = 1) -> int:
    """Key splits of a launch over `rows` tokens (portions of `seqs` prompts, or single decoded tokens): as many CTAs as fit at once when
    the rows alone leave SMs idle, never a second wave; never more than the 64-key tiles a window can hold (16 when there is no window).
    Several prompts leave half the SMs to the second segments of CTAs in which one ends (three of 33 tokens, 16 heads: 38 -> 32 us)."""
    if dtype == torch.float32:
        return 1
    dev = torch.cuda.current_device()
    if dev not in _SM_COUNT:
        _SM_COUNT[dev] = torch.cuda.get_device_properties(dev).multi_processor_count
    if r % 64 == 0 and r <= 512 and dr % 16 == 0 and dr <= 64:         # one CTA per SM, 64 (token, head) rows each
        heads = 1
        while heads < H and heads < 64:
            heads *= 2
        per = 64 // heads if portions else 1
        ctas, room = -(-rows // per) * -(-H // heads), _SM_COUNT[dev] // (2 if portions and seqs > 1 else 1)
    else:                                                              # two CTAs per SM, one token and 16 heads each
        ctas, room = rows * ((H + 15) // 16), 2 * _SM_COUNT[dev]
    most = (window + 63) // 64 + 1 if window > 0 else 16
    return max(1, min(room // ctas, most, 32))


def latent_attention(q_lat: torch.Tensor, q_rot: torch.Tensor, gate, cache: torch.Tensor, slot: int, block_table: torch.Tensor,
                     infer_state, out: torch.Tensor, rot_dims: int, window: int, scale: float, cos: torch.Tensor, sin: torch.Tensor,
                     sink: torch.Tensor = None):
    """q_lat [T, H, r], q_rot [T, H, dr] (un-rotated), gate [T, H] logits or None, out [T, H, r]; views with arbitrary token /
    head strides are taken as they are (the innermost stride must be 1).  sink fp32 [H] or None: exp(sink[h]) joins the softmax's
    denominator."""
    T, H, r = q_lat.shape
    dr = q_rot.shape[2]
    assert q_lat.stride(2) == 1 and q_rot.stride(2) == 1 and out.stride(2) == 1 and out.shape == q_lat.shape
    assert cache.shape[3] == r + dr and cache.dtype == q_lat.dtype
    assert gate is None or (gate.shape == (T, H) and gate.stride(1) == 1)
    assert sink is None or (sink.dtype == torch.float32 and sink.shape == (H,) and sink.is_contiguous())
    _lib.require_device(q_lat)
    npre = min(T, max(0, int(getattr(infer_state, "num_prefill_tokens", 0))))
    lib, es = _lib.lib(), q_lat.element_size()
    (ql_t, ql_h, _), (qr_t, qr_h, _), (o_t, o_h, _) = q_lat.stride(), q_rot.stride(), out.stride()
    gate_t = gate.stride(0) if gate is not None else 0
    half = rot_dims // 2 * 4
    ql, qr, o, g, c, sn = q_lat.data_ptr(), q_rot.data_ptr(), out.data_ptr(), _lib.ptr(gate), _lib.ptr(cos), _lib.ptr(sin)
    ts, tp = infer_state.token_seq_ids.data_ptr(), infer_state.token_positions.data_ptr()
    _, n_slots, bs, _ = cache.shape
    dtype, stream = _lib.dtype_tag_f32(q_lat.dtype), _lib.stream()
    for i, rows, portions in ((0, npre, True), (npre, T - npre, False)):       # i: the part's first row
        if rows == 0:
            continue
        nsplit = _num_splits(rows, H, r, dr, window, q_lat.dtype, portions, int(getattr(infer_state, "num_prefill_seqs", 1)))
        ws = torch.empty((rows, H, nsplit, r + 2), dtype=torch.float32, device=q_lat.device) if nsplit > 1 else None
        _lib.check((lib.sllm_latent_attention_portions if portions else lib.sllm_latent_attention)(
            ql + i * ql_t * es, ql_t, ql_h, qr + i * qr_t * es, qr_t, qr_h, c + i * half if c else None, sn + i * half if sn else None,
            g + i * gate_t * es if g else None, gate_t, cache.data_ptr(), n_slots, slot, bs, block_table.data_ptr(), block_table.shape[1],
            ts + 4 * i, tp + 4 * i, o + i * o_t * es, o_t, o_h, rows, H, r, dr, rot_dims, window, scale, _lib.ptr(sink), nsplit,
            _lib.ptr(ws), dtype, stream), "latent_attention")
