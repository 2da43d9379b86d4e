"""Rows around the layers of a step (csrc/row_ops.cu, csrc/elementwise.cu): token embeddings, rotary tables, the rows in front of the
head, greedy tokens.  Lookups and greedy tokens of tensors in host memory (the worker's logic without a GPU) are the tensor library's."""
import torch

from swiftllm_b200 import _lib


def embed_and_zero(table: torch.Tensor, ids: torch.Tensor):
    """Rows `ids` (int32) of table [V, H], and zeros of the same shape (the residual stream's start)."""
    if not ids.is_cuda:
        x = torch.embedding(table, ids, padding_idx=-1)
        return x, torch.zeros_like(x)
    x, zero = (torch.empty((ids.shape[0], table.shape[1]), dtype=table.dtype, device=table.device) for _ in range(2))
    size = table.shape[1] * table.element_size()
    _gather(ids, 0, table, x, size, None, zero, size)
    return x, zero


def gather_two(a: torch.Tensor, b: torch.Tensor, idx: torch.Tensor, offset: int = 0):
    """Rows idx + offset (idx int32) of two tables [n, d] of the same number of rows."""
    if not idx.is_cuda:
        at = idx.long() + offset
        return a.index_select(0, at), b.index_select(0, at)
    out_a, out_b = (torch.empty((idx.shape[0], t.shape[1]), dtype=t.dtype, device=t.device) for t in (a, b))
    assert a.shape[0] == b.shape[0] and b.is_contiguous()
    _gather(idx, offset, a, out_a, a.shape[1] * a.element_size(), b, out_b, b.shape[1] * b.element_size())
    return out_a, out_b


def _gather(idx, offset, a, out_a, bytes_a, b, out_b, bytes_b):
    assert idx.dtype == torch.int32 and idx.is_contiguous() and a.is_contiguous()
    _lib.require_device(a)
    _lib.check(_lib.lib().sllm_gather_rows(idx.data_ptr(), offset, idx.shape[0], a.shape[0], a.data_ptr(), out_a.data_ptr(), bytes_a,
                                           _lib.ptr(b), out_b.data_ptr(), bytes_b, _lib.stream()), "gather_rows")


def add_rmsnorm_rows(x: torch.Tensor, residual: torch.Tensor, rows: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """rms_norm(x + residual, weight) of the given rows (int32); the sum is rounded to the storage type first."""
    assert x.is_contiguous() and residual.is_contiguous() and weight.is_contiguous() and rows.is_contiguous()
    assert x.shape == residual.shape and x.dtype == residual.dtype == weight.dtype and rows.dtype == torch.int32
    _lib.require_device(x)
    out = torch.empty((rows.shape[0], x.shape[1]), dtype=x.dtype, device=x.device)
    _lib.check(_lib.lib().sllm_add_rmsnorm_rows(x.data_ptr(), residual.data_ptr(), rows.data_ptr(), weight.data_ptr(), eps, rows.shape[0],
                                                x.shape[0], x.shape[1], out.data_ptr(), _lib.dtype_tag(x.dtype), _lib.stream()),
               "add_rmsnorm_rows")
    return out


def argmax_rows(logits: torch.Tensor) -> torch.Tensor:
    """int64 [rows]: the index of each row's largest entry, the smallest among equals."""
    if not logits.is_cuda:
        return torch.argmax(logits, dim=1)
    assert logits.dim() == 2 and logits.stride(1) == 1
    _lib.require_device(logits)
    out = torch.empty((logits.shape[0],), dtype=torch.int64, device=logits.device)
    _lib.check(_lib.lib().sllm_argmax_rows(logits.data_ptr(), logits.stride(0), logits.shape[0], logits.shape[1], out.data_ptr(),
                                           _lib.dtype_tag_f32(logits.dtype), _lib.stream()), "argmax_rows")
    return out
