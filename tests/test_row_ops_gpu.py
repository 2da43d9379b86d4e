"""GPU: rows around the layers (csrc/row_ops.cu, the gathered rows of csrc/elementwise.cu) against the tensor library, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,n,spare", [(1, 1, 0), (3, 7, 0), (2, 2048, 8), (5, 16385, 0), (16, 128256, 0), (300, 512, 3)])
def test_argmax_rows(dtype, rows, n, spare):
    """Every tail of the clusters' runs, rows off the 16-byte grid, ties (the smallest index), NaN (above all), infinities."""
    from swiftllm_b200.worker.kernels.row_ops import argmax_rows
    g = torch.Generator().manual_seed(rows * n)
    x = torch.randn(rows, n + spare, generator=g).to(dtype).to(DEV)[:, :n]
    at = torch.randint(0, n, (rows, 3), generator=g)
    for kind in ("ties", "nan", "low", "zeros"):
        y = torch.full((rows, n + spare), float("-inf")) if kind == "low" else torch.zeros(rows, n + spare) - float(kind != "zeros")
        if kind in ("ties", "nan"):
            y.scatter_(1, at, 3.0 if kind == "ties" else float("nan"))
        if kind == "zeros":
            y.scatter_(1, at, -0.0)
        want = at.min(dim=1).values if kind in ("ties", "nan") else torch.zeros(rows, dtype=torch.int64)
        assert torch.equal(argmax_rows(y.to(dtype).to(DEV)[:, :n]).cpu(), want), kind
    first = (x == x.amax(dim=1, keepdim=True)).int().cpu().float().argmax(dim=1)       # the first of the largest
    assert torch.equal(argmax_rows(x).cpu(), first)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("width", [1, 6, 8, 64, 4096, 5000])
def test_gathered_rows(dtype, width):
    from swiftllm_b200.worker.kernels.row_ops import embed_and_zero, gather_two
    g = torch.Generator().manual_seed(width)
    a, b = (torch.randn(37, width, generator=g).to(dtype).to(DEV) for _ in range(2))
    ids = torch.tensor([1, 36, 1, 20, 7], dtype=torch.int32, device=DEV)
    x, zero = embed_and_zero(a, ids)
    assert torch.equal(x, a[ids.long()]) and not zero.any() and zero.shape == x.shape
    for offset in (0, -1):
        p, q = gather_two(a, b, ids, offset)
        assert torch.equal(p, a[ids.long() + offset]) and torch.equal(q, b[ids.long() + offset])
    assert embed_and_zero(a, ids[:0])[0].shape == (0, width)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hidden", [8, 1000, 1024, 4096, 8192, 14336])
def test_add_rmsnorm_of_rows(dtype, hidden):
    """The same bits as an addition over all rows, a selection and a norm in place (one thread layout per row length)."""
    from swiftllm_b200.worker.kernels.rmsnorm import rmsnorm_inplace
    from swiftllm_b200.worker.kernels.row_ops import add_rmsnorm_rows
    g = torch.Generator().manual_seed(hidden)
    x, r = (torch.randn(9, hidden, generator=g).to(dtype).to(DEV) for _ in range(2))
    w = (1 + 0.1 * torch.randn(hidden, generator=g)).to(dtype).to(DEV)
    rows = torch.tensor([8, 0, 3, 3], dtype=torch.int32, device=DEV)
    want = (x + r)[rows.long()]
    rmsnorm_inplace(want, w, 1e-5)
    keep = x.clone(), r.clone()
    assert torch.equal(add_rmsnorm_rows(x, r, rows, w, 1e-5), want)
    assert torch.equal(x, keep[0]) and torch.equal(r, keep[1])
