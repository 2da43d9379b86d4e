"""GPU: rows that share tiles with other rows (csrc/latent_attn_tc.cu, window_attn_tc.cu, prefill_attn_paged.cu, scan_ops.cu) take nothing
from keys that they do not see, and agree with 64-bit arithmetic in every part of a tile."""
import pytest
import torch

from tile_cases import DEV, TYPES, UNIT, attend, ints, normal, rel, segments, table
from tile_cases import latent_case, latent_exact, latent_run, window_case, window_columns, window_exact, window_run

pytestmark = pytest.mark.gpu


# ---------------------------------------------------------------- selective scan
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("C,N", [(2048, 16), (24, 8)])
def test_selective_scan_gate_is_the_plain_one(dtype, C, N):
    # without input to the state the output is silu(gate), rounded once: the vector path, the plain path (which a view that is not
    # aligned takes) and decoded tokens give the same bits only if they take the same exponential and quotient
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    T = 64
    one, zero = torch.ones(C, device=DEV), torch.zeros(T, 2 * N, dtype=dtype, device=DEV)
    z = normal(T, C + 8, seed=C, dtype=dtype) * 6
    A, dt = -torch.ones(C, N, device=DEV), torch.zeros(T, C, device=DEV)
    outs = []
    for off, decoded in ((0, False), (1, False), (0, True)):
        st = segments([1] * T, range(T), True) if decoded else segments([T], [0])
        gate = torch.zeros_like(z)[:, off:off + C]
        gate.copy_(z[:, :C])
        outs.append(selective_scan(torch.ones(T, C, dtype=dtype, device=DEV), dt, one, A, zero, 0, N, one, gate,
                                   torch.zeros(st.batch_size, C, N, device=DEV), st))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
