"""GPU: the order in which the CTAs of windowed prompt rows come (csrc/window_attn_tc.cu): groups together, or one behind the other where decoded rows of a round
of CTAs run beside more than a round of them.  Every row is the same in both orders, bit for bit, and as near the oracle as in test_window_boxes_gpu.py."""
import pytest
import torch

from tile_cases import TYPES, UNIT, rel, window_case, window_exact, window_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("decodes", [40, 3])                 # 160 CTAs beside 160 of the prompts: one group behind the other; 12: together
def test_order_of_groups(dtype, decodes):
    c = window_case(dtype, [(1300, 0), (700, 0), (530, 3)], [200 + 7 * i for i in range(decodes)], 16, 4, 128, 128, 64, 1024, {})
    ref, got, at = window_exact(c), window_run(c), 0
    for n, p in c.rows:
        assert rel(got[at:at + n], ref[at:at + n]) < UNIT[dtype], (n, p)
        at += n
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                            # (captured, all rows run on one stream: together)
        again = window_run(c)
    graph.replay()
    assert torch.equal(got, again)
