"""GPU: the selective scan of 16 states with staged steps (csrc/scan_ops.cu), one and two channels per lane, and the convolution's tiles,
against the rules in 64 bits."""
import pytest
import torch

from test_tile_edges_gpu import _normal, _segments

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lens,firsts,C", [
    ((1,), (0,), 8), ((31, 2), (5, 0), 72), ((32, 33, 64), (0, 9, 3), 40),                 # one channel per lane
    ((66, 4), (2, 0), 4808), ((33, 1, 32, 65), (0, 7, 3, 0), 4808)])                       # two (the last)
def test_scan_of_sixteen_states(dtype, lens, firsts, C):
    """Outputs are rounded once; the state's relative error is that of its decays' exponents: products of about 10 at most, rounded to
    24 bits, in sums of up to 66 tokens whose older part fades."""
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    N, st, T = 16, _segments(lens, firsts), sum(lens)
    base = _normal(T, 2 * C + 2 * N + 8, seed=C, dtype=dtype)
    x, z, bc = base[:, :C], base[:, C:2 * C], base[:, 2 * C:]
    dt, bias = _normal(T, C, seed=1), _normal(C, seed=2) - 3
    A, D, S0 = -(_normal(C, N, seed=3).abs() + 0.1), _normal(C, seed=4), _normal(len(lens), C, N, seed=5)
    state = S0.clone()
    y = selective_scan(x, dt, bias, A, bc, 0, N, D, z, state, st)
    steps = torch.nn.functional.softplus(dt.double() + bias.double())
    want, at = torch.empty(T, C, dtype=torch.float64, device=x.device), 0
    for i, (n, first) in enumerate(zip(lens, firsts)):
        row = int(st.seq_ids[i])
        S = S0[row].double() if first > 0 else torch.zeros(C, N, dtype=torch.float64, device=x.device)
        for t in range(at, at + n):
            S = torch.exp(steps[t, :, None] * A.double()) * S + (steps[t] * x[t].double())[:, None] * bc[t, None, :N].double()
            want[t] = ((S * bc[t, None, N:2 * N].double()).sum(1) + D.double() * x[t].double()) * torch.nn.functional.silu(z[t].double())
        at += n
        assert float((state[row].double() - S).norm() / S.norm()) < 2e-6
    assert float((y.double() - want).norm() / want.norm()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)


@pytest.mark.parametrize("taps", [3, 4])
def test_convolution_tiles(taps):
    """Segments that begin and end on every row near a tile's edge; as many channels as the vector kernel asks for at these rows."""
    from swiftllm_b200.worker.kernels.scan_ops import short_conv
    lens, firsts = (31, 1, 2, 30, 33, 5, 64, 1, 1, 88), (0, 3, 1, 0, 2, 0, 9, 1, 0, 4)
    C, T, st = 4104, sum(lens), _segments(lens, firsts)
    assert T * C >= 1 << 20
    x, w, b = _normal(T, C, seed=1, dtype=torch.bfloat16), _normal(C, taps, seed=2), _normal(C, seed=3)
    tail0 = _normal(len(lens), taps - 1, C, seed=4, dtype=torch.bfloat16)
    tail = tail0.clone()
    y = short_conv(x, w, b, tail, st, torch.bfloat16, silu=True, move_tail=True)
    at = 0
    for i, (n, first) in enumerate(zip(lens, firsts)):
        row = int(st.seq_ids[i])
        before = tail0[row].double() * (torch.arange(first - taps + 1, first, device=x.device) >= 0)[:, None]
        full = torch.cat((before, x[at:at + n].double()))
        acc = sum(full[k:k + n] * w[:, k].double() for k in range(taps)) + b.double()
        want = torch.nn.functional.silu(acc)
        assert float((y[at:at + n].double() - want).norm() / want.norm()) < 2.0 ** -8, i
        assert torch.equal(tail[row].double(), full[n:])
        at += n


@pytest.mark.parametrize("times,taps", [(7, 3), (8, 4), (27, 4), (28, 3), (29, 4)])
def test_convolution_tile_heights(times, taps):
    """Tiles of 8, 16 and 32 rows, by the number of entries: on both sides of the lines between them."""
    from swiftllm_b200.worker.kernels.scan_ops import short_conv
    lens = (31, 1, 2, 30, 33, 5, 64, 1, 1, 87) * times + (3,)
    firsts = (0, 3, 1, 0, 2, 0, 9, 1, 0, 4) * times + (0,)
    C, T, st = 4104, sum(lens), _segments(lens, firsts)
    x, w, b = _normal(T, C, seed=1, dtype=torch.bfloat16), _normal(C, taps, seed=2), _normal(C, seed=3)
    tail0 = _normal(len(lens), taps - 1, C, seed=4, dtype=torch.bfloat16)
    y = short_conv(x, w, b, tail0.clone(), st, torch.bfloat16, silu=True, move_tail=True)
    at = 0
    for i, (n, first) in enumerate(zip(lens, firsts)):
        before = tail0[i].double() * (torch.arange(first - taps + 1, first, device=x.device) >= 0)[:, None]
        full = torch.cat((before, x[at:at + n].double()))
        want = torch.nn.functional.silu(sum(full[k:k + n] * w[:, k].double() for k in range(taps)) + b.double())
        assert float((y[at:at + n].double() - want).norm() / want.norm()) < 2.0 ** -8, i
        at += n


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lens,C", [((8, 24, 3, 17, 9), 4808), ((1, 16, 33, 2, 40, 7), 16008), ((28, 24, 24, 24, 25), 4808), ((8, 7, 8, 8, 8), 4808)])
def test_scan_of_short_portions(dtype, lens, C):
    """Many short portions (the first two; the others are on the other side of the lines), and a state off the 16-byte grid; outputs are
    rounded once, states as in the test of longer ones."""
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    N, firsts, T = 16, [3 * (i % 2) for i in range(len(lens))], sum(lens)
    st = _segments(lens, firsts)
    x, z, bc = _normal(T, 2 * C, seed=C, dtype=dtype)[:, :C], _normal(T, C, seed=9, dtype=dtype), _normal(T, 2 * N, seed=8, dtype=dtype)
    dt, bias = _normal(T, C, seed=1), _normal(C, seed=2) - 3
    A, D, S0 = -(_normal(C, N, seed=3).abs() + 0.1), _normal(C, seed=4), _normal(len(lens), C, N, seed=5)
    states = [S0.clone(), torch.zeros(S0.numel() + 1, device=x.device)[1:].view_as(S0).copy_(S0)]
    outs = [selective_scan(x, dt, bias, A, bc, 0, N, D, z, s, st) for s in states]
    steps, want, at = torch.nn.functional.softplus(dt.double() + bias.double()), torch.empty(T, C, dtype=torch.float64, device=x.device), 0
    for i, (n, first) in enumerate(zip(lens, firsts)):
        S = S0[i].double() if first > 0 else torch.zeros(C, N, dtype=torch.float64, device=x.device)
        for t in range(at, at + n):
            S = torch.exp(steps[t, :, None] * A.double()) * S + (steps[t] * x[t].double())[:, None] * bc[t, None, :N].double()
            want[t] = ((S * bc[t, None, N:].double()).sum(1) + D.double() * x[t].double()) * torch.nn.functional.silu(z[t].double())
        at += n
        assert all(float((s[i].double() - S).norm() / S.norm()) < 2e-6 for s in states)
    for y in outs:
        assert float((y.double() - want).norm() / want.norm()) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)


@pytest.mark.parametrize("n", [1, 16, 33])
def test_steps_are_as_exact_as_the_plain_functions(n):
    """One input of 1 through B = 1 and no decay leaves the step in the state: no further off 64 bits, in the mean square, than log1p(exp(z))
    of the tensor library's fp32 functions, in both kernels of 16 states; logits of any size."""
    from swiftllm_b200.worker.kernels.scan_ops import selective_scan
    C, N, st = 1 << 16, 16, _segments((n,), (0,))
    z = torch.rand(C, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * 24 - 12
    ends = torch.tensor([-104.0, float("-inf"), -87.0, -30.0, 20.5, 88.0, 1e30, 0.0, -0.0], device="cuda")
    logits = torch.full((n, C), float("-inf"), device="cuda")            # steps of 0 but for the first token
    logits[0] = z
    logits[0, :9] = ends
    one = torch.ones(n, C, dtype=torch.bfloat16, device="cuda")
    state = torch.zeros(1, C, N, device="cuda")
    selective_scan(one, logits, torch.zeros(C, device="cuda"), torch.zeros(C, N, device="cuda"), one[:, :2 * N], 0, N,
                   torch.zeros(C, device="cuda"), one, state, st)
    want = torch.nn.functional.softplus(logits[0].double(), threshold=1e9)
    assert torch.equal(state[0], state[0, :, :1].expand(C, N))
    off = lambda y: float(((y.double() - want) / want)[9:].square().mean().sqrt())
    assert off(state[0, :, 0]) <= off(torch.log1p(torch.exp(logits[0])))
    got = state[0, :9, 0].double()
    assert float(got[0]) < 1e-44 and float(got[1]) == 0.0
    assert bool(((got - want[:9]).abs() <= 2.0 ** -20 * want[:9])[2:].all())
