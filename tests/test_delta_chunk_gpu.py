"""GPU: prompt portions of the gated delta rule in chunks on the tensor cores (csrc/delta_chunk.cuh) against the rule token by token in 64
bits: every width of a CTA, remainders of a chunk, carried states, values that are not finite."""
import pytest
import torch

from oracle import vorerax as O
from test_buzarax_gpu import _step

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(dtype, lens, H, G, dk, dv, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *shape: torch.randn(*shape, generator=g, device=DEV)
    T = sum(lens)
    x = dict(qkv=(r(T, (2 * G) * dk + H * dv) * scale).to(dtype), gate=r(T, H * dv).to(dtype), a=r(T, H), b=r(T, H) * 2, bias=r(H),
             rate=torch.exp(torch.linspace(-7.0, 4.5, H, device=DEV)), w=1 + 0.3 * r(dv), state=r(len(lens) + 1, H, dk, dv))
    x["q"], x["k"], x["v"] = x["qkv"].split([G * dk, G * dk, H * dv], dim=1)
    # segments whose state is carried in, and fresh ones, in rows that are not in order
    st = _step([(len(lens) - 1 - i, 40 if i % 2 == 0 else 0, n) for i, n in enumerate(lens)])
    st.num_prefill_seqs, st.num_prefill_tokens = len(lens), T
    return x, st


def _run(x, st, H, G, dk, dv):
    from swiftllm_b200.worker.kernels.head_decay import delta_rule
    state = x["state"].clone()
    return delta_rule(x["q"], x["k"], x["v"], x["a"], x["b"], x["bias"], x["rate"], x["w"], 1e-5, x["gate"], state, st, H, G, dk, dv), state


def _exact(x, lens, H, G, dk, dv):
    out, states, at = [], {}, 0
    which = torch.arange(H, device=DEV) // (H // G)
    for i, n in enumerate(lens):
        d = {c: y[at:at + n].double() for c, y in x.items() if c in ("q", "k", "v", "gate", "a", "b")}
        at += n
        q, k = (O.unit_length(d[c].view(n, G, dk))[:, which] for c in "qk")
        decay = torch.exp(-x["rate"].double() * torch.nn.functional.softplus(d["a"] + x["bias"].double()))
        beta, v, row = torch.sigmoid(d["b"]), d["v"].view(n, H, dv), len(lens) - 1 - i
        S = x["state"][row].double() if i % 2 == 0 else torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV)
        for t in range(n):
            S = decay[t][:, None, None] * S
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t])))[:, None, :]
            o = torch.einsum("hkv,hk->hv", S, q[t] * dk ** -0.5)
            out.append((O.unit_rms(o, 1e-5) * x["w"].double()).reshape(-1) * torch.nn.functional.silu(d["gate"][t]))
        states[row] = S
    return torch.stack(out), states


def _off(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lens,H,G,dk,dv", [
    ([1, 33], 4, 4, 128, 128), ([31, 97], 12, 6, 128, 128), ([32, 64, 65], 16, 8, 128, 128), ([63, 1, 2, 96, 40], 16, 8, 128, 128),
    ([129], 80, 40, 64, 160), ([50, 7], 3, 1, 40, 24), ([34, 100], 2, 2, 8, 8), ([45] * 6, 30, 10, 96, 72)])
def test_chunks_against_the_rule(dtype, lens, H, G, dk, dv):
    """Outputs are rounded once (half a unit in the last place: 2^-9 or 2^-12 at most, 0.58 of that in the mean square); the state's sums
    of up to 129 tokens are fp32 sums: 32 units of 2^-24 are far above what independent roundings of so many add up to."""
    x, st = _case(dtype, lens, H, G, dk, dv, seed=sum(lens) + dk)
    out, state = _run(x, st, H, G, dk, dv)
    ref, states = _exact(x, lens, H, G, dk, dv)
    assert _off(out, ref) < (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for row, S in states.items():
        assert _off(state[row], S) < 32 * 2.0 ** -24
    assert torch.equal(state[len(lens)], x["state"][len(lens)])


@pytest.mark.parametrize("scale", [1e-4, 300.0])
def test_scales_of_rows(scale):
    """Keys of any length are unit vectors; values carry their scale through the state."""
    lens, shape = [70, 33], (6, 3, 128, 128)
    x, st = _case(torch.bfloat16, lens, *shape, seed=3, scale=scale)
    out, state = _run(x, st, *shape)
    ref, states = _exact(x, lens, *shape)
    assert _off(out, ref) < 2.0 ** -9 and all(_off(state[r], S) < 32 * 2.0 ** -24 for r, S in states.items())


@pytest.mark.parametrize("what,value", [("v", float("inf")), ("v", float("nan")), ("k", float("nan")), ("q", float("nan")), ("a", float("nan")),
                                        ("b", float("nan")), ("a", float("inf"))])
def test_values_that_are_not_finite_reach_what_follows(what, value):
    """One entry of one token: rows before it and other heads' and sequences' rows and states stay as they are; a decay of zero (a = inf)
    only forgets."""
    lens, (H, G, dk, dv) = [70, 45], (4, 2, 64, 64)
    x, st = _case(torch.bfloat16, lens, H, G, dk, dv, seed=5)
    clean, clean_state = _run(x, st, H, G, dk, dv)
    row, head = 41, 2
    x[what][row, {"v": head * dv + 5, "q": dk + 3, "k": dk + 3, "a": head, "b": head}[what]] = value
    out, state = _run(x, st, H, G, dk, dv)
    hit = [2, 3] if what in "qk" else [head]                             # heads that share the key head
    o, c = out.float().view(-1, H, dv), clean.float().view(-1, H, dv)
    others = [h for h in range(H) if h not in hit]
    assert torch.equal(o[:, others], c[:, others]) and torch.equal(o[70:], c[70:])
    assert torch.equal(state[0], clean_state[0]) and torch.equal(state[1][others], clean_state[1][others])
    assert float((o[:row] - c[:row]).norm() / c[:row].norm()) < 2.0 ** -8          # token by token: rounded another way
    if value == float("inf") and what == "a":
        ref, states = _exact(x, lens, H, G, dk, dv)
        assert _off(out, ref) < 2.0 ** -9 and _off(state[1], states[1]) < 32 * 2.0 ** -24
    elif what == "q":
        assert not o[row, hit].isfinite().any() and torch.equal(o[row + 1:], c[row + 1:]) and torch.equal(state, clean_state)
    else:
        assert not o[row:70, hit].isfinite().any()
        if what == "v":                                                   # the state's other columns go on
            keep = [e for e in range(dv) if e != 5]
            assert _off(state[1][head][:, keep], clean_state[1][head][:, keep].double()) < 32 * 2.0 ** -24
            assert not state[1][head][:, 5].isfinite().any()


@pytest.mark.parametrize("lens,H,G,dk,dv", [
    ([8], 4, 4, 128, 128), ([9], 4, 4, 128, 128), ([1, 8, 15], 6, 3, 128, 128), ([9, 9], 48, 24, 128, 128), ([8, 8], 48, 24, 128, 128),
    ([8] * 6, 20, 10, 64, 128), ([17, 16], 4, 2, 64, 64), ([16] * 3, 4, 2, 64, 64), ([24] * 5, 20, 10, 64, 64), ([25] * 5, 20, 10, 64, 64),
    ([24], 4, 4, 32, 32), ([25], 4, 4, 32, 32), ([8] * 3, 16, 8, 96, 160), ([8] * 4, 16, 8, 96, 160)])
def test_short_portions(lens, H, G, dk, dv):
    """Both sides of the lines between batches of eight tokens and chunks."""
    x, st = _case(torch.bfloat16, lens, H, G, dk, dv, seed=sum(lens) + dv)
    out, state = _run(x, st, H, G, dk, dv)
    ref, states = _exact(x, lens, H, G, dk, dv)
    assert _off(out, ref) < 2.0 ** -9 and all(_off(state[r], S) < 32 * 2.0 ** -24 for r, S in states.items())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("noise,lens,H,dv", [(0.0, [40, 33], 2, 128), (0.0, [257], 12, 128), (1e-3, [64, 97], 2, 128), (0.0, [70], 6, 160), (0.0, [50, 64], 3, 64)])
def test_rows_of_very_different_sizes(dtype, noise, lens, H, dv):
    """Every other row of the state is 2^20 below the rest of its columns, and so are the values that (nearly) one-hot keys write into it,
    among the others in the same chunks.  A row's entries are sums of as many fp32 numbers as tokens touch it (a dozen at most, and the
    decays' product): 2^-20 of the row is sixteen units in the last place of such a number, where operands cut at 2^-38 of their column
    would leave 2^-18 and more.  With noise the small rows also
    hold the products of all keys with the large ones: twice that."""
    dk, T = 128, sum(lens)
    x, st = _case(dtype, lens, H, H, dk, dv, seed=T + dv)
    g = torch.Generator(device=DEV).manual_seed(T)
    at = torch.randint(0, dk, (T,), generator=g, device=DEV)
    small = torch.where(torch.arange(dk, device=DEV) % 2 == 0, 1.0, 2.0 ** -20)
    least = small if dtype == torch.bfloat16 else small.clamp_min(2.0 ** -10)               # what fp16 values can be
    hot = torch.nn.functional.one_hot(at, dk).float() + noise * torch.randn(T, dk, generator=g, device=DEV)
    x["k"] = hot.repeat(1, H).to(dtype)
    x["q"] = torch.nn.functional.one_hot(torch.randint(0, dk // 2, (T,), generator=g, device=DEV) * 2 + 1, dk).float().repeat(1, H).to(dtype)
    x["v"] = (x["v"].float() * least[at][:, None]).to(dtype)
    x["state"] = x["state"] * small[:, None]
    x["rate"] = torch.full((H,), 0.01, device=DEV)                               # rows stay within 2^-27 of their columns
    out, state = _run(x, st, H, H, dk, dv)
    ref, states = _exact(x, lens, H, H, dk, dv)
    assert _off(out, ref) < (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12)
    for r, S in states.items():
        row = (state[r].double() - S).norm(dim=-1) / S.norm(dim=-1).clamp_min(1e-30)
        assert float(row.max()) < 2.0 ** (-19 if noise else -20)
