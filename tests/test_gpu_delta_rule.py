"""The gated delta rule on bfloat16 prompts: a sequence's bits do not depend on its company or on a step's capacities, and keys that
nearly agree cost no precision."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(T, H, G, dim, vd, overlap, low):
    gen = torch.Generator(device=DEV).manual_seed(dim + vd)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)                              # noqa: E731
    unit = lambda x: x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()                     # noqa: E731
    common = rand(1, G, dim) * overlap ** 0.5
    qn = unit(rand(T, G, dim) * (1.0 - overlap) ** 0.5 + common) * dim ** -0.5
    kn = unit(rand(T, G, dim) * (1.0 - overlap) ** 0.5 + common)
    g = low + (1.0 - low) * torch.rand((T, H), generator=gen, device=DEV)
    return qn, kn, rand(T, H, vd).to(torch.bfloat16), g, torch.sigmoid(rand(T, H) + 4.0), rand(8, H, dim, vd) * 0.1


def _run(x, rows, lengths, slots, max_q_len):
    from mynah_slm_b200.ops import kernels
    qn, kn, v, g, beta, state = x
    G, dim, H, vd = qn.shape[1], qn.shape[2], v.shape[1], v.shape[2]
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)                           # noqa: E731
    ctx = SimpleNamespace(cu_q=i32(cu), slots=i32(slots), B=len(lengths), max_q_len=max_q_len)
    state = state.clone()
    cut = lambda a: a[rows].reshape(cu[-1], -1).contiguous()                                 # noqa: E731
    o = kernels.delta_rule(cut(qn), cut(kn), cut(v), cut(g), cut(beta), state, ctx, H, G, dim, vd)
    return o.view(cu[-1], H, vd), state


@pytest.mark.parametrize("dim,vd", [(64, 64), (128, 128), (48, 20)])
def test_a_sequence_has_the_same_bits_in_any_step(dim, vd):
    """Three pieces in one step, each alone, and in a step whose longest piece is given as its padded rows (a captured step)."""
    lengths, slots = [20, 300, 1], [5, 0, 3]
    x = _inputs(sum(lengths), 4, 2, dim, vd, 0.2, 0.9)
    o, state = _run(x, slice(0, sum(lengths)), lengths, slots, max(lengths))
    at = 0
    for n, slot in zip(lengths, slots):
        for longest in (n, 4096):
            one, s = _run(x, slice(at, at + n), [n], [slot], longest)
            assert torch.equal(one, o[at:at + n]) and torch.equal(s[slot], state[slot])
        at += n


@pytest.mark.parametrize("overlap", [0.9, 0.99])
@pytest.mark.parametrize("low", [0.5, 0.99])
def test_keys_that_nearly_agree(overlap, low):
    """beta near 1 and keys with a cosine of `overlap`: every write takes back most of what the last one left. A token's sums are
    short chains (four additions, then trees over four partial sums and eight lanes), so outputs lie about one rounding of 32 bits
    (6e-8) from 64 bits, states, which gather a rounding a token, a few: 0.6e-7 to 0.8e-7 and 0.5e-7 to 2.9e-7 in the same order of
    operations on the CPU, with some room above."""
    T, H, G, dim, vd = 384, 4, 2, 128, 64
    x = _inputs(T, H, G, dim, vd, overlap, low)
    o, state = _run(x, slice(0, T), [T], [2], T)
    qn, kn, v, g, beta, s0 = (a.double() for a in x)
    qn, kn, S = qn.repeat_interleave(H // G, 1), kn.repeat_interleave(H // G, 1), s0[2]
    ref = []
    for t in range(T):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, kn[t]))
        S = S + kn[t][:, :, None] * u[:, None, :]
        ref.append(torch.einsum("hdv,hd->hv", S, qn[t]))
    err = lambda a, r: float((a.double() - r).norm() / r.norm())                             # noqa: E731
    assert err(o, torch.stack(ref)) < 2e-7 and err(state[2], S) < 6e-7
