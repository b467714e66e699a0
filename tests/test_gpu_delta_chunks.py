"""The gated delta rule chunk by chunk against the recurrence token by token in 64 bits, and against the kernel that walks tokens."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _exact(qn, kn, v, g, beta, S, H, G):
    """One sequence in 64 bits: rows [n, heads, d]; S [H, dim, vd]."""
    kn, qn = (x.double().repeat_interleave(H // G, 1) for x in (kn, qn))
    v, g, beta, S, out = v.double(), g.double(), beta.double(), S.double(), []
    for t in range(v.shape[0]):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, kn[t]))
        S = S + kn[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hdv,hd->hv", S, qn[t]))
    return torch.stack(out), S


@pytest.mark.parametrize("H,G,dim,vd,lengths,low", [(4, 2, 128, 128, [64, 65, 1, 200, 129], 0.5), (2, 1, 32, 70, [130, 1, 140], 0.9),
                                                    (3, 3, 96, 20, [500], 0.99), (64, 64, 128, 128, [1500, 63, 900], 0.9),
                                                    (2, 2, 64, 130, [300, 40], 0.0), (16, 8, 128, 128, [2048, 1600], 0.98)])
def test_chunks_match_the_recurrence(H, G, dim, vd, lengths, low):
    """Edges of chunks and tiles, strong and weak decays (with a decay of zero among them), states that are not zero, a sequence
    without a slot (left alone), padding rows, steps of several passes. Both kernels sum in fp32: 2e-5 as for the tokens' kernel,
    and no further off than twice that kernel."""
    from mynah_slm_b200.ops import kernels
    gen = torch.Generator(device=DEV).manual_seed(dim + vd)
    T, B = sum(lengths) + 3, len(lengths)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)                  # noqa: E731
    unit = lambda x: x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()         # noqa: E731
    qn, kn = unit(rand(T, G, dim)) * dim ** -0.5, unit(rand(T, G, dim) + 0.5)     # (keys that overlap)
    v = rand(T, H, vd).to(torch.bfloat16)
    g = low + (1.0 - low) * torch.rand((T, H), generator=gen, device=DEV)
    g[T // 3] = 0.0 if low == 0.0 else 1.0
    beta = torch.sigmoid(2.0 * rand(T, H))
    slots = [B - i for i in range(B)]
    if B > 2:
        slots[1] = -1
    state0 = rand(B + 2, H, dim, vd) * 0.3
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)               # noqa: E731
    ctx = SimpleNamespace(cu_q=i32(cu), slots=i32(slots), B=B, max_q_len=max(lengths))
    outs = []
    for least in (1, 0):
        before = kernels.delta_chunk_min(least)
        try:
            st = state0.clone()
            o = kernels.delta_rule(qn.reshape(T, -1), kn.reshape(T, -1), v.reshape(T, -1), g, beta, st, ctx, H, G, dim, vd)
            outs.append((o.view(T, H, vd), st))
        finally:
            kernels.delta_chunk_min(before)
    kept = [s for s in range(B + 2) if s not in slots]
    assert torch.equal(outs[0][1][kept], state0[kept])
    err = lambda a, r: float((a.double() - r).norm() / r.norm())                 # noqa: E731
    for i, (n, slot) in enumerate(zip(lengths, slots)):
        if slot < 0:
            continue
        rows = slice(cu[i], cu[i + 1])
        ref, S = _exact(qn[rows], kn[rows], v[rows], g[rows], beta[rows], state0[slot], H, G)
        for (chunk, token), r in ((((outs[0][0][rows], outs[1][0][rows])), ref), ((outs[0][1][slot], outs[1][1][slot]), S)):
            a, b = err(chunk, r), err(token, r)
            print(f"n={n}: chunks {a:.2e}, tokens {b:.2e}")
            assert a < 2e-5 and a < 2.0 * b + 1e-7
