"""A decode step of the retention in one launch: the bits of preparation, scan and gated norm one after the other."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,dim,vd,rot,interleaved", [(16, 128, 128, 128, False), (3, 16, 24, 16, True), (2, 33, 70, 6, False),
                                                      (2, 96, 100, 32, True), (1, 64, 256, 64, False), (4, 20, 512, 0, False)])
def test_step_has_the_bits_of_the_three_launches(dtype, H, dim, vd, rot, interleaved):
    """Padding rows give zeros and leave every state alone; a position beyond the table is reported."""
    from mynah_slm_b200.ops import kernels as k
    from mynah_slm_b200.parts.position import rotary_frequencies
    g = torch.Generator(device=DEV).manual_seed(dim + vd)
    B, n = 6, 2 * H * dim + 2 * H * vd
    p = torch.randn((B, n + 8), generator=g, device=DEV).to(dtype)
    cos = sin = None
    if rot:
        f, mult = rotary_frequencies(rot, 50.0, None)
        cos, sin = k.rope_table_freqs(64, f, mult, DEV)
    decay = torch.linspace(0.8, 1.0, H, device=DEV)
    state0 = torch.randn((8, H, dim, vd), generator=g, device=DEV)
    w = torch.ones((vd,), device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)               # noqa: E731
    ctx = SimpleNamespace(B=B, T=B, is_decode=True, max_q_len=1, tok_seq=i32([0, 1, -1, 3, 4, 5]), tok_pos=i32([3, 0, 0, 63, 17, 40]),
                          cu_q=i32([0, 1, 2, 2, 3, 4, 5]), slots=i32([4, 1, -1, 6, 0, 2]), status=i32([0]))
    assert k.retention_step_ok(p, ctx, H, dim, vd) == (B * H >= 32)
    at = (0, H * dim, 2 * H * dim, 2 * H * dim + H * vd)
    st = state0.clone()
    out = k.retention_step(p, *at, cos, sin, rot, interleaved, dim ** -0.5, decay, st, w, 1e-5, ctx, H, dim, vd)
    ref_ctx = SimpleNamespace(**{**vars(ctx), "cu_q": i32([0, 1, 2, 3, 4, 5, 6])})
    st2 = state0.clone()
    qn, kn = k.retention_prep(p, at[0], at[1], H, dim, cos, sin, rot, interleaved, dim ** -0.5, ref_ctx)
    o = k.retention_scan(qn, kn, p, at[2], decay, st2, ref_ctx, H, dim, vd)
    ref = k.gated_rmsnorm(o, p[:, at[3]:at[3] + H * vd], w, H, vd, 1e-5)
    rows = [0, 1, 3, 4, 5]
    assert torch.equal(out[rows], ref[rows]) and bool((out[2] == 0).all()) and torch.equal(st, st2)
    assert int(ctx.status.item()) == 0
    if rot:
        ctx.tok_pos = i32([3, 0, 0, 64, 17, 40])
        before = st.clone()
        k.retention_step(p, *at, cos, sin, rot, interleaved, dim ** -0.5, decay, st, w, 1e-5, ctx, H, dim, vd)
        assert int(ctx.status.item()) == 2 and torch.equal(st[6], before[6])
