"""A decode step's causal convolution: rows and weights fetched together have the bits of the general kernel."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("x_dtype,out_dtype,w_dtype", [(torch.float32, torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.bfloat16, torch.float32),
                                                       (torch.float32, torch.float32, torch.float32)])
@pytest.mark.parametrize("C,taps,act,add,bias", [(1024, 3, None, True, False), (264, 4, "silu", False, True), (2048, 2, "silu", True, True),
                                                 (8, 3, None, False, False), (512, 5, None, True, False), (64, 1, "silu", False, True)])
def test_decode_step_has_the_general_kernels_bits(x_dtype, out_dtype, w_dtype, C, taps, act, add, bias):
    """Rows on 16-byte boundaries, and the same rows one element off them; padding rows and a sequence without a slot."""
    from mynah_slm_b200.ops import kernels
    g = torch.Generator(device=DEV).manual_seed(C + taps)
    B, n_slots = 5, 6
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)                    # noqa: E731
    x, w = rand(B, C).to(x_dtype), rand(C, taps).to(w_dtype)
    b = rand(C).to(w_dtype) if bias else None
    state0 = rand(n_slots + 1, max(taps - 1, 1), C) if taps > 1 else None
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)               # noqa: E731
    ctx = SimpleNamespace(tok_seq=i32([0, 1, 2, -1, 4]), cu_q=i32([0, 1, 2, 3, 4, 5]), slots=i32([4, 0, -1, 2, 5]), B=B, T=B,
                          is_decode=True, max_q_len=1)
    outs = []
    for off in (0, 1):
        rows = torch.zeros((B, C + 8), dtype=x_dtype, device=DEV)
        rows[:, off:off + C] = x
        state = state0.clone() if taps > 1 else None
        out = kernels.causal_conv(rows[:, off:off + C], w, b, state, ctx, out_dtype, act=act, add_input=add)
        outs.append((out, state))
    assert torch.equal(outs[0][0], outs[1][0])
    if taps > 1:                                             # (the last row of the state belongs to no sequence)
        assert torch.equal(outs[0][1][:n_slots], outs[1][1][:n_slots])
        assert torch.equal(outs[0][1][[1, 2, 3]], state0[[1, 2, 3]])
