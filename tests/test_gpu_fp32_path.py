"""The 32-bit path's kernels where their routes meet: whichever a size takes, the bits are the same, since every sum walks the
same order."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("K", [20, 64, 512, 516, 1000, 2304])
@pytest.mark.parametrize("M,N", [(1, 1185), (2, 1184), (3, 40), (16, 1000), (17, 33), (33, 1024), (40, 1030), (161, 1025), (300, 2100),
                                 (700, 4100)])
def test_products_have_the_same_bits_by_every_route(M, N, K):
    """Few rows with long and short slabs, tiles of both sizes, against the general kernel (rows that no 16-byte load can start at)."""
    from mynah_slm_b200.ops.lib import call, ptr, stream_ptr
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    a, w = (torch.randn((r, K), generator=g, device=DEV) for r in (M, N))
    out, ref = (torch.full((M, N + 3), 7.0, device=DEV) for _ in range(2))
    call("mynah_gemm_f32", ptr(a), ptr(w), ptr(out), M, N, K, K, K, N + 3, stream_ptr())
    a1 = torch.nn.functional.pad(a, (0, 1)).contiguous()                          # row stride K + 1: not a multiple of four
    call("mynah_gemm_f32", ptr(a1), ptr(w), ptr(ref), M, N, K, K + 1, K, N + 3, stream_ptr())
    assert torch.equal(out, ref) and bool((out[:, N:] == 7.0).all())
    exact = a.double() @ w.double().T
    assert float((out[:, :N].double() - exact).norm() / exact.norm()) < K ** 0.5 * 2.0 ** -23


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,KV,HD,window", [(4, 2, 8, 0), (4, 4, 64, 20), (2, 1, 128, 0), (3, 1, 136, 0), (2, 2, 256, 70)])
def test_prompt_attention_with_and_without_vectors(dtype, H, KV, HD, window):
    """Query rows on 16-byte boundaries or off them: the same bits. Keys and values behind the last position are no numbers."""
    from mynah_slm_b200.ops import kernels
    g = torch.Generator(device=DEV).manual_seed(HD)
    lens_q, past = [1, 16, 17, 50], [130, 0, 63, 5]
    T, n_pages = sum(lens_q), 12
    q = torch.randn((T, H * HD), generator=g, device=DEV).to(dtype)
    kc, vc = (torch.randn((n_pages, KV, 64, HD), generator=g, device=DEV).to(dtype) for _ in range(2))
    ids, indptr = [], [0]
    for n, p in zip(lens_q, past):
        pages = [len(ids) + i for i in range(-(-(n + p) // 64))]
        for c in (kc, vc):
            c[pages[-1], :, (n + p - 1) % 64 + 1:] = float("nan")
        ids += pages
        indptr.append(len(ids))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)               # noqa: E731
    pt = kernels.PageTableView(i32(indptr), i32(ids), i32([0] * 4), n_pages)
    cu, kvl, status = i32(np.cumsum([0] + lens_q).tolist()), i32([n + p for n, p in zip(lens_q, past)]), i32([0])
    outs = []
    for pad in (0, 1):
        rows = torch.nn.functional.pad(q, (0, pad)).contiguous()
        out = torch.zeros((T, H * HD), dtype=dtype, device=DEV)
        kernels.attn_prefill_generic(rows, out, 4, max(lens_q), H, KV, HD, kc, vc, cu, kvl, pt, window, status)
        outs.append(out)
    assert int(status.item()) == 0 and bool(torch.isfinite(outs[0]).all()) and torch.equal(outs[0], outs[1])
