"""The decode attention that gives a (sequence, kv head) one CTA: the same bits as norm, rotation, cache write, pages and merge one
launch after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,KV,HD,window,norm,rope,write", [(16, 8, 128, 0, True, True, True), (16, 8, 64, 100, True, True, True),
                                                             (16, 1, 128, 0, False, True, True), (24, 8, 128, 64, True, False, True),
                                                             (8, 8, 64, 0, False, False, True), (16, 4, 128, 70, True, True, False)])
def test_short_sequences_have_the_bits_of_the_separate_launches(H, KV, HD, window, norm, rope, write):
    """Lengths at a page's first and last row, of one page to four, padding rows, rows behind the last position no numbers."""
    from mynah_slm_b200.ops import kernels as k
    g = torch.Generator(device=DEV).manual_seed(H + KV)
    B = 480 // KV + 8
    lens = [[1, 64, 65, 128, 0, 129, 192, 193, 256, 37][b % 10] for b in range(B)]
    assert k.attn_decode_short(B, H, KV, 4) and not k.attn_decode_short(B, H, KV, 5) and not k.attn_decode_short(8, 8, 8, 4)
    # where a CTA a page or three launches are the faster form (figures at the rule)
    assert not k.attn_decode_short(28, 16, 8, 3) and not k.attn_decode_short(64, 16, 16, 1) and not k.attn_decode_short(250, 8, 8, 4)
    assert k.attn_decode_short(28, 16, 8, 1) and k.attn_decode_short(28, 64, 8, 4) and k.attn_decode_short(250, 16, 8, 4)
    indptr, ids = [0], []
    for n in lens:
        ids += list(range(len(ids), len(ids) + -(-n // 64)))
        indptr.append(len(ids))
    n_pages = len(ids)
    perm = torch.randperm(n_pages, generator=torch.Generator().manual_seed(1)).tolist()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)               # noqa: E731
    pt = k.PageTableView(i32(indptr), i32([perm[i] for i in ids]), i32([0] * B), n_pages)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    kc, vc = rand(n_pages, KV, 64, HD), rand(n_pages, KV, 64, HD)
    for b, n in enumerate(lens):                                                   # what is not there yet
        if n:
            last, row = perm[ids[indptr[b + 1] - 1]], (n - 1) % 64 + (0 if write else 1)
            kc[last, :, row:], vc[last, :, row:] = float("nan"), float("nan")
    qkv = rand(B, (H + 2 * KV) * HD)
    qg, kg = (rand(HD) + 1.0, rand(HD) + 1.0) if norm else (None, None)
    cos, sin = k.rope_table(300, HD, 1e4, DEV) if rope else (None, None)
    pos, kvl, status = i32([max(n - 1, 0) for n in lens]), i32(lens), i32([0])
    seq = i32([b if n else -1 for b, n in enumerate(lens)])
    scratch = torch.full((k.attn_decode_scratch_floats(B, H, HD, 4),), float("nan"), device=DEV)
    out, ref = (torch.full((B, H * HD), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    k1, v1, k2, v2, q2 = kc.clone(), vc.clone(), kc.clone(), vc.clone(), qkv.clone()
    k.attn_decode_fused(qkv, out, B, H, KV, HD, qg, kg, 1e-6, cos, sin, pos, k1, v1, write, kvl, pt, window, 4, scratch, None, status)
    k.qk_norm_rope_store(q2, H, KV, HD, qg, kg, 1e-6, cos, sin, HD if rope else 0, seq, pos, pt, k2 if write else None, v2 if write else None, status)
    k.attn_decode_tc(q2, ref, B, H, KV, HD, k2, v2, kvl, pt, window, 4, scratch, status)
    assert int(status.item()) == 0 and bool(torch.isfinite(out).all())
    assert torch.equal(out, ref) and torch.equal(k1.nan_to_num(5.0), k2.nan_to_num(5.0)) and torch.equal(v1.nan_to_num(5.0), v2.nan_to_num(5.0))
    # an index that must be refused is reported, and nothing is read or written there
    bad = k.PageTableView(pt.indptr, torch.full_like(pt.ids, n_pages), pt.base, n_pages)
    k.attn_decode_fused(qkv, out, B, H, KV, HD, qg, kg, 1e-6, cos, sin, pos, k1, v1, write, kvl, bad, window, 4, scratch, None, status)
    assert int(status.item()) & 1 and bool((out == 0).all())
