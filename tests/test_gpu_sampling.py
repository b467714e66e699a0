"""The one-launch draw against the plain sampler, at the edges of its routes: lists of candidates (a bound from the groups'
maxima, many equal logits, more places than finite logits), rows that fit shared memory or do not, rows that no 16-byte load
can start at, and the penalties and the ring inside the launch."""
import numpy as np
import pytest
import torch

from plain.sampler import PlainSampler

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rows(rng, V, kind):
    lg = (rng.standard_normal((4, V)) * 2.0).astype(np.float32)
    if kind == "equal":                                    # far more than 256 logits share the largest values
        lg = np.round(lg)
        lg[1, :] = 0.5
    elif kind == "masked":                                 # fewer finite logits than places
        lg[:, 7:] = -np.inf
        lg[2, V - 1] = 3.0
    elif kind == "crowd":                                  # 400 of the largest probabilities share their leading eleven bits
        lg = np.minimum(lg, 2.0)
        for b in range(4):
            lg[b, rng.permutation(V)[:400]] = 9.0 + 2e-4 * rng.permutation(400)
    elif kind == "sharp":                                  # all but a few exponentials vanish
        lg *= 40.0
    return lg


@pytest.mark.parametrize("V,kind", [(300, "plain"), (32767, "plain"), (32768, "plain"), (65541, "plain"), (32771, "equal"),
                                    (40000, "equal"), (1003, "equal"), (50000, "masked"), (900, "masked"), (33000, "sharp"),
                                    (400001, "plain"), (60000, "plain"), (400004, "plain"), (5000, "crowd"), (40000, "crowd")])
@pytest.mark.parametrize("temp,top_k,top_p,min_p", [(0.6, 20, 0.95, 0.0), (1.0, 128, 0.9, 0.0), (1.0, 129, 1.0, 0.0),
                                                    (0.8, 0, 0.9, 0.0), (1.0, 0, 1.0, 0.1), (0.9, 257, 1.0, 0.0), (0.0, 20, 1.0, 0.0)])
def test_routes_match_plain_sampler(V, kind, temp, top_k, top_p, min_p):
    """The same token from the same generator state. Equal logits make equal probabilities, which ids tell apart."""
    from mynah_slm_b200.ops import kernels
    rng = np.random.default_rng(V + top_k)
    plain = [PlainSampler(temp=temp, top_k=top_k, top_p=top_p, min_p=min_p, rng_state=101 + i) for i in range(4)]
    state = torch.tensor([101 + i for i in range(4)], dtype=torch.int64, device=DEV)
    params = torch.tensor([temp, top_p, min_p, float(top_k), 1.0, 0.0, 0.0, 0.0], dtype=torch.float32, device=DEV)
    for _ in range(3):
        lg = _rows(rng, V, kind)
        with np.errstate(all="ignore"):
            want = [p.sample(lg[b].copy()) for b, p in enumerate(plain)]
        got = kernels.sample(torch.from_numpy(lg.copy()).to(DEV), params, state, None).cpu().tolist()
        assert got == want


@pytest.mark.parametrize("V,rows", [(30000, 160), (200003, 24)])
def test_many_rows_draw_as_few_do(V, rows):
    """Steps of more CTAs than SMs leave long rows where they are, small ones take them into shared memory: the same tokens."""
    from mynah_slm_b200.ops import kernels
    lg = torch.randn((rows, V), generator=torch.Generator(device=DEV).manual_seed(V), device=DEV) * 2.0
    for temp, top_k in ((0.0, 0), (0.9, 20), (0.9, 200), (1.0, 0)):
        params = torch.tensor([temp, 0.9, 0.0, float(top_k), 1.0, 0.0, 0.0, 0.0], dtype=torch.float32, device=DEV)
        many, few = (torch.arange(5, 5 + rows, dtype=torch.int64, device=DEV) for _ in range(2))
        got = kernels.sample(lg.clone(), params, many, None)
        for at in range(0, rows, 6):
            assert torch.equal(kernels.sample(lg[at:at + 6].clone(), params, few[at:at + 6], None), got[at:at + 6])
        assert torch.equal(many, few)


def test_a_row_of_very_many_logits():
    """Tens of millions of equal probabilities a digit: their summed masses exceed what counts and low bits can hold in 32 bits. Half of
    the row is e times as likely as the other half; the walk goes through the first half by id, then through the second. A place
    may be off by as much as the two sums' roundings make of 40 million (2^-22 of the place: 10)."""
    from mynah_slm_b200.ops import kernels
    half = 20_000_003
    lg = torch.zeros((1, 2 * half), device=DEV)
    lg[0, half:] = -1.0
    params = torch.tensor([1.0, 1.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0], dtype=torch.float32, device=DEV)
    share = 1.0 / (1.0 + np.exp(-1.0))
    sides = set()
    for seed in range(1, 9):
        z = (seed + 0x9E3779B97F4A7C15) & (2 ** 64 - 1)
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
        u = ((z ^ (z >> 31)) >> 11) / 2.0 ** 53
        want = u / share * half if u < share else half + (u - share) / (1.0 - share) * half
        got = int(kernels.sample(lg.clone(), params, torch.tensor([seed], dtype=torch.int64, device=DEV), None).item())
        assert abs(got - want) < 32, (seed, got, want)
        sides.add(u < share)
    assert len(sides) == 2


@pytest.mark.parametrize("V", [500, 40002])
@pytest.mark.parametrize("temp,top_k", [(0.0, 0), (0.9, 20), (0.9, 0)])
def test_penalties_and_ring_inside_the_draw(V, temp, top_k):
    """Draw after draw with a window of five tokens: the ring holds repeats, and what it holds decides the next draw."""
    from mynah_slm_b200.ops import kernels
    rng, W, stride, B = np.random.default_rng(3), 5, 8, 3
    plain = [PlainSampler(temp=temp, top_k=top_k, top_p=0.95, repeat_penalty=1.4, freq_penalty=0.3, presence_penalty=0.2,
                          penalty_window=W, rng_state=7 + i) for i in range(B)]
    ring = tuple(torch.zeros(shape, dtype=torch.int32, device=DEV) for shape in ((B + 1, stride), (B + 1,), (B + 1,)))
    state = torch.tensor([7 + i for i in range(B)] + [99], dtype=torch.int64, device=DEV)
    params = torch.tensor([temp, 0.95, 0.0, float(top_k), 1.4, 0.3, 0.2, float(W)], dtype=torch.float32, device=DEV)
    slots = torch.tensor([0, 1, -1, 2], dtype=torch.int32, device=DEV)
    base = rng.standard_normal((4, V)).astype(np.float32)
    base[:, [3, V // 2, V - 2]] += 6.0                                            # three favourites: tokens come again
    for _ in range(14):
        lg = base + 0.3 * rng.standard_normal((4, V)).astype(np.float32)
        want = [p.sample(lg[row].copy()) for p, row in zip(plain, (0, 1, 3))]
        got = kernels.sample(torch.from_numpy(lg.copy()).to(DEV), params, state, slots, ring=ring).cpu().tolist()
        assert [got[0], got[1], got[3]] == want
        for p, t in zip(plain, want):
            p.accept(t)
    assert ring[1].cpu().tolist() == [W] * B + [0] and int(state[B]) == 99
