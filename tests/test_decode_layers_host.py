"""The host's side of the one-launch decode step (ops/decode_layers.py), without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from mynah_slm_b200.ops import decode_layers
from mynah_slm_b200.ops.lib import KernelError


class Rows:
    """Stands for a tensor on the device."""
    def __init__(self, shape, dtype=torch.float32, is_cuda=True, contiguous=True):
        self.shape, self.dtype, self.is_cuda, self.contiguous = torch.Size(shape), dtype, is_cuda, contiguous

    def is_contiguous(self):
        return self.contiguous

    def dim(self):
        return len(self.shape)

    def data_ptr(self):
        return 0


@pytest.fixture
def steps(monkeypatch):
    """A plan of two layers of 64 whose launches are noted instead of made."""
    made = []
    monkeypatch.setattr(decode_layers, "offer", lambda name, *args: made.append((name, args)) is None)
    monkeypatch.setattr(decode_layers, "stream_ptr", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    sizes = dict(D=64, H=1, KV=1, HD=64, F=64, eps=1e-6, qk_eps=1e-6, gain_dtype=0, qk_dtype=0, cos=None, sin=None)
    cache = torch.zeros((2, 4, 1, 64, 64), dtype=torch.bfloat16)
    plan = decode_layers.DecodeLayers([[0] * 12] * 2, sizes, [(cache, cache, 0)], torch.device("cpu"))
    return plan, made


def _ctx(rows, splits=1):
    pages = SimpleNamespace(indptr=Rows([rows + 1]), ids=Rows([4]), base=Rows([rows]), n_pages=4)
    return SimpleNamespace(T=rows, is_decode=True, decode_splits=splits, pages=[pages], kv_len=Rows([rows]), status=Rows([1]))


RUNTIME = SimpleNamespace(sm_count=148)


@pytest.mark.parametrize("x", [Rows([2, 64], torch.bfloat16), Rows([2, 64], is_cuda=False), Rows([2, 64], contiguous=False), Rows([128]),
                               Rows([2, 32]), Rows([1, 64]), Rows([2, 128])])
def test_other_rows_are_refused(steps, x):
    """What an embedding returns is checked before the kernel writes to it."""
    plan, made = steps
    with pytest.raises(KernelError, match="residual"):
        plan.forward(x, _ctx(2), RUNTIME)
    assert not made
    plan.forward(Rows([2, 64]), _ctx(2), RUNTIME)
    assert [name for name, _ in made] == ["mynah_decode_layers"]


def test_tags_begin_again_before_they_wrap(steps):
    """Six tags a launch of two layers. Before a launch would pass the limit, everything that carries tags is cleared: the words,
    the partial results at hand and those that an older captured step still uses, and the count in the kernel's own keeping."""
    plan, made = steps
    plan.TAG_LIMIT = 20
    plan.forward(Rows([1, 64]), _ctx(1, splits=2), RUNTIME)
    small = plan.part
    plan.forward(Rows([1, 64]), _ctx(1, splits=640), RUNTIME)
    assert plan.part is not small
    tagged = (plan.sync, plan.words, plan.part, small)
    for t in tagged:
        t.fill_(7)
    plan.forward(Rows([1, 64]), _ctx(1), RUNTIME)                    # tags 13 to 18
    assert all(bool((t == 7).all()) for t in tagged)
    plan.count_launch()                                              # 24 would be too many
    assert not any(bool(t.any()) for t in tagged)
    plan.sync.fill_(7)
    plan.count_launch()
    plan.count_launch()
    assert bool((plan.sync == 7).all())
    plan.count_launch()
    assert not bool(plan.sync.any())


def test_partial_results_take_room_by_runs_and_rows(steps):
    """One sequence decoded from its first page to its 640th, then a batch of eight: what is held, outgrown buffers included, stays
    within four times what the last step needs (16 times that, and 80 times as much outgrown, with a row a page for eight rows)."""
    plan, made = steps
    for splits in range(1, 641):
        plan.forward(Rows([1, 64]), _ctx(1, splits=splits), RUNTIME)
    held = lambda: plan.part.numel() + sum(t.numel() for t in plan._retired)       # noqa: E731
    assert 160 * 66 <= plan.part.numel() <= held() <= 4 * 160 * 66
    plan.forward(Rows([8, 64]), _ctx(8, splits=640), RUNTIME)
    assert 8 * 160 * 66 <= plan.part.numel() <= held() <= 4 * 8 * 160 * 66


def test_runs_of_every_page_count_fit():
    """A sequence of up to 16 pages is cut in twos, a longer one in fours; none has more runs than a step of its splits holds."""
    for s in range(1, 700):
        assert decode_layers.most_runs(s) == max(-(-n // (2 if n <= 16 else 4)) for n in range(1, s + 1))


def test_padded_and_unpadded_steps_take_the_same_route(steps):
    """A captured step has its rows padded to a power of two and its page splits to one or to a multiple of sixteen; the rule
    gives the same answer for the uncaptured step."""
    from mynah_slm_b200.engine.engine import Engine
    plan, made = steps
    for columns, dim, pages in [(c, 64, 1) for c in (64, 9728, 12288, 20000)] + [(64, d, p) for d in (64, 128) for p in range(1, 800, 3)]:
        plan.sizes["F"], plan.sizes["HD"] = columns, dim
        for rows in range(1, 20):
            assert plan.takes(_ctx(rows, pages)) == plan.takes(_ctx(Engine._bucket(rows), max(4, Engine._pages_bucket(pages))))


def test_long_caches_take_the_layers_one_by_one(steps):
    """Where the one launch measured slower; not where the layers one by one would have the general attention kernel only."""
    plan, made = steps
    for heads, dim, rows, pages, one in [(4, 128, 8, 368, True), (4, 128, 8, 384, False), (16, 128, 8, 368, True), (16, 128, 8, 384, False), (16, 128, 4, 736, True), (16, 128, 1, 1008, True),
                                         (16, 64, 8, 224, True), (16, 64, 8, 240, False), (32, 128, 8, 512, False), (32, 128, 8, 528, True),
                                         (64, 64, 8, 48, True), (64, 64, 8, 64, False), (64, 64, 4, 112, True), (64, 64, 1, 448, True)]:
        plan.sizes.update(H=heads, KV={4: 2, 64: 32}.get(heads, 8), HD=dim)
        assert plan.takes(_ctx(rows, pages)) is one


def test_a_declined_launch_is_not_offered_again(steps, monkeypatch):
    """Fewer SMs to use than the device has: the step goes on layer by layer, and so do those after it."""
    plan, made = steps
    assert plan.takes(_ctx(1)) and plan.forward(Rows([1, 64]), _ctx(1), RUNTIME) is True
    monkeypatch.setattr(decode_layers, "offer", lambda name, *args: False)
    assert plan.takes(_ctx(1)) and plan.forward(Rows([1, 64]), _ctx(1), RUNTIME) is False
    assert not plan.takes(_ctx(1))
    with pytest.raises(KernelError, match="declined behind"):
        plan.forward(Rows([1, 64]), _ctx(1), RUNTIME, range(1, 2))


def test_what_an_entry_point_may_answer(monkeypatch):
    """0: launched; 1: declined, not counted as a launch; anything else is an error."""
    from mynah_slm_b200.ops import lib
    answers = SimpleNamespace(entry=lambda rc: rc, mynah_last_error=lambda: b"sizes are not supported")
    monkeypatch.setattr(lib, "load", lambda: answers)
    before = lib.launch_count()
    assert lib.offer("entry", 0) is True and lib.launch_count() == before + 1
    assert lib.offer("entry", 1) is False and lib.launch_count() == before + 1
    with pytest.raises(KernelError, match="not supported"):
        lib.offer("entry", -1)
    lib.add_launches(-1)
