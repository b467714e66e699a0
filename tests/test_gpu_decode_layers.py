"""Decode steps whose layers run in one launch (ops/decode_layers.py), against the plain implementation and against the
layers run one by one."""
import numpy as np
import pytest
import torch

from helpers import BF16_REL, assert_close, make_folder
from plain.model import PlainQwen3

pytestmark = pytest.mark.gpu


def _cfg(layers, hidden, heads, kv, dim, ffn, window=None):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=layers, hidden_size=hidden,
                num_attention_heads=heads, num_key_value_heads=kv, head_dim=dim, intermediate_size=ffn, vocab_size=515,
                rope_theta=10000.0, rms_norm_eps=1e-6, tie_word_embeddings=True, max_position_embeddings=4096, hidden_act="silu",
                attention_bias=False, rope_scaling=None, use_sliding_window=window is not None, sliding_window=window,
                max_window_layers=1, eos_token_id=1)


# one sequence of a single page and several rows that are not a power of two; pages that end where the step begins or ends
# (63 -> 64 -> 65); more units a CTA than are summed at a time (feed-forwards of 8,192); columns that are no multiple of a
# slot's 1,024 or of a warp's 128; groups of 1, 2, 3, 4 and 8 query heads; windows shorter than a page and longer; 768 runs of
# pages, five a CTA
CASES = [
    (_cfg(2, 64, 1, 1, 64, 64), [5]),
    (_cfg(2, 192, 6, 2, 64, 320), [63, 1, 130]),
    (_cfg(3, 1088, 8, 1, 64, 1216), [64, 3, 700, 65, 128, 62, 191]),
    (_cfg(2, 1024, 16, 8, 128, 3072), [62, 126, 500, 1, 1000, 333, 64, 129]),
    (_cfg(2, 2560, 8, 2, 128, 8192), [200, 31]),
    (_cfg(3, 256, 4, 4, 128, 8192, window=20), [300, 19, 70]),
    (_cfg(3, 512, 34, 17, 64, 704, window=100), [700, 99, 101, 230]),
    (_cfg(2, 512, 32, 32, 64, 512), [620, 610, 600, 590, 580, 570, 639, 560]),
]
# And with few CTAs, so that each has several of everything: both groups of warps at work and passing over each other's pages, more
# jobs than the table holds (102 on three CTAs), queries kept from job to job, several merges, units in several turns.
FEW = [(1, 3), (2, 3), (2, 20), (3, 20), (5, 3), (6, 3), (6, 20), (7, 20)]


@pytest.mark.parametrize("i,ctas", [(i, None) for i in range(len(CASES))] + FEW)
def test_one_launch_a_step(tmp_path, i, ctas):
    from mynah_slm_b200.engine.engine import Engine, StepEntry
    cfg, lens = CASES[i]
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=i)
    plain = PlainQwen3.from_folder(folder)
    rng = np.random.default_rng(i)
    steps = 4
    seqs = [rng.integers(0, cfg["vocab_size"], size=n + steps).tolist() for n in lens]
    refs = [plain.forward(q) for q in seqs]
    room = sum(-(-(n + steps) // 64) * 64 for n in lens)
    rows = {}
    for one in (True, False):
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=room + 64, max_seqs=len(lens) + 1)
        assert eng.decode_layers is not None
        if ctas is not None:
            eng.runtime.sm_count = ctas
        took = []
        takes = eng.decode_layers.takes
        eng.decode_layers.takes = lambda ctx: took.append(takes(ctx) and one) or took[-1]
        # what a page holds beyond its sequence's end must not matter
        for t in eng.cache.keys + eng.cache.values:
            t.fill_(float("nan"))
        slots = [eng.open_sequence() for _ in lens]
        eng.step([StepEntry(s, q[:n], ()) for s, q, n in zip(slots, seqs, lens)])
        rows[one] = [eng.step([StepEntry(s, [q[n + t]], (0,)) for s, q, n in zip(slots, seqs, lens)]).cpu().numpy() for t in range(steps)]
        eng.check_status()
        assert any(took) == one
        if one:
            # a step again, with the rows in another order: a sequence's bits do not depend on its row
            for s in slots:
                eng.close_sequence(s)
            slots = [eng.open_sequence() for _ in lens]
            eng.step([StepEntry(s, q[:n], ()) for s, q, n in zip(slots, seqs, lens)])
            back = eng.step([StepEntry(s, [q[n]], (0,)) for s, q, n in list(zip(slots, seqs, lens))[::-1]]).cpu().numpy()
            assert np.array_equal(back[::-1], rows[True][0])
    for t in range(steps):
        for b, n in enumerate(lens):
            assert_close(refs[b][n + t][None], rows[True][t][b][None], BF16_REL, f"one launch, sequence {b}, step {t}")
            assert_close(refs[b][n + t][None], rows[False][t][b][None], BF16_REL, f"layer by layer, sequence {b}, step {t}")


def test_a_row_beyond_the_splits_is_left_alone(tmp_path, monkeypatch):
    """A sequence with more pages than the launch was given splits: reported at once, its neighbour as ever."""
    from mynah_slm_b200.engine.engine import Engine, EngineError, StepEntry
    cfg = _cfg(2, 256, 4, 2, 64, 320)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=3)
    seqs = [np.random.default_rng(n).integers(0, cfg["vocab_size"], size=n + 1).tolist() for n in (300, 40)]
    rows = []
    for splits in (5, 1):
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=512, max_seqs=2, use_graphs=False)
        slots = [eng.open_sequence() for _ in seqs]
        eng.step([StepEntry(s, q[:-1], ()) for s, q in zip(slots, seqs)])
        eng.check_status()
        monkeypatch.setattr(Engine, "_decode_pages", staticmethod(lambda n, splits=splits: splits))
        rows.append(eng.step([StepEntry(s, q[-1:], (0,)) for s, q in zip(slots, seqs)]).cpu().numpy()[1])
        if splits == 5:
            eng.check_status()
        else:
            with pytest.raises(EngineError, match="refused an index: a decode launch too small for a sequence$"):
                eng.check_status()
    assert np.array_equal(*rows)


def test_tags_begin_again(tmp_path):
    """Steps across the point where the tags begin again, captured, looped and launched: the same bits."""
    from mynah_slm_b200.engine.engine import Engine, StepEntry
    cfg = _cfg(2, 256, 4, 2, 64, 320)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=3)
    toks = np.random.default_rng(0).integers(0, cfg["vocab_size"], size=330).tolist()
    rows = []
    for graphs, limit in ((True, None), (True, 20), (False, 20)):
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=512, max_seqs=2, use_graphs=graphs)
        if limit is not None:
            eng.decode_layers.TAG_LIMIT = limit                      # three launches of six tags
        slot = eng.open_sequence()
        eng.step([StepEntry(slot, toks[:310], ())])
        rows.append([eng.step([StepEntry(slot, [t], (0,))]).cpu().numpy() for t in toks[310:]])
        if graphs:
            rows[-1].append(eng.decode_loop([slot], [5], 9).cpu().numpy())
            assert (int(eng.decode_layers.sync[0]) <= 18) == (limit is not None)
        eng.check_status()
    for a, b in ((rows[0], rows[1]), (rows[0][:20], rows[2])):
        assert len(a) == len(b) and all(np.array_equal(u, v) for u, v in zip(a, b))


def test_a_sequence_has_the_same_bits_in_every_batch_of_the_one_launch(tmp_path, monkeypatch):
    """Alone and with one, two, three and seven others, captured (padded to a bucket) and launched, among them sequences on both
    sides of the page count that decides how long the attention's runs are. What is compared are the logits behind the layers:
    the head's product is the same for every number of rows up to 16."""
    from mynah_slm_b200.engine import engine as engine_module
    from mynah_slm_b200.engine.engine import Engine, StepEntry
    monkeypatch.setattr(engine_module, "PROMPT_GRAPH_MAX_ROWS", 0)   # every prompt by the same launches
    cfg = _cfg(2, 512, 8, 4, 128, 704)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=5)
    lens = [700, 1500, 1024, 1023, 3, 64, 200, 1100]                 # (1,024 + 1 positions are the first of seventeen pages)
    rng = np.random.default_rng(0)
    seqs = [rng.integers(0, cfg["vocab_size"], size=n + 1).tolist() for n in lens]
    got = {}
    for graphs in (True, False):
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=7168, max_seqs=8, use_graphs=graphs)
        for who in ([0], [1], [2], [3], [4], [0, 1], [2, 0, 3], [7, 1, 4, 0], list(range(8)), [3, 2, 1, 0, 6], [2, 1]):
            slots = [eng.open_sequence() for _ in who]
            for s, i in zip(slots, who):                             # (one by one: a prompt's bits may depend on its batch)
                eng.step([StepEntry(s, seqs[i][:-1], ())])
            rows = eng.step([StepEntry(s, seqs[i][-1:], (0,)) for s, i in zip(slots, who)]).cpu().numpy()
            for i, row in zip(who, rows):
                assert np.array_equal(got.setdefault(i, row), row), (graphs, who, i)
            for s in slots:
                eng.close_sequence(s)
        eng.check_status()


def test_what_a_step_leaves_does_not_depend_on_what_is_asked_of_it(tmp_path):
    """The same tokens with logits wanted, with none wanted and with taps: the same bits in the cache, and the logits' too."""
    from mynah_slm_b200.engine.engine import Engine, StepEntry
    cfg = _cfg(3, 512, 8, 4, 64, 704, window=100)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=6)
    lens, steps = [130, 700, 64, 3, 5], 6
    seqs = [np.random.default_rng(n).integers(0, cfg["vocab_size"], size=n + steps).tolist() for n in lens]
    caches, rows = [], []
    for how in ("captured", "taps", "nothing wanted"):
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1280, max_seqs=5, use_graphs=how == "captured")
        for t in eng.cache.keys + eng.cache.values:
            t.zero_()
        slots = [eng.open_sequence() for _ in seqs]
        for s, q, n in zip(slots, seqs, lens):
            eng.step([StepEntry(s, q[:n], ())])
        for i in range(steps):
            taps = {} if how == "taps" else None
            want = () if how == "nothing wanted" and i < steps - 1 else (0,)
            out = eng.step([StepEntry(s, [q[n + i]], want) for s, q, n in zip(slots, seqs, lens)], taps=taps)
            if taps is not None:
                assert sorted(taps) == ["embed", "final_norm", "layer0", "layer1", "layer2"]
                assert not torch.equal(taps["layer0"], taps["layer1"])
        eng.check_status()
        rows.append(out.cpu().numpy())
        caches.append([t.cpu() for t in eng.cache.keys + eng.cache.values])
    for r, c in zip(rows[1:], caches[1:]):
        assert np.array_equal(rows[0], r)
        assert all(torch.equal(a, b) for a, b in zip(caches[0], c))


def test_a_row_whose_squares_overflow(tmp_path):
    """1 / rms of an infinite mean square is 0: such a row's logits are those of a row of zeros, as layer by layer, and its
    neighbour's are as ever."""
    from mynah_slm_b200.engine.engine import Engine, StepEntry
    cfg = dict(_cfg(2, 256, 4, 2, 64, 320), tie_word_embeddings=False)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=3)
    out = {}
    for one in (True, False):
        for big in (True, False):
            eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=256, max_seqs=2)
            if not one:
                eng.decode_layers = None
            if big:
                eng.model.embedding.table[7] *= 1e21
            slots = [eng.open_sequence() for _ in range(2)]
            out[one, big] = eng.step([StepEntry(slots[0], [7], (0,)), StepEntry(slots[1], [9], (0,))]).cpu().numpy()
            eng.check_status()
    for one in (True, False):
        assert not out[one, True][0].any() and out[one, False][0].any()
        assert np.array_equal(out[one, True][1], out[one, False][1])


@pytest.mark.parametrize("graphs", [True, False])
def test_a_declined_launch_leaves_the_layers_one_by_one(tmp_path, monkeypatch, graphs):
    """Where the one launch cannot be made, steps with and without taps go on as in an engine without it."""
    from mynah_slm_b200.engine.engine import Engine, StepEntry
    from mynah_slm_b200.ops import decode_layers
    cfg = _cfg(2, 256, 4, 2, 64, 320)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=3)
    toks = np.random.default_rng(0).integers(0, cfg["vocab_size"], size=76).tolist()
    offered = []
    monkeypatch.setattr(decode_layers, "offer", lambda name, *args: offered.append(name) is not None)
    rows = []
    for has in (True, False):
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=256, max_seqs=1, use_graphs=graphs)
        if not has:
            eng.decode_layers = None
        slot = eng.open_sequence()
        eng.step([StepEntry(slot, toks[:70], ())])
        rows.append([eng.step([StepEntry(slot, [t], (0,))], taps={} if i == 3 else None).cpu().numpy() for i, t in enumerate(toks[70:])])
        eng.check_status()
    assert len(offered) == 1 and all(np.array_equal(a, b) for a, b in zip(*rows))


@pytest.mark.parametrize("graphs", [True, False])
def test_a_wait_that_is_given_up_is_reported_and_over(tmp_path, graphs):
    """With no patience at all a step gives up the first wait for another CTA's words: it ends, says so, and the steps after it are
    as ever (the tags have moved on, nothing that it left passes for a later step's)."""
    from mynah_slm_b200.engine.engine import Engine, EngineError, StepEntry
    cfg = _cfg(2, 1024, 16, 8, 128, 3072)
    folder = make_folder(tmp_path, "one", torch.bfloat16, config=cfg, seed=3)
    lens = [300, 20, 700]
    seqs = [np.random.default_rng(n).integers(0, cfg["vocab_size"], size=n + 2).tolist() for n in lens]

    def steps(eng):
        slots = [eng.open_sequence() for _ in lens]
        for s, q in zip(slots, seqs):
            eng.step([StepEntry(s, q[:-2], ())])
        out = [eng.step([StepEntry(s, [q[i]], (0,)) for s, q in zip(slots, seqs)]).cpu().numpy() for i in (-2, -1)]
        for s in slots:
            eng.close_sequence(s)
        return out
    engines = [Engine.from_folder(folder, dtype="bfloat16", max_tokens=1280, max_seqs=3, use_graphs=graphs) for _ in range(2)]
    want = steps(engines[0])
    want = steps(engines[0])                             # (the second time prompts are captured, too)
    engines[0].check_status()
    eng = engines[1]
    eng.decode_layers.WAIT_LOOKS = 0
    steps(eng)
    with pytest.raises(EngineError, match="a bounded wait inside a kernel ran out"):
        eng.check_status()
    eng.decode_layers.WAIT_LOOKS = type(eng.decode_layers).WAIT_LOOKS
    eng._graphs.clear()                                  # (they were captured with no patience)
    assert all(np.array_equal(a, b) for a, b in zip(want, steps(eng)))
    eng.check_status()
