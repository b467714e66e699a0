"""The ring of slots that the one-launch decode step feeds its two groups of warps from (csrc/decode_layers.cu), as a model: no
group may take a slot before its filling has landed, in whatever order the copies land, and none may wait for good."""
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "mynah_slm_b200", "csrc", "decode_layers.cu")


def _constant(name):
    with open(SOURCE) as f:
        return int(re.search(rf"\b{name} = (\d+)[,;]", f.read()).group(1))


SLOTS, RUN = _constant("SLOTS"), _constant("RUN")


def _walk(jobs, look, rng):
    """Fillings 0 .. 2 * sum(jobs) - 1, two a page, the pages of job j for group j % 2. The producer asks for them in order, a
    slot's next one once the group that owns the last has handed it back; they land in any order. `look(r, i)` says what a group
    that wants filling i sees. True: all read after landing. False: one read too early. None: nobody can go on."""
    owner = [j % 2 for j, n in enumerate(jobs) for _ in range(2 * n)]
    n = len(owner)
    r = {"issued": 0, "landed": [0] * SLOTS, "seen": [0, 0]}
    in_flight, returned = [], [False] * n
    mine = [[i for i in range(n) if owner[i] == g] for g in (0, 1)]
    at = [0, 0]
    while at[0] < len(mine[0]) or at[1] < len(mine[1]):
        moves = []
        if r["issued"] < n and (r["issued"] < SLOTS or returned[r["issued"] - SLOTS]):
            moves.append(("ask", 0))
        moves += [("land", k) for k in range(len(in_flight))]
        for g in (0, 1):
            if look is _seen_by_all and r["seen"][g] < n and owner[r["seen"][g]] != g and _parity(r, r["seen"][g]):
                moves.append(("pass", g))
            if at[g] < len(mine[g]) and look(r, mine[g][at[g]]) and (look is not _seen_by_all or r["seen"][g] == mine[g][at[g]]):
                moves.append(("take", g))
        if not moves:
            return None
        what, k = rng.choice(moves)
        if what == "ask":
            in_flight.append(r["issued"])
            r["issued"] += 1
        elif what == "land":
            r["landed"][in_flight.pop(k) % SLOTS] += 1
        elif what == "pass":
            r["seen"][k] += 1
        else:
            i = mine[k][at[k]]
            if r["landed"][i % SLOTS] != i // SLOTS + 1:
                return False
            returned[i] = True
            at[k] += 1
            r["seen"][k] = i + 1
    return True


def _parity(r, i):
    return r["landed"][i % SLOTS] % 2 != (i // SLOTS) % 2


def _issued_first(r, i):                                  # what the kernel does
    return r["issued"] > i and _parity(r, i)


def _seen_by_all(r, i):                                   # every group looks at the other's fillings as it passes over them
    return _parity(r, i)


def _results(look, runs=4000):
    rng = random.Random(1)
    out = set()
    for _ in range(runs):
        jobs = [rng.randint(1, RUN) for _ in range(rng.randint(1, 7))]
        out.add(_walk(jobs, look, rng))
    return out


def test_no_slot_is_taken_before_its_filling_has_landed():
    assert _results(_issued_first) == {True}


@pytest.mark.parametrize("look,fault", [(_parity, False), (_seen_by_all, None)])
def test_the_model_sees_what_the_other_ways_miss(look, fault):
    """The parity alone takes a slot too early; looking at the other group's fillings can wait for good."""
    assert fault in _results(look)
