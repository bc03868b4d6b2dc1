"""What the kernels' sources have to say about their bounded waits; a lost signal cannot be staged on a GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"


@pytest.mark.parametrize("name,alone", [("gemm_sm100.cu", 0), ("gemm_pair_sm100.cu", 0), ("attn_tc_sm100.cu", 1), ("attn_latent_sm100.cu", 3)])
def test_no_lane_leaves_a_warp_wide_role_by_itself(name, alone):
    """Lanes that run out of polls one by one would leave the rest alone at the next ``elect.sync`` or ``tcgen05.ld``, which wait for
    all 32.  The waits of these roles fail for the whole warp (``gave_up``) or are voted on at once (``warp_ok``); ``alone``
    waits belong to threads that take no warp-wide steps (cp.async loaders, a single issuing lane)."""
    text = re.sub(r"//.*", "", (CSRC / name).read_text())
    text = text[text.index("__global__"):]
    waits = re.findall(r"(warp_ok\()?\b(mbar_wait\w*|lat_mbar_wait|lat_warp_wait|attn_wait<TMA>)(\([^;]*?p\.status, \w+[^;]*?\))", text)
    assert len(waits) >= 4
    assert sum(not voted and "gave_up" not in args for voted, _, args in waits) == alone, waits


def _lanes(runs_out, signal, order):
    """The lanes of a warp at one wait, one step of one lane at a time in the given order: poll, and after ``runs_out`` polls the
    steps of ``warp_gives_up`` (sign off; read the word; poll; withdraw by compare-and-swap).  Returns each lane's answer."""
    n, word, answer = len(runs_out), 0, {}
    state = [("poll", 0, 0)] * n
    t = 0
    for lane in order:
        if lane in answer:
            continue
        t += 1
        full, bit = (1 << n) - 1, 1 << lane
        step, polls, seen = state[lane]
        if step == "poll":
            if t > signal:
                answer[lane] = True
            state[lane] = ("poll", polls + 1, 0) if polls + 1 < runs_out[lane] else ("sign", 0, 0)
        elif step == "sign":
            word |= bit
            state[lane] = ("read", 0, 0)
        elif step == "read":
            if word == full:
                answer[lane] = False
            state[lane] = ("look", 0, word)
        elif step == "look":
            state[lane] = ("swap" if t > signal else "read", 0, seen)
        elif word == seen:                                   # swap
            word &= ~bit
            state[lane] = ("poll", 0, 0)
        else:
            state[lane] = ("read", 0, 0)
    return answer


@pytest.mark.parametrize("lanes", [2, 3, 5])
def test_lanes_give_up_together(lanes):
    """Whatever the interleaving and whenever the signal comes, the lanes give one answer, and all give one."""
    import random
    rng, seen = random.Random(lanes), set()
    for _ in range(4000):
        order = [rng.randrange(lanes) for _ in range(60 * lanes)] + list(range(lanes)) * 400
        got = _lanes([rng.randrange(1, 5) for _ in range(lanes)], rng.randrange(0, 20 * lanes), order)
        assert len(got) == lanes and len(set(got.values())) == 1, got
        seen |= set(got.values())
    assert seen == {True, False}
