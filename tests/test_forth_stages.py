"""The Forth family's two machines (forth.cuh): a program's first steps on a
lane, then the warp's engine, where they can go wrong: runs of jumps that go in
circles, loops that only the stack's depth or a tested value ends, code that
writes over itself, and soups whose pair counts straddle the lanes of a warp."""
import numpy as np
import pytest

from cubff_gb300 import LANGUAGES, abi
from oracle import oracle as O
from tests.test_interp_host import check, host_lib  # noqa: F401

FORTHS = [lang for lang in LANGUAGES if lang.startswith("forth")]
NOOP = 0x20


def loop(rng, ops, length):
    """A program that jumps back over `length` random ops for ever, runs of
    no-ops and forward jumps between them."""
    prog = []
    for _ in range(length):
        prog.append(int(rng.choice(ops)))
        for _ in range(int(rng.integers(0, 3))):
            prog.append(NOOP if rng.random() < 0.5 else 0x80)
    return prog + [0xC0 | min(63, len(prog) - 1 + int(rng.integers(0, 2)))]


@pytest.mark.parametrize("lang", FORTHS)
@pytest.mark.parametrize("kind", ["circles", "depth", "tested", "writes", "own code"])
def test_loops_against_oracle(host_lib, lang, kind):  # noqa: F811
    rng = np.random.default_rng([LANGUAGES.index(lang), len(kind)])
    arith = [4, 5, 6, 8, 9, 0xA, 0xB, 0x41, 0x7F]
    ops = {"circles": [NOOP, 0x80, 0x81, 0xC0, 0xC3], "depth": arith + [0x42, 0x43, 0x44, 4],
           "tested": arith + [7, 7], "writes": arith + [0, 1, 2, 3, 0xC, 0xD, 7],
           "own code": [2, 3, 0xC, 0xD, 0x40, 0x48, 8, 4, 0x50]}[kind]
    for trial in range(250):
        tape = np.full(128, NOOP, dtype=np.uint8)
        if trial % 3 == 0:
            tape[64:] = rng.integers(0, 256, 64)
        lead = int(rng.integers(0, 30))
        tape[:lead] = [int(x) for x in rng.choice([NOOP, 0x41, 0x42], lead)]
        prog = loop(rng, ops, int(rng.integers(1, 9)))
        if kind == "circles":
            prog = [int(x) for x in rng.choice([NOOP, 0x80, 0x82, 0xC0, 0xC1, 0xC5, 0xC9], 40)]
        tape[lead:lead + len(prog)] = prog
        check(host_lib, lang, tape)


@pytest.mark.gpu
@pytest.mark.parametrize("lang,n", [("forth", 2), ("forthcopy", 14), ("forthtrivial", 16),
                                    ("forthtrivial_reset", 18), ("forth", 66),
                                    ("forthtrivial_reset", 1026)])
def test_pair_counts_around_a_warp(lang, n):
    epochs, want = 40, []
    soup = O.OracleSim(lang, n, 21, 1 << 21).run(
        lambda e, s, o, r: want.append((o, r)) or False, 1, max_epochs=epochs)
    eng = abi.Engine(0)
    s = abi.Soup(eng, lang, n, 21, 1 << 21)
    ops, raw = s.run(epochs)
    assert [(int(o), int(r)) for o, r in zip(ops, raw)] == want
    assert np.array_equal(s.read(), soup)
    s.close()
    eng.close()
