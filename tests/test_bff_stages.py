"""The BFF family's two machines (bff.cuh): the lane's forward part and the
warp's engine, where they can go wrong: loops whose batched iterations meet
each other's bytes, that write into their own code or run to the step limit,
and soups whose pair counts straddle the lanes of a warp."""
import numpy as np
import pytest

from cubff_gb300 import LANGUAGES, abi
from oracle import oracle as O
from tests.test_interp_host import check, host_lib  # noqa: F401

BFFS = [lang for lang in LANGUAGES if lang.startswith("bff")]


def commands(lang):
    """Command bytes in the order "[]+-.,<>{}" (None: the language has none)."""
    if lang == "bff_noheads_4bit":
        return list(range(0x26, 0x30))
    if lang == "bff_perm":
        return [9, 10, 5, 6, 7, 8, 1, 2, 3, 4]
    if lang == "bff_selfmove":
        return [5, 6, 2, 3, None, 4, 1, 0, None, None]
    return list(b"[]+-.,<>{}")


@pytest.mark.parametrize("lang", BFFS)
def test_loops_of_strides_against_oracle(host_lib, lang):  # noqa: F811
    """One or two copies or counts among head moves of every small stride, the
    heads anywhere (the loop's own code and overlapping ranges among it)."""
    rng = np.random.default_rng(77 + LANGUAGES.index(lang))
    c = dict(zip("[]+-.,<>{}", commands(lang)))
    noop = 0x31 if lang == "bff_noheads_4bit" else 20 if lang in ("bff_perm", "bff_selfmove") else 113
    for trial in range(1200):
        moves = "".join(rng.choice(list("<>{}"), rng.integers(0, 5)))
        acts = "".join(rng.choice(list(".,.,+-"), rng.integers(1, 3)))
        tail = "".join(rng.choice(list("<>{}")) * int(rng.integers(0, 5)) for _ in range(2))
        lead = "".join(rng.choice(list("<>{}"), rng.integers(0, 40)))
        prog = lead + "+[" + moves + acts[:1] + tail + acts[1:] + "]" + "[" * int(trial % 7 == 0)
        tape = rng.integers(0, 256, 128).astype(np.uint8)
        if trial % 3 == 0:
            tape[:] = noop
        elif trial % 3 == 1:
            tape[tape == 0] = 1
        pos = int(rng.integers(2, 70))
        for ch in prog:
            if pos < 128 and c[ch] is not None:
                tape[pos] = c[ch]
                pos += 1 + int(rng.integers(0, 2)) * (trial & 1)
        check(host_lib, lang, tape)


@pytest.mark.gpu
@pytest.mark.parametrize("lang,n", [("bff", 2), ("bff_noheads", 14), ("bff_perm", 16),
                                    ("bff8", 18), ("bff_selfmove", 62), ("bff_noheads_4bit", 66),
                                    ("bff", 1026)])
def test_pair_counts_around_a_warp(lang, n):
    """Soups seeded with a copier, so that many pairs jump, against the oracle."""
    c = commands(lang)
    data = np.random.default_rng(n).integers(0, 256, (n, 64)).astype(np.uint8)
    body = [c[0], c[5], c[7], c[9], c[1]]
    data[::2, :2] = [64, 0]
    data[::2, 2:2 + len(body)] = [b for b in body if b is not None] + [20] * body.count(None)
    epochs = 24
    want = []
    load = np.array([1, n, 0], dtype=np.uint64).tobytes() + data.tobytes()
    soup = O.OracleSim(lang, n, 9, 1 << 20, load=load).run(
        lambda e, s, o, r: want.append((o, r)) or False, 1, max_epochs=epochs)
    eng = abi.Engine(0)
    s = abi.Soup(eng, lang, n, 9, 1 << 20)
    s.write(data.tobytes())
    ops, raw = s.run(epochs)
    assert [(int(o), int(r)) for o, r in zip(ops, raw)] == want
    assert np.array_equal(s.read(), soup)
    s.close()
    eng.close()
