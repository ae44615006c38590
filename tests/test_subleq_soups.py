"""The SUBLEQ languages' pipelined epochs at the edges of a warp and a block (32
and 128 pairs) and over soups that share a launch, against the oracle."""
import numpy as np
import pytest

from cubff_gb300 import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def jumpy(n, seed):
    """Small bytes, so that many programs jump about and modify themselves."""
    rng = np.random.default_rng(seed)
    data = rng.integers(0, 128, (n, 64)).astype(np.uint8)
    data[rng.random((n, 64)) < 0.1] = 255
    return data


def oracle_run(lang, n, seed, prob, data, epochs, **kw):
    want = []
    load = np.array([1, n, 0], dtype=np.uint64).tobytes() + data.tobytes()
    soup = O.OracleSim(lang, n, seed, prob, load=load, **kw).run(
        lambda e, s, o, r: want.append((o, r)) or False, 1, max_epochs=epochs)
    return want, soup


@pytest.mark.parametrize("lang", ["subleq", "rsubleq4"])
@pytest.mark.parametrize("n,epochs,prob", [(2, 3, 1 << 20), (62, 70, 1 << 18), (256, 66, 0),
                                           (258, 64, 1 << 30), (1022, 5, 1 << 22)])
def test_soups_around_a_block(lang, n, epochs, prob):
    data = jumpy(n, n)
    want, want_soup = oracle_run(lang, n, 9, prob, data, epochs)
    eng = abi.Engine(0)
    s = abi.Soup(eng, lang, n, 9, prob)
    s.write(data.tobytes())
    ops, raw = s.run(epochs)
    assert [(int(o), int(r)) for o, r in zip(ops, raw)] == want
    assert np.array_equal(s.read(), want_soup)
    s.close()
    eng.close()


@pytest.mark.parametrize("lang", ["subleq", "rsubleq4"])
def test_soups_that_share_launches(lang):
    """Sizes on both sides of a block, one soup 2-D (some pairs not evaluated)."""
    epochs, sizes = 70, [2, 258, 512, 130, 384]
    eng = abi.Engine(0)
    csr = O.grid_pattern(24, 16, 1)
    soups, wants = [], []
    for i, n in enumerate(sizes):
        data = jumpy(n, 50 + i)
        kw = {"pairing": O.PAIR_PATTERN, "pattern": csr} if n == 384 else {}
        wants.append(oracle_run(lang, n, i, 1 << (18 + i), data, epochs, **kw))
        s = abi.Soup(eng, lang, n, i, 1 << (18 + i), abi.PAIR_PATTERN if kw else abi.PAIR_SHUFFLE)
        if kw:
            s.set_pattern(*csr)
        s.write(data.tobytes())
        soups.append(s)
    got = abi.batch_run(eng, soups, epochs)
    for s, ops, (want, want_soup) in zip(soups, got, wants):
        assert [int(o) for o in ops] == [o for o, _ in want]
        assert np.array_equal(s.read(), want_soup)
        s.close()
    eng.close()
