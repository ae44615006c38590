"""2-D pairing at the edges of the matching kernel's warps, blocks and clusters
(1024 threads a block; 1, 2, 4 and 8 blocks from 4096 programs up), on lists of
several shapes, against the oracle."""
import numpy as np
import pytest

from cubff_gb300 import abi
from oracle import oracle as O
from tests import harness

pytestmark = pytest.mark.gpu


def lists(shape, n, seed):
    rng = np.random.default_rng(seed)
    if shape == "ring":     # long chains of edges that block one another
        return O.lists_to_csr([[(i + 1) % n] for i in range(n)], n)
    if shape == "star":     # nearly all edges meet in one program
        return O.lists_to_csr([[1]] + [[0] for _ in range(n - 1)], n)
    if shape == "few":      # most programs propose nothing
        return O.lists_to_csr([[int((i + 7) % n)] if i % 97 == 0 else [] for i in range(n)], n)
    return O.lists_to_csr([[int(j) for j in rng.integers(0, n, rng.integers(0, 6)) if j != i]
                           for i in range(n)], n)


@pytest.mark.parametrize("shape,n,epochs", [
    ("ring", 2, 5), ("random", 34, 70), ("star", 66, 3), ("random", 1026, 5), ("ring", 4096, 3),
    ("random", 4098, 3), ("few", 8190, 3), ("star", 9000, 3), ("ring", 16386, 2),
    ("random", 32770, 2), ("random", 70002, 2)])
def test_matching_equals_the_oracle(shape, n, epochs):
    csr = lists(shape, n, n)
    soup = abi.Soup(harness.engine(), "bff", n, 3, 1 << 24, abi.PAIR_PATTERN)
    soup.set_pattern(*csr)
    ops, _raw = soup.run(epochs)
    got = soup.read()
    soup.close()
    want_ops, want = [], {}

    def cb(e, s, o, r):
        want_ops.append(o)
        if e == epochs:
            want["soup"] = s.copy()
        return e >= epochs
    O.OracleSim("bff", n, 3, 1 << 24, pairing=O.PAIR_PATTERN, pattern=csr).run(cb)
    assert [int(x) for x in ops] == want_ops
    assert np.array_equal(got, want["soup"])
