"""Soups in which nearly every program runs long, through the kernels whose lanes
then take on long programs side by side: per epoch (at sizes on both sides of the
step to wide warps, with pairs that are not evaluated and a ragged end), scores,
and pipelined; against the oracle."""
import numpy as np
import pytest

from cubff_gb300 import abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LOOPS = {"bff8": b"@\x00+aaaaa}aa]", "bff8_noheads": b"+aaaaa>aa]", "bff": b"@\x00[,>}]",
         "forth": bytes([0x41, 0x08, 0x04, 0x00, 0x02, 0xC4]),
         "forthcopy": bytes([0x41, 0x08, 0x04, 0x04, 0x02, 0xC4]),
         "forthtrivial": bytes([0x0C, 0x08, 0x04, 0x3E, 0xC3]),
         "forthtrivial_reset": bytes([0x0C, 0x08, 0x04, 0x3E, 0xC3])}


def crowd_of(lang, n, seed, random_every):
    """A loop at the head of all programs but every so many."""
    data = np.random.default_rng(seed).integers(0, 256, (n, 64)).astype(np.uint8)
    body = np.frombuffer(LOOPS[lang], dtype=np.uint8)
    keep = np.arange(n) % random_every != random_every - 1
    data[keep, :body.size] = body
    return data.reshape(-1)


@pytest.mark.parametrize("lang,n,indices,random_every", [
    ("forthtrivial", 16, 8, 99), ("forth", 18, 9, 4), ("forthcopy", 1030, 500, 9),
    ("forthtrivial_reset", 29182, 14591, 12), ("forthtrivial", 29186, 14590, 30),
    ("forth", 29250, 14625, 3), ("bff8", 29184, 14592, 40), ("bff8_noheads", 29188, 14000, 6),
    ("bff8", 130, 65, 20), ("bff", 514, 257, 9)])
def test_epoch_of_long_programs(lang, n, indices, random_every):
    want = crowd_of(lang, n, n, random_every)
    dev = torch.from_numpy(want.copy()).cuda()
    perm = np.random.default_rng(1).permutation(n).astype(np.uint32)
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    ops, raw = O.mutate_and_run(lang, want, perm, 1234567, 1 << 20, indices)
    d_perm = torch.from_numpy(perm.view(np.int32)).cuda()
    abi.check(abi.lib().cubff_mutate_and_run(
        abi.language_id(lang), dev.data_ptr(), d_perm.data_ptr(), 1234567, 1 << 20,
        counts.data_ptr(), counts.data_ptr() + 8, n, indices, None))
    assert counts.tolist() == [ops, raw]
    assert np.array_equal(dev.cpu().numpy(), want)


@pytest.mark.parametrize("lang,n,count", [("forthtrivial", 8, 7), ("forthtrivial_reset", 13, 13),
                                          ("forth", 9, 9), ("forthcopy", 6, 5), ("bff8", 10, 9),
                                          ("bff8_noheads", 4, 4)])
def test_scores_of_long_programs(lang, n, count):
    soup = crowd_of(lang, n, 3 * n, 3)
    want = O.check_selfrep(lang, soup, 99, n)[:count]
    dev = torch.from_numpy(soup).cuda()
    res = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    abi.check(abi.lib().cubff_check_selfrep(abi.language_id(lang), dev.data_ptr(), 99, n, count,
                                            res.data_ptr(), None))
    got = res.cpu().numpy()
    assert got[:count].tolist() == [int(x) for x in want]
    assert (got[count:] == -1).all()


@pytest.mark.parametrize("lang,n", [("forthtrivial", 16), ("forthcopy", 66), ("forth", 1030),
                                    ("forthtrivial_reset", 258), ("bff8", 128),
                                    ("bff8_noheads", 1022)])
@pytest.mark.parametrize("random_every", [2, 12])
def test_pipelined_epochs_of_long_programs(lang, n, random_every):
    data = crowd_of(lang, n, n + random_every, random_every)
    epochs, want = 12, []
    load = np.array([1, n, 0], dtype=np.uint64).tobytes() + data.tobytes()
    soup = O.OracleSim(lang, n, 9, 1 << 20, load=load).run(
        lambda e, s, o, r: want.append((o, r)) or False, 1, max_epochs=epochs)
    eng = abi.Engine(0)
    for lanes in (4, 32, 64):
        eng.set_tuning(lang, n, 1, lanes_per_pair64=lanes, steps_per_visit=64, claim_min=20,
                       long_visits=1, first_visit_steps=64)
        s = abi.Soup(eng, lang, n, 9, 1 << 20)
        s.write(data.tobytes())
        ops, raw = s.run(epochs)
        assert [(int(o), int(r)) for o, r in zip(ops, raw)] == want
        assert np.array_equal(s.read(), soup)
        s.close()
    eng.close()
