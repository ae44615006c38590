"""The per-epoch, self-replication and single-tape kernels at the edges of
their blocks and warps (8 pairs a warp, 4 programs a block), on soups where many
pairs jump, against the oracle."""
import ctypes
import threading

import numpy as np
import pytest

from cubff_gb300 import LANGUAGES, abi
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def soup_of(lang, n, seed):
    """Random programs, every third one a loop that copies."""
    data = np.random.default_rng(seed).integers(0, 256, (n, 64)).astype(np.uint8)
    if lang.startswith("bff"):
        data[::3, :7] = np.frombuffer(b"@\x00[,>}]", dtype=np.uint8)
    elif lang.startswith("forth"):
        data[::3, :6] = [0x08, 0x04, 0x0C, 0x04, 0x0D, 0xC4]
    return data.reshape(-1)


@pytest.mark.parametrize("lang,n,indices", [("bff", 2, 1), ("bff_noheads", 14, 7), ("forth", 16, 8),
                                            ("forthtrivial", 18, 5), ("bff_perm", 64, 32),
                                            ("bff8_noheads", 66, 33), ("forthcopy", 1030, 400),
                                            ("subleq", 258, 100)])
def test_epoch_kernel_edges(lang, n, indices):
    want = soup_of(lang, n, n)
    dev = torch.from_numpy(want.copy()).cuda()
    perm = np.random.default_rng(1).permutation(n).astype(np.uint32)
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    ops, raw = O.mutate_and_run(lang, want, perm, 1234567, 1 << 22, indices)
    d_perm = torch.from_numpy(perm.view(np.int32)).cuda()
    abi.check(abi.lib().cubff_mutate_and_run(
        abi.language_id(lang), dev.data_ptr(), d_perm.data_ptr(), 1234567, 1 << 22,
        counts.data_ptr(), counts.data_ptr() + 8, n, indices, None))
    assert counts.tolist() == [ops, raw]
    assert np.array_equal(dev.cpu().numpy(), want)


@pytest.mark.parametrize("lang,n,count", [("bff", 1, 1), ("bff_noheads", 8, 3), ("forth", 8, 5),
                                          ("bff_selfmove", 130, 129), ("forthtrivial_reset", 36, 33)])
def test_selfrep_kernel_edges(lang, n, count):
    soup = soup_of(lang, n, 3 * n)
    want = O.check_selfrep(lang, soup, 99, n)[:count]
    dev = torch.from_numpy(soup).cuda()
    res = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    abi.check(abi.lib().cubff_check_selfrep(abi.language_id(lang), dev.data_ptr(), 99, n, count,
                                            res.data_ptr(), None))
    got = res.cpu().numpy()
    assert got[:count].tolist() == [int(x) for x in want]
    assert (got[count:] == -1).all()


def test_single_tapes_from_many_threads():
    """More threads than result slots, every language, each its own tapes."""
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        for lang in LANGUAGES:
            tape = soup_of(lang, 2, int(rng.integers(1 << 30)))
            want = tape.copy()
            want_ops, want_raw = O.evaluate(lang, want)
            ops, raw = ctypes.c_uint64(0), ctypes.c_uint64(0)
            abi.check(abi.lib().cubff_eval_pair(abi.language_id(lang), tape.ctypes.data,
                                                ctypes.byref(ops), ctypes.byref(raw)))
            if (ops.value, raw.value) != (want_ops, want_raw) or not np.array_equal(tape, want):
                bad.append((seed, lang))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(24)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
