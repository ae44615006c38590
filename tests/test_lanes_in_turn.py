"""The machines as the kernels run them (tests/native/lanes_host.cu): the first
stage and SUBLEQ on one lane of interleaved words, the second stage by 32 lanes
that take turns between two syncs, in several orders.  CUDA promises no more than
that; lanes that have to stay in step would end with other tapes, counts or
collectives here."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from cubff_gb300 import LANGUAGES
from oracle import oracle as O
from tests.test_interp_host import CRAFTED, dense_bytes

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
SO = os.path.join(HERE, "_native", "liblanes_host.so")
SRC = os.path.join(HERE, "native", "lanes_host.cu")
STAGED = [lang for lang in LANGUAGES if "subleq" not in lang]
ORDERS = [0, 1, 12345]


@pytest.fixture(scope="module")
def lanes_lib():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    csrc = os.path.join(REPO, "cubff_gb300", "csrc")
    deps = [SRC] + [os.path.join(csrc, f) for f in os.listdir(csrc) if f.endswith((".cuh", ".h"))]
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        subprocess.run([nvcc, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", csrc,
                        "-I", os.path.join(REPO, "include"), SRC, "-o", SO], check=True)
    L = ctypes.CDLL(SO)
    u32, vp = ctypes.c_uint32, ctypes.c_void_p
    L.lanes_evaluate.restype = ctypes.c_int
    L.lanes_evaluate.argtypes = [ctypes.c_int, vp, u32, u32, u32, u32, vp, vp, vp]
    return L


def check(L, lang, tape, stride, lane, order, steps_on=0):
    want = tape.copy()
    ops, raw = O.evaluate(lang, want)
    got = tape.copy()
    c = np.zeros(3, dtype=np.uint32)
    st = L.lanes_evaluate(LANGUAGES.index(lang), got.ctypes.data, stride, lane, order, steps_on,
                          c[0:].ctypes.data, c[1:].ctypes.data, c[2:].ctypes.data)
    case = (lang, order, steps_on, bytes(tape).hex())
    assert st == 0, (st, case)
    assert (int(c[0]), int(c[1])) == (ops, raw), case
    assert np.array_equal(got, want), case
    # What changed is written back: a changed tape must say so.
    assert c[2] or np.array_equal(want, tape), case


def tapes_of(lang, count, seed):
    rng = np.random.default_rng([seed, LANGUAGES.index(lang)])
    dense = dense_bytes(lang)
    for trial in range(count):
        if trial % 4 == 0:
            tape = rng.integers(0, 256, 128, dtype=np.uint8)
        else:
            tape = dense[rng.integers(0, dense.size, 128)].astype(np.uint8)
            if trial % 4 == 2:
                mask = rng.random(128) < 0.8
                tape[mask] = rng.integers(0, 256, int(mask.sum()), dtype=np.uint8)
            elif trial % 4 == 3:
                tape[64:] = tape[:64]
        yield tape


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("lang", STAGED)
def test_lanes_in_turn_match_oracle(lanes_lib, lang, order):
    for i, tape in enumerate(tapes_of(lang, 160, 31)):
        check(lanes_lib, lang, tape, (8, 16, 32)[i % 3], i * 5 + 3, order)


@pytest.mark.parametrize("lang", ["bff_noheads", "bff", "bff8", "forth"])
def test_crafted_loops_in_turn(lanes_lib, lang):
    for i, prog in enumerate(CRAFTED[lang]):
        tape = np.zeros(128, dtype=np.uint8)
        tape[:len(prog)] = np.frombuffer(prog, dtype=np.uint8)
        check(lanes_lib, lang, tape, 8, i, ORDERS[i % 3])
        tape[len(prog):] = 0x61
        check(lanes_lib, lang, tape, 8, i, ORDERS[(i + 1) % 3])


@pytest.mark.parametrize("lang", ["forthtrivial_reset", "bff"])
def test_pairs_of_an_evolved_soup_in_turn(lanes_lib, lang):
    n = 1 << 11
    soup = O.OracleSim(lang, n, 3, 1 << 20).run(lambda *a: False, 1, max_epochs=200)
    progs = soup.reshape(n, 64)
    tapes = np.concatenate([progs[0::2], progs[1::2]], axis=1)
    raws = [O.evaluate(lang, t.copy())[1] for t in tapes]
    for i, k in enumerate(np.argsort(raws)[::-1][:48]):
        check(lanes_lib, lang, tapes[k].copy(), 8, i, ORDERS[i % 3])


@pytest.mark.parametrize("stride", [16, 32])
@pytest.mark.parametrize("lang", ["subleq", "rsubleq4"])
def test_subleq_on_words_matches_oracle(lanes_lib, lang, stride):
    rng = np.random.default_rng([stride, len(lang)])
    for trial in range(3000):
        tape = rng.integers(0, 256, 128, dtype=np.uint8)
        if trial % 2:
            small = rng.random(128) < 0.6
            tape[small] = rng.integers(0, 24, int(small.sum()))
        check(lanes_lib, lang, tape, stride, trial, 0)
    for prog in CRAFTED[lang]:
        tape = np.zeros(128, dtype=np.uint8)
        tape[:len(prog)] = np.frombuffer(prog, dtype=np.uint8)
        check(lanes_lib, lang, tape, stride, 5, 0)


CROWDS = [lang for lang in STAGED if lang.startswith(("forth", "bff8"))]


@pytest.mark.parametrize("lang", CROWDS)
def test_programs_taken_on_by_a_lane(lanes_lib, lang):
    """All of a program on its lane, or so many steps before the warp takes it."""
    for i, tape in enumerate(tapes_of(lang, 1500, 47)):
        check(lanes_lib, lang, tape, 8, i, ORDERS[i % 3], (1 << 14, 7, 256, 1, 40)[i // 4 % 5])


def test_copy_backwards_of_equal_bytes_runs_in_batches(lanes_lib):
    """A copy loop whose heads part ways on a palindrome: nothing changes, so its
    iterations run 32 at a time until the heads have been around."""
    half = np.arange(1, 65, dtype=np.uint8) + 150
    tape = np.concatenate([half, half[::-1]])
    prog = b"+[{.>]"
    tape[:len(prog)] = list(prog)
    tape[128 - len(prog):] = list(prog[::-1])
    check(lanes_lib, "bff_noheads", tape, 8, 3, 0)
    assert 0 < lanes_lib.lanes_rounds() < 100, lanes_lib.lanes_rounds()
