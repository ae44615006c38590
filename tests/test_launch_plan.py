"""How many pairs a warp holds and how many blocks a pipelined launch has
(launch_plan.h), and runs on the GPU at sizes on both sides of each step."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from cubff_gb300 import LANGUAGES, abi
from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
SO = os.path.join(HERE, "_native", "liblaunch_plan_host.so")
SRC = os.path.join(HERE, "native", "launch_plan_host.cu")
SMS, NARROW, WIDE = 152, 5, 4


@pytest.fixture(scope="module")
def plan():
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
    u32 = ctypes.c_uint32
    L.launch_plan.argtypes = [ctypes.c_int, ctypes.c_uint64, u32, ctypes.c_int, ctypes.c_int,
                              ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    L.claims.argtypes = [u32, u32, u32]

    def run(lang, pairs, lanes_per_pair64=32):
        out = np.zeros(2, dtype=np.uint32)
        L.launch_plan(LANGUAGES.index(lang), pairs, lanes_per_pair64, SMS, NARROW, WIDE,
                      out[0:].ctypes.data, out[1:].ctypes.data)
        return int(out[0]), int(out[1])

    run.claims = L.claims
    return run


def test_every_claim_threshold_can_be_met(plan):
    """A busy warp (one lane of those that hold pairs is) claims under every
    threshold but the highest, and sooner under a lower one."""
    for width in (8, 16, 32):
        needs = [next(i for i in range(width + 1) if plan.claims(i, width, c)) for c in range(1, 33)]
        assert needs == sorted(needs) and needs[-1] == width
        assert all(n < width for n in needs[:32 - 32 // width])
        assert needs[19] == -(-20 * width // 32)


@pytest.mark.parametrize("lang", LANGUAGES)
def test_every_launch_keeps_its_warps_busy(plan, lang):
    """No launch is empty or larger than what is resident; a wide one has lanes
    enough for the warps it was chosen for."""
    for pairs in [1, 2, 511, 4095, 4097, 8192, 32768, 65536, 97280, 194559, 194560, 1 << 20, 1 << 30]:
        for per64 in (1, 16, 32, 48, 64):
            width, grid = plan(lang, pairs, per64)
            resident = SMS * (NARROW if width == plan(lang, 1)[0] else WIDE)
            assert 1 <= grid <= resident
            if width > plan(lang, 1)[0]:
                assert grid * 4 >= min(3 * SMS, resident * 4)
            assert (grid - 1) * 4 * width < pairs


@pytest.mark.parametrize("lang,programs,pairs_of_a_warp", [
    ("bff", 1 << 17, 8), ("bff", 16 * 50790, 32), ("bff_noheads", 60 * 50790, 32),
    ("bff8", 1 << 14, 8), ("bff8", 1 << 15, 16), ("bff8", 60 * 50790, 32),
    ("forth", 1 << 15, 8), ("forth", 1 << 16, 32), ("subleq", 1 << 12, 16), ("subleq", 1 << 22, 16)])
def test_width_by_the_size_of_the_launch(plan, lang, programs, pairs_of_a_warp):
    """A saturated launch's warps hold 32 pairs (8 to a warp, it ran at 0.9 of the
    speed of one pair a lane); a soup's 8, or where lanes share long pairs more."""
    assert plan(lang, programs // 2)[0] == pairs_of_a_warp


@pytest.mark.parametrize("lang", ["bff", "forth", "subleq"])
def test_fewer_lanes_are_had_by_asking(plan, lang):
    """The minimum of lanes is for launches that ask for the default or more: one
    that leaves room for others gets as few as it asks for, on any device."""
    pairs = 2000
    assert plan(lang, pairs, 64) == plan(lang, pairs, 32)  # all pairs at once
    grids = [plan(lang, pairs, per64)[1] for per64 in (1, 4, 8, 16, 24, 31, 32)]
    assert grids == sorted(grids) and len(set(grids[:5])) == 5
    assert grids[3] <= grids[-1] // 3


@pytest.mark.gpu
@pytest.mark.parametrize("lang,n,count", [("bff8", 29182, 1), ("bff8_noheads", 29186, 1),
                                          ("forth", 58366, 1), ("forthtrivial", 58370, 1),
                                          ("bff", 48642, 8), ("bff_perm", 48638, 8)])
def test_runs_on_both_sides_of_a_step(lang, n, count):
    """Soups just below and above the size from which warps are wide, some of them
    of programs that all run long, against the oracle."""
    epochs = 3
    data = []
    for i in range(count):
        soup = O.init_programs(O.seed_of(5 + i, 0), n).reshape(n, 64).copy()
        if i % 2 == 0:  # most pairs alike: a loop that goes on for ever
            body = {"bff8": b"+aaaaaaa]", "bff8_noheads": b"+aaaaaaa]"}.get(lang, b"+[<.]")
            if lang.startswith("forth"):
                body = bytes([0x41, 0x08, 0x04, 0x0C, 0xC2])
            soup[: n - n // 8, 2:2 + len(body)] = np.frombuffer(body, dtype=np.uint8)
        data.append(soup)
    eng = abi.Engine(0)
    soups = [abi.Soup(eng, lang, n, 5 + i) for i in range(count)]
    for s, d in zip(soups, data):
        s.write(d.tobytes())
    got = abi.batch_run(eng, soups, epochs)
    for i in range(count):
        want = []
        load = np.array([1, n, 0], dtype=np.uint64).tobytes() + data[i].tobytes()
        end = O.OracleSim(lang, n, 5 + i, load=load).run(
            lambda e, s, o, r: want.append(o) or False, 1, max_epochs=epochs)
        assert got[i].tolist() == want
        assert np.array_equal(soups[i].read(), end)
        soups[i].close()
    eng.close()
