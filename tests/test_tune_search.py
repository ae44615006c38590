"""The launch-shape tuner's search (tune_search.h) on the host, over made-up times."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from cubff_gb300 import abi

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
SO = os.path.join(HERE, "_native", "libtune_search_host.so")
SRC = os.path.join(HERE, "native", "tune_search_host.cu")
DEFAULT = (32, 64, 20, 1, 64)
FIELDS = [f for f, _ in abi.Tuning._fields_]


@pytest.fixture(scope="module")
def search():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    os.makedirs(os.path.dirname(SO), exist_ok=True)
    csrc = os.path.join(REPO, "cubff_gb300", "csrc")
    deps = [SRC, os.path.join(csrc, "tune_search.h")]
    if not os.path.exists(SO) or any(os.path.getmtime(d) > os.path.getmtime(SO) for d in deps):
        subprocess.run([nvcc, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", csrc,
                        "-I", os.path.join(REPO, "include"), SRC, "-o", SO], check=True)
    L = ctypes.CDLL(SO)
    timer = ctypes.CFUNCTYPE(ctypes.c_double, ctypes.POINTER(abi.Tuning))

    def run(visits, time_of, lanes_same=1 << 30):
        shape = abi.Tuning(*DEFAULT)
        seen = []

        def call(p):
            seen.append(tuple(getattr(p.contents, f) for f in FIELDS))
            return time_of(dict(zip(FIELDS, seen[-1])))

        n = L.tune_search(int(visits), ctypes.byref(shape), timer(call), lanes_same)
        assert n == len(seen)
        return tuple(getattr(shape, f) for f in FIELDS), seen

    return run


def test_only_the_lanes_are_tried_where_only_they_matter(search):
    best, seen = search(False, lambda t: 1.0)
    assert best == DEFAULT
    assert {s[1:] for s in seen} == {DEFAULT[1:]} and len(seen) == 5
    best, _ = search(False, lambda t: 0.8 if t["lanes_per_pair64"] == 64 else 1.0)
    assert best == (64,) + DEFAULT[1:]


def test_equal_launches_are_timed_once(search):
    best, seen = search(False, lambda t: 1.0, lanes_same=32)
    assert [s[0] for s in seen] == [32, 16, 24] and best == DEFAULT


@pytest.mark.parametrize("visits", [False, True])
def test_noise_changes_nothing_and_hides_nothing(search, visits):
    """Times that differ by 2 % leave the default; a shape that is really 10 %
    faster is found among them."""
    rng = np.random.default_rng(3)
    for _ in range(20):
        assert search(visits, lambda t: rng.uniform(0.98, 1.0))[0] == DEFAULT
        best, _ = search(visits, lambda t: rng.uniform(0.98, 1.0) *
                         (0.9 if t["lanes_per_pair64"] == 48 else 1.0))
        assert best == (48,) + DEFAULT[1:]


def test_all_knobs_of_subleq(search):
    best, _ = search(True, lambda t: 1.0 - 0.1 * (t["claim_min"] == 8) - 0.1 * (t["steps_per_visit"] == 16))
    assert best == (32, 16, 8, 1, 64)
