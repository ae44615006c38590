"""Forth programs on a warp that rewrite their own code are stepped one by one
for a while (forth.cuh, `plain`).  The last such step may jump back and so meet
the cycle check; where the steps by runs then go on, that same state must not be
checked again: a segment of no steps has no length to divide the rest by."""
import os
import subprocess
import sys

import pytest

from cubff_gb300 import LANGUAGES
from tests.test_interp_host import host_lib  # noqa: F401

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FORTHS = [lang for lang in LANGUAGES if lang.startswith("forth")]

# A forthtrivial_reset tape whose last plain step renews the snapshot at a
# position that the steps by runs start from again.
TAPE = ("06066d760c645d7904000802460002426f080c0c7d0c6a0d090d0309030d0776090b085d0b7d0600657c45005a0406"
        "744f67064f6e5246030c0763010a0d070d5c074247410104016b700372534b7546545a04086c03560a620a0d6e0405"
        "056a46020b5e7006000a405d6e535b6104560878736003677a0801757000084f6f6e")


def in_child(code):
    """A division by zero ends the process: kept out of this one."""
    r = subprocess.run([sys.executable, "-c", code], cwd=REPO, capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout[-500:], r.stderr[-500:])


def test_snapshot_renewed_by_the_last_plain_step(host_lib):  # noqa: F811
    in_child(f"""
import numpy as np
from tests.test_interp_host import SO, check
import ctypes
lib = ctypes.CDLL(SO)
for f in (lib.host_evaluate, lib.host_evaluate_lane):
    f.restype, f.argtypes = ctypes.c_uint32, [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
check(lib, "forthtrivial_reset", np.frombuffer(bytes.fromhex({TAPE!r}), dtype=np.uint8).copy())
""")


@pytest.mark.parametrize("lang", FORTHS)
def test_programs_that_rewrite_their_code(host_lib, lang):  # noqa: F811
    """Commands and constants throughout, back jumps now and then, halves alike."""
    in_child(f"""
import numpy as np
from tests.test_interp_host import SO, check
import ctypes
lib = ctypes.CDLL(SO)
for f in (lib.host_evaluate, lib.host_evaluate_lane):
    f.restype, f.argtypes = ctypes.c_uint32, [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
rng = np.random.default_rng(9)
dense = np.array(list(range(14)) * 3 + list(range(0x40, 0x80)), dtype=np.uint8)
for trial in range(6000):
    tape = dense[rng.integers(0, dense.size, 128)]
    back = rng.integers(16, 128, int(rng.integers(1, 5)))
    tape[back] = 0xC0 | np.minimum(back - 1, rng.integers(0, 63, back.size))
    if trial % 2:
        tape[64:] = np.where(rng.random(64) < 0.1, 0x13, tape[:64])
    check(lib, {lang!r}, tape)
""")
