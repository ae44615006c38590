"""The mutation draws of a pair 32 at a time (mutation_word, common.cuh) against
the draws one by one, on the host; and epochs whose keys lie where 32 draws
differ in more than their low bits, against the oracle."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from cubff_gb300 import abi
from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
GOLDEN = 0x9E3779B97F4A7C15  # added to a key before it is hashed


@pytest.mark.parametrize("prob", [0, 1, 1 << 18, 1 << 29, (1 << 30) - 1, 1 << 30, (1 << 32) - 1])
def test_words_equal_the_draws(prob):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src = os.path.join(HERE, "native", "mutation_host.cu")
    so = os.path.join(HERE, "_native", "libmutation_host.so")
    csrc = os.path.join(REPO, "cubff_gb300", "csrc")
    os.makedirs(os.path.dirname(so), exist_ok=True)
    deps = [src, os.path.join(csrc, "common.cuh")]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", csrc,
                        src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.mutation_words_differ.restype = ctypes.c_uint64
    lib.mutation_words_differ.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint32]
    rng = np.random.default_rng(prob)
    keys = rng.integers(0, 1 << 64, 60000, dtype=np.uint64)
    # Half of them with the sum's low 32 bits around a multiple of 2^30.
    near = (rng.integers(0, 4, 30000) << 30) - rng.integers(-2, 40, 30000) - (GOLDEN & 0xFFFFFFFF)
    keys[:30000] = (keys[:30000] & ~np.uint64(0xFFFFFFFF)) | (near & 0xFFFFFFFF).astype(np.uint64)
    assert lib.mutation_words_differ(keys.ctypes.data, len(keys), prob) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("lang", ["bff", "forth", "subleq"])
def test_epochs_where_the_keys_cross(lang):
    torch = pytest.importorskip("torch")
    n = 6
    # Pair k's draws have keys (n * key + k) * 128 + i: the 128 of one pair cross
    # a multiple of 2^30 after the constant is added.
    found = 0
    for j in range(40):
        first = (((j << 30) - GOLDEN - 100) % (1 << 64)) // 128
        if first % n >= n // 2:
            continue
        found += 1
        key = first // n
        want = np.random.default_rng(j).integers(0, 256, n * 64).astype(np.uint8)
        dev = torch.from_numpy(want.copy()).cuda()
        perm = np.arange(n, dtype=np.uint32)
        ops, raw = O.mutate_and_run(lang, want, perm, key, 1 << 29, n // 2)
        d_perm = torch.from_numpy(perm.view(np.int32)).cuda()
        counts = torch.zeros(2, dtype=torch.int64, device="cuda")
        abi.check(abi.lib().cubff_mutate_and_run(
            abi.language_id(lang), dev.data_ptr(), d_perm.data_ptr(), key, 1 << 29,
            counts.data_ptr(), counts.data_ptr() + 8, n, n // 2, None))
        assert counts.tolist() == [ops, raw]
        assert np.array_equal(dev.cpu().numpy(), want)
    assert found >= 10
