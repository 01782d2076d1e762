"""Rules of the entropy stage that guard its memory accesses, compiled for the host (tests/native/entropy_rules.cu)
and checked against unbounded integers."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "entropy_rules.cu")
HDRS = [os.path.join(ROOT, "falcons_b200", "csrc", h) for h in ("entropy_rules.cuh", "fse.cuh")]
OUT = os.path.join(ROOT, "tests", "native", "_build", "libentropy_rules.so")


@pytest.fixture(scope="module")
def rules():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    if not os.path.exists(OUT) or os.path.getmtime(OUT) < max(map(os.path.getmtime, [SRC, *HDRS])):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.check_call([nvcc, "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC", "-x", "cu",
                               "-gencode", "arch=compute_100a,code=sm_100a", SRC, "-o", OUT])
    lib = ctypes.CDLL(OUT)
    lib.rules_chain_part_count.argtypes = [ctypes.c_ulonglong] * 2
    lib.rules_chain_part_count.restype = ctypes.c_ulonglong
    lib.rules_fse_block.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("n", [0, 1, 1 << 20, (1 << 31) - 1, 1 << 31, (1 << 31) + 1, (1 << 32) - 1, 1 << 32, 1 << 40])
def test_parts_of_a_chain(rules, n):
    """A chain without checkpoints is one part whatever its length (a second part would start from a checkpoint
    that there is none of); one beyond the decoder's 32-bit count is refused."""
    whole = 0 if n == 0 else 1 if n < 1 << 32 else 2 ** 64 - 1
    assert rules.rules_chain_part_count(n, 0) == whole
    for part in (64, 1024, 65536):
        assert rules.rules_chain_part_count(n, part) == -(-n // part)
