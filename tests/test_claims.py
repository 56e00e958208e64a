"""Claims of pool entries by many threads at once (claim_entries in
csrc/edp_device.cuh, run on the CPU from a host build of the same source): no
entry is granted twice, whatever mix of lengths is refused at the pool's end."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest
from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("claims") / "libclaims.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                    "-Xcompiler", "-fPIC,-pthread", "-shared", "-o", str(out),
                    str(ROOT / "tests/native/claims_harness.cu")], check=True)
    handle = ctypes.CDLL(str(out))
    handle.claims.restype = ctypes.c_int64
    handle.claims.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_int64,
                              ctypes.c_void_p]
    return handle


def grants(lib, lengths, threads, capacity):
    starts = np.zeros(lengths.size, dtype=np.int64)
    lib.claims(threads, lengths.size // threads, lengths.ctypes.data, capacity,
               starts.ctypes.data)
    granted = starts >= 0
    order = np.argsort(starts[granted])
    return starts[granted][order], lengths[granted][order]


@pytest.mark.parametrize("seed", range(4))
def test_no_entry_is_granted_twice(lib, seed):
    rng = np.random.default_rng(seed)
    threads, each = 8, 4000
    # Long lists among many short ones, far more in all than the pool holds.
    lengths = rng.integers(1, 40, size=threads * each).astype(np.int32)
    lengths[rng.random(lengths.size) < 0.1] = 3000
    capacity = 500_000
    starts, sizes = grants(lib, lengths, threads, capacity)
    assert len(starts) > 100
    assert (starts[1:] >= starts[:-1] + sizes[:-1]).all()
    assert starts[-1] + sizes[-1] <= capacity


def test_a_refused_claim_leaves_room_for_shorter_ones(lib):
    lengths = np.array([60, 50, 40, 1], dtype=np.int32)
    starts, sizes = grants(lib, lengths, 1, 100)
    np.testing.assert_array_equal(starts, [0, 60])
    np.testing.assert_array_equal(sizes, [60, 40])
