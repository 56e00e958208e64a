"""The ends of the look-back state (csrc/edp_prims.cu).  A wait that runs out:
the kernel returns, its own error bit is set and named by no capacity, nothing
is left behind for the next launch (the tiles waited for are tickets that no
block takes).  And the epochs' start over after 2^30 launches, over words that
an old launch left."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest
from conftest import ROOT

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WAIT = 4096  # EDP_ERR_BIT_WAIT
LAST_EPOCH = (1 << 30) - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("look_back") / "liblookback.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-fmad=false", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    "-o", str(out), str(ROOT / "tests/native/look_back_harness.cu")], check=True)
    return ctypes.CDLL(str(out))


# Tiles: 4,096 elements of a scan, 2,048 keys of a radix pass.
@pytest.mark.parametrize("missing,epoch", [(0, 0), (1, 0), (3, 0), (0, LAST_EPOCH)])
@pytest.mark.parametrize("n", [4095, 4096, 4097, 8192, 100_001])
def test_scan(lib, n, missing, epoch):
    values = np.random.default_rng(n).integers(0, 9, size=n).astype(np.int32)
    out, errors = np.zeros(n + 1, dtype=np.int32), np.zeros(2, dtype=np.int32)
    assert lib.look_back_scan(values.ctypes.data_as(ctypes.c_void_p), n, 1000, missing, epoch,
                              out.ctypes.data_as(ctypes.c_void_p),
                              errors.ctypes.data_as(ctypes.c_void_p)) == 0
    assert errors[0] == (WAIT if missing else 0) and errors[1] == 0
    np.testing.assert_array_equal(out, np.concatenate([[0], np.cumsum(values)]))


@pytest.mark.parametrize("missing,epoch", [(0, 0), (1, 0), (3, 0), (0, LAST_EPOCH)])
@pytest.mark.parametrize("n", [2049, 4096, 50_001])
def test_sort(lib, n, missing, epoch):
    keys = np.random.default_rng(n).integers(0, 1 << 16, size=n).astype(np.uint64)
    out, positions = np.zeros(n, dtype=np.uint64), np.zeros(n, dtype=np.int32)
    errors = np.zeros(2, dtype=np.int32)
    assert lib.look_back_sort(keys.ctypes.data_as(ctypes.c_void_p), n, 1000, missing, epoch,
                              out.ctypes.data_as(ctypes.c_void_p),
                              positions.ctypes.data_as(ctypes.c_void_p),
                              errors.ctypes.data_as(ctypes.c_void_p)) == 0
    assert errors[0] == (WAIT if missing else 0) and errors[1] == 0
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(out, keys[order])
    np.testing.assert_array_equal(positions, order)


def test_the_bit_names_no_capacity():
    from peel_b200.sizing import _POOL_OF_BIT
    from peel_b200.solver import _decode_status

    assert WAIT not in _POOL_OF_BIT
    with pytest.raises(RuntimeError, match="wait ran out"):
        _decode_status([0] * 9 + [WAIT] + [0] * 6)
