"""Launch shapes and workspace sizes that follow from the device at hand, on the CPU."""
import ctypes
import os
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("shapes") / "shapes.so"
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(cuda), "-o", str(so),
                    str(HERE / "kernel_shapes.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("n", [128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("sms", [1, 2, 7, 15, 16, 31, 32, 36, 63, 64, 74, 127, 128, 132, 148, 200])
def test_tridiagonalisation_shape(lib, n, sms):
    out = (ctypes.c_longlong * 5)()
    lib.hh_shape_of(n, sms, out)
    smem_rows, threads, rows, grid, smem = out
    assert 1 <= grid <= sms   # a cooperative grid: one CTA per SM at most
    assert threads % 32 == 0 and n % threads == 0
    assert smem >= 16 * n * (3 + rows * smem_rows) and smem <= 227 * 1024 - 4096
    if smem_rows:
        assert grid * rows >= n   # rows in shared memory: each has a CTA of its own group
    assert smem_rows == (n <= 1024 and 8 * sms >= n)


# many parameter sets of a small circuit: their Hamiltonian partials alone are more than the estimate's fixed slack
@pytest.mark.parametrize("sets", [1, 64, 5000, 16384, 32768])
def test_worker_estimate_covers_the_partials(lib, sets):
    lib.worker_bytes.restype = lib.ham_partial_bytes.restype = ctypes.c_double
    lib.worker_bytes.argtypes = [ctypes.c_longlong] * 4 + [ctypes.c_int]
    joint, mats = sets << 14, 4 * sets
    need = 16 * joint + 16 * mats + sets * lib.ham_partial_bytes()
    assert lib.worker_bytes(joint, mats, sets, sets, 444) >= need
