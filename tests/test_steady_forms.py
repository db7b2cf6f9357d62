"""Angle-independent operation lists (steady decomposition, Pauli frame) against the lists they stand for, on the CPU."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("steady") / "steady.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(HERE / "steady_forms.cpp"),
                    *(str(HERE.parent / "invariantq_b200/csrc" / f) for f in ("iq_sched.cpp", "iq_jitgen.cpp"))], check=True)
    d = ctypes.CDLL(str(so))
    d.steady_error.restype = d.frame_error.restype = ctypes.c_double
    d.structure.restype = ctypes.c_uint64
    return d


@pytest.mark.parametrize("n", [3, 4, 6])
@pytest.mark.parametrize("count", [1, 5, 40, 400])
def test_steady_decomposition(lib, n, count):
    for seed in range(12):
        assert lib.steady_error(n, count, 100 * n + seed) < 1e-13 * (10 + count)


@pytest.mark.parametrize("n", [2, 3, 5])
@pytest.mark.parametrize("count", [1, 8, 60, 300])
def test_pauli_frame(lib, n, count):
    for seed in range(12):
        assert lib.frame_error(n, count, 100 * n + seed) < 1e-13 * (10 + count)


@pytest.mark.parametrize("kind,n,depth", [(0, 14, 6), (0, 20, 20), (1, 16, 5), (2, 16, 5), (1, 20, 12), (2, 20, 12)])
def test_structure_does_not_depend_on_angles(lib, kind, n, depth):
    assert len({lib.structure(kind, n, depth, s) for s in range(6)} | {0}) == 2
