"""A phase a caller asks for is applied however small it is: the plans of state programs drop a phase only where it is
exactly 1."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="session")
def shipped(tmp_path_factory):
    out = tmp_path_factory.mktemp("shipped") / "libshipped.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out), str(REPO / "tests" / "plan_shipped.cpp"),
                    *(str(REPO / "invariantq_b200" / "csrc" / f) for f in ("iq_sched.cpp", "iq_jitgen.cpp"))], check=True)
    return ctypes.CDLL(str(out))


def apply_shipped(lib, n, ops, state, M=12, c=4, R=4, stages=8, budget=160.0):
    """State after ops (LSB-first qubit list, matrix), and [passes, stages, merged diagonals]."""
    ks = np.array([len(q) for q, _ in ops], np.int32)
    qs = np.full((len(ops), 5), -1, np.int32)
    offs = np.zeros(len(ops), np.int64)
    flat, off = [], 0
    for i, (q, u) in enumerate(ops):
        qs[i, :len(q)] = q
        offs[i] = off
        flat.append(np.asarray(u, np.complex128).reshape(-1))
        off += flat[-1].size
    pool = np.concatenate(flat)
    st = np.ascontiguousarray(state, np.complex128).copy()
    counts, err = np.zeros(3, np.int32), ctypes.create_string_buffer(256)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)   # noqa: E731
    rc = lib.shipped_apply(n, M, c, R, stages, ctypes.c_double(budget), len(ops), p(ks), p(qs), p(pool), p(offs), p(st),
                           p(counts), err, 256)
    assert rc == 0, err.value.decode()
    return st, counts


def _ry(t):
    return np.array([[np.cos(t / 2), -np.sin(t / 2)], [np.sin(t / 2), np.cos(t / 2)]])


CX = np.array([[1, 0, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0], [0, 1, 0, 0]], complex)   # control local bit 0


# Rounds that differ from the identity by the phase e alone (every rotation is undone behind a CX that keeps them from
# merging): 1000 e on one half of the amplitudes, 2^-3.5 each.  Rounding: ~6000 products of two roundings of 1.1e-16
# each, at random: sqrt(6000) * 2.2e-16 * 2^-3.5 = 1.5e-15; ten times that.
@pytest.mark.parametrize("e", [1e-15, 1.9e-15, 2.1e-15, 5e-15, 1e-13])
def test_small_phases_add_up(shipped, e):
    n, rounds = 7, 1000
    ops = [([q], np.array([[1, 1], [1, -1]]) / np.sqrt(2)) for q in range(n)]
    p = np.diag([1.0, np.exp(1j * e)])
    for _ in range(rounds):
        ops += [([0], p), ([0, 1], CX), ([0], _ry(0.3)), ([0, 1], CX), ([0], _ry(-0.3)), ([0, 1], CX)]
        ops += [([0], _ry(0.3)), ([0, 1], CX), ([0], _ry(-0.3))]
    got, _ = apply_shipped(shipped, n, ops, np.eye(1 << n, 1).ravel())
    want = np.eye(1 << n, 1).ravel().astype(np.clongdouble)
    i = np.arange(1 << n)
    for q, u in ops:
        if len(q) == 2:
            want = want[np.where(i & 1, i ^ 2, i)]
            continue
        u = np.asarray(u).astype(np.clongdouble)
        x = want.reshape(-1, 2, 1 << q[0])
        want = np.stack((u[0, 0] * x[:, 0] + u[0, 1] * x[:, 1], u[1, 0] * x[:, 0] + u[1, 1] * x[:, 1]), 1).reshape(-1)
    assert float(abs(got - want).max()) <= 1.5e-14
