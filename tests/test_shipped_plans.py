"""The plans the library runs, emulated on the CPU (tests/plan_shipped.cpp): state programs in the steady decomposition and
single-set gradients in their Pauli frame, with the diagonals of each register stage merged."""
import ctypes

import numpy as np
import pytest

from invariantq_b200.circuits import tfim_terms
from tests import adjoint_ref as ar
from tests.test_scheduler_emulated import (apply_lsb_numpy, brickwall_ops, gen_ops, oracle_apply, rand_unitary, superop_lsb,
                                           to_lsb)
from tests.test_steady_phases import apply_shipped, shipped  # noqa: F401  (fixture)


@pytest.mark.parametrize("n,M,c,R,stages,budget,seed", [
    (7, 12, 4, 4, 8, 160.0, 0), (10, 10, 4, 4, 8, 160.0, 1), (13, 11, 4, 4, 6, 60.0, 2), (14, 12, 4, 4, 8, 160.0, 3),
    (14, 12, 4, 4, 4, 160.0, 4), (14, 12, 4, 4, 5, 160.0, 5), (13, 11, 3, 4, 8, 120.0, 6), (13, 11, 5, 3, 6, 60.0, 7),
    (14, 12, 5, 5, 8, 500.0, 8)])
def test_random_gates(port, shipped, n, M, c, R, stages, budget, seed):  # noqa: F811
    rng = np.random.default_rng(100 + seed)
    ops = gen_ops(rng, n, 80, kmax=R)
    start = rand_unitary(rng, 64)[:, 0].repeat(1 << (n - 6)) / 2.0 ** ((n - 6) / 2)
    want = oracle_apply(port, start.astype(np.complex128), n, ops)
    got, _ = apply_shipped(shipped, n, [to_lsb(*o) for o in ops], start, M, c, R, stages, budget)
    assert np.max(np.abs(got - want)) < 1e-12


@pytest.mark.parametrize("stages", [4, 5, 8])
def test_brickwall(port, shipped, stages):  # noqa: F811
    n = 15
    ops = brickwall_ops(n, 10, 3)
    want = oracle_apply(port, np.eye(1 << n, 1, dtype=complex).ravel().copy(), n, ops)
    got, (_, _, merged) = apply_shipped(shipped, n, [to_lsb(*o) for o in ops], np.eye(1 << n, 1).ravel(), stages=stages)
    assert np.max(np.abs(got - want)) < 1e-12 and merged > 0


def test_channels(shipped):  # noqa: F811
    from invariantq_b200.channels import build_kraus_channel
    from invariantq_b200.gates import gate_matrix
    nq, rng = 7, np.random.default_rng(4)
    chans = [build_kraus_channel(*a) for a in (("depolarizing", [1e-3]), ("amp_damping", [2e-3]), ("phase_damping", [1e-3]))]
    cx = gate_matrix("cx")[np.ix_([0, 2, 1, 3], [0, 2, 1, 3])]
    ops = []
    for layer in range(3):
        for q in range(nq):
            u = gate_matrix("u3", list(rng.uniform(0, 2 * np.pi, 3)))
            ops += [([nq + q], u), ([q], np.conj(u)), ([q, nq + q], superop_lsb(chans[0]))]
        for q in range(layer % 2, nq - 1, 2):
            ops += [([nq + q + 1, nq + q], cx), ([q + 1, q], cx)]
            ops += [([k, nq + k], superop_lsb(ch)) for k in (q, q + 1) for ch in chans[1:]]
    rho = rng.normal(size=1 << (2 * nq)) + 1j * rng.normal(size=1 << (2 * nq))
    want = rho.copy()
    for q, u in ops:
        want = apply_lsb_numpy(want, 2 * nq, q, u)
    got, _ = apply_shipped(shipped, 2 * nq, ops, rho)
    assert np.max(np.abs(got - want)) < 1e-12 * np.max(np.abs(want))


def _grad(lib, n, ops, theta, coeffs, paulis, M=11, c=4, stages=8, budget=160.0, R=4):
    cols = [np.array([o[k] for o in ops], np.int32) for k in range(4)]
    th, co = np.ascontiguousarray(theta, np.float64), np.ascontiguousarray(coeffs, np.float64)
    e, g, counts, err = ctypes.c_double(), np.zeros(len(theta)), np.zeros(3, np.int32), ctypes.create_string_buffer(256)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)   # noqa: E731
    rc = lib.shipped_adjoint(n, len(ops), *(p(a) for a in cols), p(th), len(co), p(co), "".join(paulis).encode(), M, c, R,
                             stages, ctypes.c_double(budget), ctypes.byref(e), p(g), len(theta), p(counts), err, 256)
    assert rc == 0, err.value.decode()
    return e.value, g, counts


def _check(port, lib, n, ops, theta, coeffs, paulis, **plan):
    e, g, counts = _grad(lib, n, ops, theta, coeffs, paulis, **plan)
    scale = max(1.0, np.abs(coeffs).sum())
    assert abs(e - ar.energy(port, n, ops, theta, coeffs, paulis)) < 1e-12 * scale
    assert np.max(np.abs(g - ar.param_shift(port, n, ops, theta, coeffs, paulis))) < 1e-11 * scale
    return counts


@pytest.mark.parametrize("n,layers,plan", [(7, 3, {}), (8, 3, {"M": 9}), (9, 2, {"M": 9, "stages": 4}), (9, 2, {"R": 3}),
                                           (8, 2, {"R": 5, "budget": 500.0})])
def test_tfim_gradient(port, shipped, n, layers, plan):  # noqa: F811
    rng = np.random.default_rng(n)
    ops = ar.tfim_ops(n, layers)
    theta = rng.uniform(0, 2 * np.pi, ar.n_params(ops))
    dgr, gdz, _ = _check(port, shipped, n, ops, theta, *tfim_terms(n, 0.7), **plan)
    if plan.get("R", 4) <= 4:
        assert dgr and gdz   # both merged forms took part


@pytest.mark.parametrize("n,ngates,seed,plan", [(7, 60, 1, {}), (8, 90, 2, {"M": 9, "budget": 60.0, "stages": 4}),
                                                (9, 120, 3, {"M": 9}), (8, 90, 4, {"R": 3})])
def test_mixed_gates_gradient(port, shipped, n, ngates, seed, plan):  # noqa: F811
    """Every gate kind, strings of X, Y and Z that do and do not commute with the frame, angles at which rotations
    are exactly 0, exactly a Pauli operator, and at the frame's threshold."""
    rng = np.random.default_rng(seed)
    ops = ar.random_ansatz(rng, n, ngates)
    theta = rng.uniform(-4 * np.pi, 4 * np.pi, ar.n_params(ops))
    special = np.array([0.0, np.pi, np.pi / 2, -np.pi / 2, 3 * np.pi, -np.pi])
    theta[::4] = special[np.arange(len(theta[::4])) % len(special)]
    _check(port, shipped, n, ops, theta, rng.normal(size=8), ["".join(rng.choice(list("IXYZ"), n)) for _ in range(8)], **plan)


def test_rescaled_sweep(port, shipped):  # noqa: F811
    """301 RX / RY steps whose divisors are about 1/sqrt(2): the backward list restores its scale every 120 steps."""
    n, ops, p = 7, [], 0
    for layer in range(43):
        for q in range(n):
            ops.append((ar.RY if (layer + q) % 2 else ar.RX, q, -1, p))
            p += 1
        ops += [(ar.CZ, q, q + 1, -1) for q in range(n - 1)]
    rng = np.random.default_rng(5)
    theta = np.where(rng.random(p) < 0.5, np.pi / 2, -np.pi / 2) + rng.normal(scale=1e-3, size=p)
    assert _check(port, shipped, n, ops, theta, *tfim_terms(n, 0.6), M=9)[2] == 2
