"""Single-set gradients of one ansatz share their plans, whatever the angles: neighbouring one-qubit gates that multiply into
one, among them those whose product is more often a flip than not (CPU)."""
import ctypes

import numpy as np
import pytest

from invariantq_b200.circuits import tfim_terms
from tests import adjoint_ref as ar
from tests.test_shipped_plans import _check
from tests.test_steady_phases import shipped  # noqa: F401  (fixture)

RX, RY, RZ, U3, P, CZ, CX, H, X, SX = range(1, 11)
ROWS = {"ry rz": (RY, RZ), "rz ry": (RZ, RY), "p rx p": (P, RX, P), "u3": (U3,), "rx ry": (RX, RY), "h": (H,), "h rz": (H, RZ), "h ry": (H, RY), "ry h": (RY, H),
        "sx ry": (SX, RY), "rx rz rx": (RX, RZ, RX), "ry rz ry": (RY, RZ, RY), "rx rx": (RX, RX), "u3 u3": (U3, U3),
        "rz h rz": (RZ, H, RZ), "rz sx rz": (RZ, SX, RZ), "p h p ry": (P, H, P, RY), "rz sx rz sx rz": (RZ, SX, RZ, SX, RZ),
        "rx ry rx": (RX, RY, RX), "x ry": (X, RY), "rx rz ry": (RX, RZ, RY), "h rx h": (H, RX, H)}


def ansatz(n, row, layers, link):
    ops, p = [], 0
    for layer in range(layers):
        for g in row:
            for q in range(n):
                ops.append((g, q, -1, p if g in (RX, RY, RZ, U3, P) else -1))
                p += {U3: 3, RX: 1, RY: 1, RZ: 1, P: 1}.get(g, 0)
        ops += [(link, q, (q + 1) % n, -1) for q in range(n)]
    return ops


def check_one_structure(shipped, n, ops):  # noqa: F811
    cols = [np.array([o[k] for o in ops], np.int32) for k in range(4)]
    shipped.shipped_structure.restype = ctypes.c_uint64
    p = lambda a: ctypes.c_void_p(a.ctypes.data)   # noqa: E731
    for backward in (0, 1):
        seen = set()
        for seed in range(8):
            th = np.random.default_rng(seed).uniform(0, 2 * np.pi, max(1, ar.n_params(ops)))
            seen.add(shipped.shipped_structure(n, len(ops), *(p(a) for a in cols), p(th), backward))
        assert len(seen) == 1 and 0 not in seen


@pytest.mark.parametrize("link", [CZ, CX])
@pytest.mark.parametrize("row", ROWS)
def test_one_structure(shipped, row, link):  # noqa: F811
    check_one_structure(shipped, 10, ansatz(10, ROWS[row], 3, link))


@pytest.mark.parametrize("seed", range(16))
def test_one_structure_of_mixed_gates(shipped, seed):  # noqa: F811
    n = 7 + seed % 4
    check_one_structure(shipped, n, ar.random_ansatz(np.random.default_rng(seed), n, 20 * (1 + seed % 5)))


@pytest.mark.parametrize("row", ["h ry", "rx rz rx", "rz h rz", "u3 u3"])
def test_gradient(port, shipped, row):  # noqa: F811
    n = 8
    ops = ansatz(n, ROWS[row], 2, CX)
    theta = np.random.default_rng(3).uniform(0, 2 * np.pi, ar.n_params(ops))
    _check(port, shipped, n, ops, theta, *tfim_terms(n, 0.8))
